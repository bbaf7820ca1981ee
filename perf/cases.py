"""Performance cases: the calls a user of the engine makes, with sizes over the range they are made at.

Each case is one call (or the few calls that belong together) through the Python
binding, which is a thin layer over the C ABI (include/pimc_gb300.h):

* ``node`` / ``action``  NodeModel- and Action-level calls with host arrays: what the
  pi-qmc adapters issue, one call per node evaluation or bisection level of a move
  decided on the host.
* ``chain``     one or a few replicas with every move recorded: a parity or debugging
  run, and pi-qmc's one clone per process.
* ``steps``     the production loop: a block of section attempts and one energy
  measurement of every replica as one graph, the configurations copied out after it.
* ``loop``      the same block driven from host buffers: paths up, moves, energies,
  paths down, over replicas that all differ.
* ``displace``  rigid displacement moves, which every equilibration interleaves.
* ``estimate``  the energy estimators on stored configurations.
* ``serve``     one round of a serving loop with a simulation leaving and one arriving.

Systems are the dots and electron gases of ``pimc_gb300.workloads``.  Launch
shapes are the engine's defaults.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "pi-qmc_gb300"))

import pimc_gb300  # noqa: E402
from pimc_gb300 import serving, workloads  # noqa: E402

TAU = 1.0 / 25.6  # the batch and serving workloads' time step


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a node model behind pi-qmc's own sampler: one slice pair of a 20-electron dot
        dict(name="node_dot20_one", op="node", system="dot", n=20, nslice=256, level=5, batch=1),
        # the 27 x 27 determinants of the electron gas over a section's worth of many walkers
        dict(name="node_heg54_batch", op="node", system="heg", n=54, nslice=512, level=5,
             batch=1024),
        # one bisection level of a move decided on the host, Ewald sums on level 0
        dict(name="action_heg54_one", op="action", system="heg", n=54, nslice=512, level=5,
             batch=1, at=0, precision="fp64"),
        # the same for many proposals of a dot at an upper level
        dict(name="action_dot20_batch", op="action", system="dot", n=20, nslice=1024, level=5,
             batch=512, at=1, precision="fp64"),
        # a single clone of the fixed-node dot in FP64, every move recorded
        dict(name="chain_dot20_fp64", op="chain", system="dot", n=20, nslice=1024, level=5,
             nodes=True, precision="fp64", replicas=1, attempts=64),
        # production sweep of the fixed-node dot
        dict(name="steps_dot20_mixed", op="steps", system="dot", n=20, nslice=1024, level=5,
             nodes=True, precision="mixed", replicas=304, attempts=640),
        # production sweep of the two-electron dot: thousands of small replicas
        dict(name="steps_dot2_fp64", op="steps", system="dot", n=2, nslice=256, level=4,
             nodes=False, precision="fp64", replicas=9728, attempts=32),
        # the periodic electron gas with Ewald sums and free-particle nodes
        dict(name="steps_heg54_mixed", op="steps", system="heg", n=54, nslice=512, level=5,
             nodes=True, precision="mixed", replicas=152, attempts=64),
        # uneven replicas driven from host buffers
        dict(name="loop_batch_mixed", op="loop", system="batch", n=32, precision="mixed",
             replicas=1024, attempts=16, mix=1),
        # equilibration of the electron gas by rigid displacements
        dict(name="displace_heg54", op="displace", system="heg", n=54, nslice=512, level=5,
             nodes=True, precision="fp64", replicas=19, attempts=4, nmoving=1),
        # estimators on stored configurations of the electron gas
        dict(name="estimate_heg54_fp64", op="estimate", system="heg", n=54, nslice=512, level=5,
             nodes=False, precision="fp64", replicas=8, window=16),
        # one round of a server holding a mix of dots
        dict(name="serve_round_mixed", op="serve", system="batch", n=32, precision="mixed",
             replicas=128, mix=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["node", "action", "chain", "steps", "steps", "loop", "displace", "estimate",
                     "serve"])
    c = dict(op=op, precision=rng.choice(["fp64", "mixed"]))
    if op in ("loop", "serve"):
        c.update(system="batch", n=rng.randint(8, 32), mix=rng.randrange(1 << 20),
                 replicas=_log_int(rng, 16, 512 if op == "loop" else 128))
        if op == "loop":
            c["attempts"] = rng.randint(4, 16)
        return c
    heg = rng.random() < 0.4
    c["system"] = "heg" if heg else "dot"
    c["level"] = rng.randint(3, 5)
    c["nslice"] = 2 * _log_int(rng, 40, 256)
    # closed shells of the grid the periodic paths start from, or any dot
    c["n"] = rng.choice([8, 14, 16, 27, 40, 54]) if heg else _log_int(rng, 2, 40)
    if op == "node":
        c["batch"] = _log_int(rng, 1, 1024)
        c["n"] = max(4, c["n"])
    elif op == "action":
        c["batch"] = _log_int(rng, 1, 64 if heg else 1024)
        c["at"] = rng.randint(0, c["level"] - 1)
    elif op == "estimate":
        c.update(nodes=False, replicas=_log_int(rng, 1, 8 if heg else 64), window=rng.choice([4, 8, 16, 32]))
    else:
        c["nodes"] = heg or (c["n"] > 3 and rng.random() < 0.7)
        if op == "chain":
            c.update(replicas=rng.randint(1, 4), attempts=rng.randint(16, 64))
        elif op == "steps":
            c.update(replicas=_log_int(rng, 1, 64 if c["nodes"] else 1024),
                     attempts=rng.randint(16, 64))
        else:
            c.update(replicas=_log_int(rng, 1, 19), attempts=rng.randint(1, 4),
                     nmoving=rng.randint(1, 2))
    return c


# ------------------------------------------------------------------ systems and paths
def _precision(case):
    return (pimc_gb300.PIMC_PREC_MIXED if case.get("precision") == "mixed"
            else pimc_gb300.PIMC_PREC_FP64)


def _system(case):
    """Workload keywords of a case's system (dots: ceil(n/2) up, floor(n/2) down)."""
    n, m, lev = case["n"], case["nslice"], case["level"]
    nodes = case.get("nodes", case["op"] == "node")
    up, dn = (n + 1) // 2, n // 2
    if case["system"] == "heg":
        kind = [pimc_gb300.PIMC_NODES_FREE if nodes else 0] * 2
        # the 54-electron gas's time step, so that links are as long as in production
        kw = workloads.heg54(n=n, nslice=m, nlevel=lev, node_kind=kind)
        beta = kw["beta"] * m / 512.0
        kw.update(beta=beta, node_temperature=1.0 / workloads.heg54()["beta"])
        return kw
    beta = 10.0 if n == 2 else (20.0 if m == 1024 else m * TAU)
    kind = [pimc_gb300.PIMC_NODES_SHO if nodes else 0] * 2
    kw = workloads.dot20_fn(counts=[up, dn], nslice=m, beta=beta, nlevel=lev, node_kind=kind)
    if not (n == 20 and m == 1024):  # the batch workload's node temperature
        kw["node_temperature"] = 0.25
    return kw


def _walkers(kw, nrep, rng):
    """Closed harmonic paths, sampled mode by mode: [nrep][nslice][npart][3].

    Dots: the oscillator's own thermal paths.  Electron gas: paths confined to a
    tenth of the lattice spacing about the sites of a simple-cubic grid."""
    m, n = kw["nslice"], sum(kw["counts"])
    tau = kw["beta"] / m
    if kw.get("mover", 0):
        side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
        spacing = kw["cell"] / side
        omega = 0.5 / (0.1 * spacing) ** 2
        sites = np.array([[i, j, k] for i in range(side) for j in range(side)
                          for k in range(side)], float)[:n] * spacing
        sites += -kw["cell"] / 2 + spacing / 2
    else:
        omega, sites = 1.0, None
    k = np.arange(m // 2 + 1)
    stiff = 4.0 * np.sin(math.pi * k / m) ** 2 / tau + omega * omega * tau
    z = rng.normal(size=(nrep, m // 2 + 1, n, 3)) + 1j * rng.normal(size=(nrep, m // 2 + 1, n, 3))
    z *= (math.sqrt(0.5 * m) / np.sqrt(stiff))[None, :, None, None]
    z[:, 0] = z[:, 0].real * math.sqrt(2.0)
    if m % 2 == 0:
        z[:, -1] = z[:, -1].real * math.sqrt(2.0)
    x = np.fft.irfft(z, n=m, axis=1)
    return x if sites is None else x + sites


def _start_paths(kw, nrep, rng):
    """Initial paths: thermal walkers where they cross no node, else paths constant in time."""
    if any(kw.get("node_kind", [0])) and not kw.get("mover", 0):
        n = sum(kw["counts"])
        return np.repeat(rng.normal(size=(nrep, 1, n, 3)), kw["nslice"], axis=1)
    return _walkers(kw, nrep, rng)


def _pinned(n):
    return torch.empty(int(n), dtype=torch.float64).pin_memory().numpy()


def _equilibrate(eng, attempts, rounds=4, ndisp=8):
    """Moves away from constant paths: whole-path displacements and bisection."""
    for _ in range(rounds):
        eng.run_displace(ndisp, [1.0, 1.0, 1.0], 1, -1)
        eng.run_sections(attempts)


def _engine(case, seed, rng):
    kw = _system(case)
    tabs, ew = pimc_gb300.coulomb_tables(kw)
    eng = pimc_gb300.Engine(kw, case["replicas"], tabs, ew, seed=seed,
                            precision=_precision(case))
    eng.upload_paths(_start_paths(kw, case["replicas"], rng).ravel())
    if any(kw["node_kind"]) and case["system"] == "dot":
        _equilibrate(eng, workloads.sweep_attempts(kw))
    return kw, tabs, ew, eng


_shared_tables = None


def _batch_tables():
    """The pair tables every dot of the batch and serving workloads shares."""
    global _shared_tables
    if _shared_tables is None:
        kw = workloads.dot20_fn(counts=[2, 2], nslice=256, beta=256 * TAU)
        _shared_tables = pimc_gb300.coulomb_tables(kw)[0]
    return _shared_tables


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    op = case["op"]
    if op in ("node", "action"):
        kw = _system(case)
        tabs, ew = pimc_gb300.coulomb_tables(kw)
        eng = pimc_gb300.Engine(kw, 1, tabs, ew, seed=seed, precision=_precision(case))
        return dict(op=op, eng=eng, **_arrays(case, kw, rng))
    if op == "serve":
        return _prepare_serve(case, seed, rng)
    if op == "loop":
        kws = workloads.batch_dots(case["replicas"], seed=case["mix"], slices=(128, 256, 512),
                                   nmax=case["n"])
        base = _batch_tables()
        eng = pimc_gb300.Engine.batch(kws, [workloads.tables_for(k, base) for k in kws],
                                      seed=seed, precision=_precision(case))
        eng.upload_paths([_start_paths(k, 1, rng)[0] for k in kws])
        _equilibrate(eng, 96)
        host = _pinned(eng.offsets[-1])
        eng.download_paths(flat=True, out=host)
        return dict(op=op, eng=eng, host=host, attempts=case["attempts"])
    kw, tabs, ew, eng = _engine(case, seed, rng)
    st = dict(op=op, eng=eng, host=_pinned(eng.offsets[-1]))
    if op == "estimate":
        st["window"] = case["window"]
        if ew is not None:
            st["rcut"] = 0.5 * kw["cell"]
            st["est"], st["vgrid"] = pimc_gb300.ewald_estimator_tables(kw, st["rcut"],
                                                                       kw["ewald_kcut"])
    else:
        st["attempts"] = case["attempts"]
        st["nmoving"] = case.get("nmoving", 1)
    return st


def _arrays(case, kw, rng):
    """Host arrays of the NodeModel- and Action-level calls."""
    b, n = case["batch"], sum(kw["counts"])
    if case["op"] == "node":
        # slice pairs (t, t + M/2); a dot's walkers, made without the node, get
        # their second bead near the first, where moves that cross no node keep it
        half = kw["nslice"] // 2
        x = _walkers(kw, -(-b // half), rng)
        r1 = np.ascontiguousarray(x[:, :half].reshape(-1, n, 3)[:b])
        r2 = np.ascontiguousarray(x[:, half:2 * half].reshape(-1, n, 3)[:b])
        if not kw.get("mover", 0):
            r2 = r1 + 0.05 * rng.normal(size=r1.shape)
        return dict(r1=r1, r2=r2)
    nsec = (1 << case["level"]) + 1
    x = _walkers(kw, b, rng)
    start = rng.integers(0, kw["nslice"], size=b)
    sl = (start[:, None] + np.arange(nsec)[None]) % kw["nslice"]
    sec = np.ascontiguousarray(x[np.arange(b)[:, None], sl])
    ip = rng.integers(0, n, size=b).astype(np.int32)
    mov = sec[np.arange(b), :, ip].copy()
    # a bisection move at level `at`: the beads between its end points are new
    tau = kw["beta"] / kw["nslice"]
    mov[:, 1:-1] += math.sqrt(0.5 * tau * (1 << case["at"])) * rng.normal(size=mov[:, 1:-1].shape)
    return dict(sections=sec, movings=mov, iparts=ip, level=case["at"])


def _prepare_serve(case, seed, rng):
    slots = case["replicas"]
    reqs = workloads.serve_stream(slots + 64, seed=case["mix"], nmax=2 * case["n"],
                                  slices=(64, 128, 256, 512))
    server = pimc_gb300.Server(slots, 4 << 30, 2 * case["n"], 512, 5, case["n"], seed=seed,
                               precision=_precision(case))
    base = _batch_tables()
    sched = serving.ServeLoop(server)
    todo = []
    for i, (_, kw, sweeps) in enumerate(reqs):
        r = serving.Request(i, kw, workloads.tables_for(kw, base), _start_paths(kw, 1, rng)[0],
                            max(1, int(sweeps * workloads.sweep_attempts(kw))))
        todo.append((kw, r.tables, r.path, sched.round_attempts(r)))
    st = dict(op="serve", server=server, todo=todo, next=0, slots=[], turn=0)
    for _ in range(slots):
        st["slots"].append(_admit(st))
    server.run()
    return st


def _admit(st):
    kw, tabs, path, ra = st["todo"][st["next"] % len(st["todo"])]
    slot = st["server"].admit(kw, tabs, path, st["next"], ra)
    st["next"] += 1
    return slot


def run(st):
    op = st["op"]
    if op == "node":
        err, det, d1, d2 = st["eng"].node_evaluate(0, st["r1"], st["r2"])
        return dict(err=err, det=det, d1=d1, d2=d2)
    if op == "action":
        return st["eng"].action_difference(st["level"], st["sections"], st["movings"], st["iparts"])
    if op == "serve":
        # a finished simulation leaves with its path, a waiting one takes its slot,
        # then a round, and the energies of the simulations that are due
        srv, slots = st["server"], st["slots"]
        k = st["turn"] % len(slots)
        out = srv.download_path(slots[k])
        srv.release(slots[k])
        slots[k] = _admit(st)
        st["turn"] += 1
        srv.run()
        due = [slots[i] for i in range(st["turn"] % 4, len(slots), 4)]
        return dict(path=out, energies=srv.energies(due))
    eng = st["eng"]
    if op == "chain":
        rec = eng.run_sections(st["attempts"], records=True)
        return dict(rec, path=eng.download_paths(flat=True, out=st["host"]))
    if op == "steps":
        e = eng.run_steps(st["attempts"], 1)
        return dict(energy=e, path=eng.download_paths(flat=True, out=st["host"]))
    if op == "loop":
        eng.upload_paths(st["host"])
        eng.run_sections(st["attempts"])
        e = eng.thermo_energy()
        return dict(energy=e, path=eng.download_paths(flat=True, out=st["host"]))
    if op == "displace":
        rec = eng.run_displace(st["attempts"], [1.0, 1.0, 1.0], st["nmoving"], -1, records=True)
        return dict(rec, path=eng.download_paths(flat=True, out=st["host"]))
    out = dict(thermo=eng.thermo_energy(), virial=eng.virial_energy(st["window"]),
               coulomb=eng.coulomb_energy())
    if "est" in st:
        out["ewald"] = eng.ewald_coulomb_energy(1.0, st["rcut"], st["est"], st["vgrid"])
    return out


# ------------------------------------------------------------------ necessary work
def _eval_flops(n):
    """One Slater evaluation: factorisation, inverse, both gradients, one new column."""
    return 2.0 * n ** 3 + 18.0 * n * n + 60.0 * n


def work(case):
    op = case["op"]
    if op == "serve":
        n, links, m = case["n"], 32, 256
        return dict(bytes=case["replicas"] * m * n * 48.0,
                    flops=case["replicas"] * (8 * 2 * 31 * _eval_flops(n // 2) +
                                              8 * 2 * links * n * 60.0 + m * n * n / 8 * 40.0))
    if op == "loop":
        n, m = (case["n"] + 2) / 2, 298
        per = case["attempts"] * (31 * _eval_flops(n / 2) + 63 * n * 60.0) + m * n * n / 2 * 40.0
        return dict(bytes=case["replicas"] * m * n * 48.0, flops=case["replicas"] * per)
    n, m, lev = case["n"], case["nslice"], case["level"]
    heg, nsec = case["system"] == "heg", (1 << lev) + 1
    half, mid = (n + 1) // 2, (1 << lev) - 1
    if op == "node":
        b = case["batch"]
        fill = half * half * (60.0 if heg else 30.0)
        return dict(bytes=b * (6.0 * n + 2 * n + 2) * 8, flops=b * (_eval_flops(half) + fill))
    kvec = 257.0 if heg else 0.0
    if op == "action":
        b = case["batch"]
        links = 1 << (lev - case["at"])
        f = links * n * 2 * 60.0 + (mid * kvec * n * 16.0 if case["at"] == 0 else 0.0)
        return dict(bytes=b * nsec * (n + 1) * 24.0, flops=b * f)
    r = case["replicas"]
    path = m * n * 24.0
    measure = m * (n * (n - 1) / 2 * 40.0 + n * 30.0 + kvec * 6)
    if op == "estimate":
        return dict(bytes=r * path, flops=r * (3 * measure + m * kvec * n * 12.0))
    if op == "displace":
        f = m * n * 2 * 60.0 + m * kvec * 40.0
        if case["nodes"]:
            f += m / 2 * _eval_flops(half)
        return dict(bytes=2 * r * path, flops=r * case["attempts"] * f)
    att = case["attempts"]
    per = 2 * (1 << lev) * n * 60.0 + mid * kvec * 40.0
    if case["nodes"]:
        per += mid * _eval_flops(half)
    return dict(bytes=2 * r * path,
                flops=r * (att * per + (measure if op == "steps" else 0.0)))


# ------------------------------------------------------------------ 64-bit values
def _image(kw, v):
    """SuperCell::pbc: minimum image of vectors longer than half the shortest side."""
    cell = kw["cell"]
    far = (v * v).sum(-1, keepdims=True) > 0.25 * cell * cell
    return np.where(far, v - cell * (np.floor(v / cell + 1000.5) - 1000), v)


def _norm(v):
    return np.sqrt((v * v).sum(-1))


def _pair_terms(tab, q, s2, want):
    """The tabulated pair action's series at (q, s^2): 'u', 'ut' or the derivatives 'd'."""
    g, nd = tab["ugrid"], tab["norder"] + 1
    z = q * tab["rgridinv"]
    x = np.log(np.maximum(z, 1e-300)) * tab["logrratioinv"]
    low, high = z < 1, x >= tab["ngpts"] - 1
    i = np.where(low, 0, np.where(high, tab["ngpts"] - 2, x)).astype(np.int64)
    x = np.where(low, 0.0, np.where(high, 1.0, x - i))
    if want == "d":
        uq, us = np.zeros_like(q), np.zeros_like(q)
        for k in range(nd - 1, -1, -1):
            uq = uq * s2 + (g[i + 1, 0, k] - g[i, 0, k])
        for k in range(nd - 1, 0, -1):
            us = us * s2 + k * ((1 - x) * g[i, 0, k] + x * g[i + 1, 0, k])
        return uq * tab["logrratioinv"] / q, us
    row = 1 if want == "ut" else 0
    if s2 is None:
        return (1 - x) * g[i, row, 0] + x * g[i + 1, row, 0]
    a = np.zeros_like(q)
    for k in range(nd - 1, -1, -1):
        a = a * s2 + ((1 - x) * g[i, row, k] + x * g[i + 1, row, k])
    return a


def _species(kw):
    return np.repeat(np.arange(len(kw["counts"])), kw["counts"])


def _table(tabs, a, b):
    for t in tabs:
        if tuple(sorted(t["species"])) == (min(a, b), max(a, b)):
            return t
    return None


def _exact_node(case, kw, rng):
    a = _arrays(case, kw, rng)
    n, cell = kw["counts"][0], kw["cell"]
    r1, r2 = a["r1"][:, :n], a["r2"][:, :n]
    mass, tau = 1.0, kw["beta"] / kw["nslice"]
    temp = kw.get("node_temperature", 1.0 / kw["beta"])
    if kw["node_kind"][0] == pimc_gb300.PIMC_NODES_SHO:
        w = kw["node_omega"][0]
        ch, c = math.cosh(0.5 * w / temp), 0.5 * mass * w / math.sinh(0.5 * w / temp)
        q = ((r2 ** 2).sum(-1)[:, :, None] + (r1 ** 2).sum(-1)[:, None, :]) * ch
        rho = np.exp(-c * (q - 2 * np.einsum("bid,bjd->bij", r2, r1)))  # [i of r2][j of r1]
        g1 = rho[..., None] * 2 * c * (r2[:, :, None] - ch * r1[:, None])
        g2 = rho[..., None] * 2 * c * (r1[:, None] - ch * r2[:, :, None])
    else:
        al = mass * temp * cell * cell
        nmax = 1 + int(2.0 * math.sqrt(al))
        nome, pref, kk = math.exp(-math.pi ** 2 / al), math.sqrt(math.pi / al), 2 * math.pi / cell
        x = _image(kw, r1[:, None] - r2[:, :, None])
        v, dv = np.ones_like(x), np.zeros_like(x)
        for m in range(1, nmax):
            v += 2 * nome ** (m * m) * np.cos(m * kk * x)
            dv -= 2 * kk * m * nome ** (m * m) * np.sin(m * kk * x)
        v, dv = pref * v, pref * dv
        rho = v.prod(-1)
        g1 = np.stack([dv[..., 0] * v[..., 1] * v[..., 2], v[..., 0] * dv[..., 1] * v[..., 2],
                       v[..., 0] * v[..., 1] * dv[..., 2]], -1)
        g2 = -g1
    inv = np.linalg.inv(rho)
    l1 = np.einsum("bji,bijd->bjd", inv, g1)
    l2 = np.einsum("bji,bijd->bid", inv, g2)
    b, np_ = len(r1), sum(kw["counts"])
    d1, d2 = np.full((b, np_), 200.0), np.full((b, np_), 200.0)
    d1[:, :n] = np.sqrt(2 * mass / (tau * ((l1 ** 2).sum(-1) + 1e-15)))
    d2[:, :n] = np.sqrt(2 * mass / (tau * ((l2 ** 2).sum(-1) + 1e-15)))
    return dict(err=None, det=np.linalg.det(rho), d1=d1, d2=d2)


def _long_range(kw, ew, x):
    """evalLongRange of slices [...][npart][3] (charges -1)."""
    dk = 2 * 3.14159265358979 / kw["cell"]
    out = np.zeros(x.shape[:-2])
    for k, v in zip(ew["kvec"], ew["vk"]):
        rho = np.exp(1j * dk * (x @ k.astype(float))).sum(-1)
        out += 2 * v * (rho.real ** 2 + rho.imag ** 2)
    return out * ew["one_over_2v"] + ew["self_energy"]


def _exact_action(case, kw, rng):
    tabs, ew = pimc_gb300.coulomb_tables(kw)
    a = _arrays(case, kw, rng)
    lev, step = case["at"], 1 << case["at"]
    sp = _species(kw)
    tau = kw["beta"] / kw["nslice"]
    ds = np.zeros(case["batch"])
    for b in range(case["batch"]):
        ip, sec = int(a["iparts"][b]), a["sections"][b][::step]
        for sign, own in ((1.0, a["movings"][b][::step]), (-1.0, sec[:, ip])):
            link = _image(kw, own[1:] - own[:-1])
            t = (link ** 2).sum() * 0.5 / (tau * step)
            w = kw.get("sho_omega", [0.0] * len(kw["counts"]))[sp[ip]]
            if w > 0:
                wt = w * tau * step
                rr = (own[1:] ** 2).sum(-1) + (own[:-1] ** 2).sum(-1)
                t += (w * (rr * math.cosh(wt) - 2 * (own[1:] * own[:-1]).sum(-1)) /
                      (2 * math.sinh(wt))).sum()
                t -= ((own[1:] - own[:-1]) ** 2).sum() / (2 * tau * step)
            for j in range(len(sp)):
                tab = _table(tabs, sp[ip], sp[j])
                if j == ip or tab is None:
                    continue
                d = _image(kw, own - sec[:, j])
                q = 0.5 * (_norm(d[1:]) + _norm(d[:-1]))
                s2 = ((d[1:] - d[:-1]) ** 2).sum(-1) / (q * q) if lev < 3 else None
                t += step * _pair_terms(tab, q, s2, "u").sum()
            ds[b] += sign * t
        if ew is not None and lev == 0:
            new = sec.copy()
            new[:, ip] = a["movings"][b]
            ds[b] += tau * (_long_range(kw, ew, new[1:-1]) - _long_range(kw, ew, sec[1:-1])).sum()
    return ds


def _exact_estimate(case, kw, rng):
    tabs, ew = pimc_gb300.coulomb_tables(kw)
    paths = _start_paths(kw, case["replicas"], rng)
    sp, m, nw = _species(kw), kw["nslice"], case["window"]
    tau, n = kw["beta"] / kw["nslice"], len(_species(kw))
    om = kw.get("sho_omega", [0.0] * len(kw["counts"]))
    out = dict(thermo=[], virial=[], coulomb=[], ewald=[])
    if ew is not None:
        rcut = 0.5 * kw["cell"]
        est, vgrid = pimc_gb300.ewald_estimator_tables(kw, rcut, kw["ewald_kcut"])
    for x in paths:
        back = np.roll(x, 1, axis=0)  # bead of the slice before
        d = _image(kw, x - back)
        utau = 1.5 / tau - (d ** 2).sum(-1) / (2 * tau * tau)
        fm, fp = -d / tau, -_image(kw, x - np.roll(x, -1, axis=0)) / tau
        w = np.array([om[s] for s in sp])
        if w.any():
            csch, coth = 1 / np.sinh(w * tau), 1 / np.tanh(w * tau)
            ch = np.cosh(w * tau)
            r0, r1 = (back ** 2).sum(-1), (x ** 2).sum(-1)
            utau += 1.5 * w * coth + 0.5 * w * w * ((r1 + r0) * (1 - coth ** 2) + 2 * (
                x * back).sum(-1) * ch * csch ** 2) + 0.5 * ((d ** 2).sum(-1) / tau - 3) / tau
            for f, o, dd in ((fm, back, d), (fp, np.roll(x, -1, axis=0), -fp * tau)):
                f -= (w * csch)[:, None] * (x * ch[:, None] - o) - dd / tau
        coul, ewc = 0.0, 0.0
        for i in range(n):
            for j in range(i):
                e = _image(kw, x[:, i] - x[:, j])
                r = _norm(e)
                coul += (1.0 / r).sum()
                if ew is not None:
                    near = r < rcut
                    g = (r[near] * (1000 / rcut)).astype(np.int64)
                    y = r[near] - g * (rcut / 1000)
                    ewc += (1.0 / r[near] + (1 - y) * vgrid[g] + y * vgrid[g + 1]).sum()
                tab = _table(tabs, sp[i], sp[j])
                if tab is None:
                    continue
                p, rp = np.roll(e, 1, axis=0), np.roll(r, 1)
                q = 0.5 * (r + rp)
                s2 = ((e - p) ** 2).sum(-1) / (q * q)
                utau[:, i] += _pair_terms(tab, q, s2, "ut")
                uq, us = _pair_terms(tab, q, s2, "d")
                # the link (t-1, t) acts on its end bead (fm at t) and its start (fp at t-1)
                f1 = -(uq / (2 * r))[:, None] * e - us[:, None] * (
                    2 * (e - p) / (q * q)[:, None] - (s2 / (q * r))[:, None] * e)
                f0 = -(uq / (2 * rp))[:, None] * p - us[:, None] * (
                    2 * (p - e) / (q * q)[:, None] - (s2 / (q * rp))[:, None] * p)
                fm[:, i] += f1
                fm[:, j] -= f1
                fp[:, i] += np.roll(f0, -1, axis=0)
                fp[:, j] -= np.roll(f0, -1, axis=0)
        lr = _long_range(kw, ew, x).sum() if ew is not None else 0.0
        out["thermo"].append((utau.sum() + lr) / m)
        out["coulomb"].append(coul / m)
        f, tot = fm + fp, utau.sum() + lr
        for t0 in range(0, m, nw):
            wlen = min(nw, m - t0) if t0 // nw >= (m - 1) // nw else nw
            rav, r0, fav = 0.0, 0.0, 0.0
            for k in range(min(nw, m - t0)):
                rav = rav + d[t0 + k]
                r0 = r0 + (wlen - k) * d[t0 + k] / wlen
                fav = fav + f[t0 + k]
                tot -= (1 - 1 / wlen) * 1.5 / tau * n + (f[t0 + k] * rav).sum() / (2 * tau)
            tot += (fav * r0).sum() / (2 * tau)
        out["virial"].append(tot / m)
        if ew is not None:
            out["ewald"].append((ewc + _long_range(kw, est, x).sum()) / m)
    return {k: np.array(v) for k, v in out.items() if v}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    op = case["op"]
    if op not in ("node", "action", "estimate"):
        return None  # a Markov chain: its decisions replay thousands of attempts
    kw = _system(case)
    if op == "node":
        return _exact_node(case, kw, rng)
    if op == "action":
        return _exact_action(case, kw, rng)
    return _exact_estimate(case, kw, rng)

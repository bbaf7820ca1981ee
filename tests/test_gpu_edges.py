"""Kernel branches at the sizes and inputs where they can go wrong, against plain
FP64 numpy or the C++ restatement (oracle/port.cc)."""
import numpy as np
import pytest

import oracle_lib as O
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pimc():
    import pimc_gb300
    pimc_gb300.build.build()
    return pimc_gb300


def _image(cell, v):
    """SuperCell::pbc in FP64 (src/util/SuperCell.cc:25-34)."""
    far = ((v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2]) > 0.25 * cell * cell
    img = v - cell * (np.floor((1.0 / cell) * v + 1000.5) - 1000)
    return np.where(far[:, None], img, v)


def _edge_vectors(cell, rng):
    """Differences at and next to the cutoff sphere, half-box components and box multiples."""
    out = []
    steps = [0.0, 1e-16, -1e-16, 3e-8, -3e-8, 9e-6, -9e-6, 1.1e-5, -1.1e-5, 4.2e-5, -4.2e-5, 1e-3,
             -1e-3]
    for f in steps:
        for _ in range(4):
            u = rng.normal(size=3)
            out.append(u / np.linalg.norm(u) * 0.5 * cell * (1 + f))
        out += [[0.5 * cell * (1 + f), 0.3 * cell, -0.1], [-0.5 * cell * (1 + f), 0.0, 0.2],
                [0.9 * cell, -0.5 * cell * (1 + f), 1e-9], [1.5 * cell * (1 + f), 0.1, 0.0],
                [cell * (1 + f), -cell * (1 + f), 0.01], [2.5 * cell * (1 + f), 0.2, -0.3],
                [1e-320, 0.6 * cell * (1 + f), 1e-30]]
    return np.array(out)


@pytest.mark.parametrize("cell", [10.0, 24.37179114151822])
def test_minimum_image_edges(pimc, cell):
    # One pair per slice, its difference at an edge of the minimum image; particle
    # 1 sits at the origin, so the difference is exactly particle 0's position.
    # (1/r is continuous across the cutoff; a wrong image changes it by O(1).)
    rng = np.random.default_rng(5)
    v = _edge_vectors(cell, rng)
    m = len(v) + len(v) % 2
    v = np.concatenate([v, v[:m - len(v)]])
    kw = W.dot2(nslice=m, nlevel=3, beta=m * 0.01, cell=cell, sho_omega=[0.0, 0.0])
    tabs, _ = pimc.coulomb_tables(kw)
    x = np.zeros((m, 2, 3))
    x[:, 0] = v
    ref = np.linalg.norm(_image(cell, v), axis=1)
    e = pimc.Engine(kw, 1, tabs)
    e.upload_paths([x])
    assert abs(e.coulomb_energy()[0] - (1 / ref).sum() / m) <= 1e-13 * (1 / ref).sum() / m
    port = O.PortOracle(O.make_config(**kw), tabs)
    port.set_path(x)
    want = port.thermo_energy()
    assert abs(e.thermo_energy()[0] - want) <= 1e-12 * abs(want)
    mixed = pimc.Engine(kw, 1, tabs, precision=pimc.PIMC_PREC_MIXED)
    mixed.upload_paths([x])
    assert abs(mixed.thermo_energy()[0] - want) <= 1e-5 * abs(want)


def _pg_images(al, cell, x):
    """Periodic Gaussian and its derivative by nine images: every term positive."""
    m = np.arange(-4, 5)[:, None, None, None, None]
    g = np.exp(-al * (x - m * cell) ** 2)
    return g.sum(0), (-2 * al * (x - m * cell) * g).sum(0)


@pytest.mark.parametrize("al2", [8.0, 19.999999, 20.000001, 39.999999, 40.000001, 400.0])
@pytest.mark.parametrize("n", [2, 9, 17])
def test_periodic_gaussian_images(pimc, al2, n):
    # Free-particle nodes on both sides of the line between the series and the
    # images, and with and without the second one, with separations up to exactly
    # half the box.  Forward error of the determinant and of the gradients: n eps
    # of the norms that enter.
    cell = 16.0
    kw = W.heg54(n=2 * n, nslice=64, nlevel=3, coulomb=0, ewald=0, cell=cell, beta=2.0,
                 node_temperature=al2 / cell ** 2)
    rng = np.random.default_rng(n)
    nb = 12
    r1 = rng.uniform(-cell / 2, cell / 2, size=(nb, 2 * n, 3))
    r2 = r1 + 0.15 * cell * rng.normal(size=r1.shape) / np.sqrt(al2)
    r2[0, 0] = r1[0, 1] + [cell / 2, 0.3 * cell, 0.0]
    r2[1, 1] = r1[1, 0] + [cell / 2, -cell / 2, cell / 2]
    r2[2, 0] = r1[2, 0]
    e = pimc.Engine(kw, 1)
    err, det, d1, _ = e.node_evaluate(0, r1, r2)
    x = r1[:, None, :n] - r2[:, :n, None]  # [b][i of r2][j of r1]
    x = x - cell * np.floor(x / cell + 0.5)
    v, dv = _pg_images(al2 / cell ** 2, cell, x)
    rho = v.prod(-1)
    grad = np.stack([dv[..., 0] * v[..., 1] * v[..., 2], v[..., 0] * dv[..., 1] * v[..., 2],
                     v[..., 0] * v[..., 1] * dv[..., 2]], -1)
    cond = np.linalg.cond(rho)
    # the series errs by ~1e-13 of its largest element where it cancels
    tol = (1e-12 if al2 < 20 else 1e-13) * n * cond
    assert not err.any()
    assert np.all(np.abs(det - np.linalg.det(rho)) <= tol * np.abs(det))
    inv = np.linalg.inv(rho)
    log = np.einsum("bji,bijd->bjd", inv, grad)
    ref = np.sqrt(2 / (kw["beta"] / 64 * ((log ** 2).sum(-1) + 1e-15)))
    size = np.einsum("bji,bijd->bjd", np.abs(inv), np.abs(grad)).sum(-1)
    slack = tol[:, None] * size * np.sqrt(kw["beta"] / 64 / 2) * ref ** 2 + 1e-12 * ref
    assert np.all(np.abs(d1[:, :n] - ref) <= slack)


@pytest.mark.parametrize("nlevel", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("counts,block", [([1], 32), ([1, 1], 64), ([3, 2], 32), ([4, 5], 256),
                                          ([17, 18], 128)])
def test_every_level_at_once(pimc, nlevel, counts, block):
    # The levels' links share a warp's lanes: one to six levels, fewer partners than
    # a warp takes at once up to several rounds of them, one to eight warps.
    kw = W.dot2(counts=counts, sho_omega=[1.0] * len(counts), nslice=64, beta=3.0, nlevel=nlevel)
    tabs, _ = pimc.coulomb_tables(kw)
    cfg = O.make_config(**kw)
    x = W.initial_path(cfg, "gauss", seed=3)
    port = O.PortOracle(cfg, tabs)
    port.set_path(x)
    ref = port.run(60)
    e = pimc.Engine(kw, 1, tabs)
    e.configure(block, 0, 0, 2)
    e.upload_paths([x])
    rec = e.run_sections(60, records=True)
    for k in ("ifirst1", "ipart", "reject_level"):
        assert np.array_equal(rec[k][0], ref[k]), k
    for k in ("ds", "lnt"):
        a, b = rec[k][0][:, :nlevel + 1], ref[k][:, :nlevel + 1]
        assert np.all(np.abs(a - b) <= 1e-12 * np.maximum(np.abs(b), 1.0)), k
    assert np.abs(e.download_paths()[0] - port.get_path()).max() <= 1e-12


@pytest.mark.parametrize("nlevel,cell", [(3, 4.3), (4, 6.1), (5, 8.6), (6, 12.2), (4, 30.0)])
def test_periodic_mover_images(pimc, nlevel, cell):
    # Boxes at the smallest width the periodic mover takes, where its image choices
    # need their exponentials, and one where they are certain.
    kw = W.dot2(counts=[2, 1], sho_omega=[0.0, 0.0], nslice=128, beta=128 * 0.02, nlevel=nlevel,
                cell=cell, mover=1)
    tabs, _ = pimc.coulomb_tables(kw)
    cfg = O.make_config(**kw)
    rng = np.random.default_rng(1)
    x = np.cumsum(rng.normal(size=(128, 3, 3)) * 0.14, axis=0)
    x -= np.linspace(0, 1, 128)[:, None, None] * x[-1]
    x += rng.uniform(-cell / 2, cell / 2, size=(1, 3, 3))
    x -= cell * np.floor(x / cell + 0.5)
    port = O.PortOracle(cfg, tabs)
    port.set_path(x)
    ref = port.run(200)
    e = pimc.Engine(kw, 1, tabs)
    e.upload_paths([x])
    rec = e.run_sections(200, records=True)
    for k in ("ifirst1", "ipart", "reject_level"):
        assert np.array_equal(rec[k][0], ref[k]), k
    a, b = rec["lnt"][0][:, :nlevel + 1], ref["lnt"][:, :nlevel + 1]
    assert np.all(np.abs(a - b) <= 1e-12 * np.maximum(np.abs(b), 1.0))
    assert np.abs(e.download_paths()[0] - port.get_path()).max() <= 1e-12


DISPLACE = {
    # (system, first paths): node models with and without cached entries, Ewald sums
    # with and without cached structure factors, odd slice counts
    "dot5_fn": (W.dot20_fn(counts=[3, 2], nslice=40, beta=2.0, nlevel=2, node_temperature=0.5),
                "const"),
    "dot5_fn_uncached": (W.dot20_fn(counts=[3, 2], nslice=16, beta=1.0, nlevel=3,
                                    node_temperature=0.5), "const"),
    "dot18_fn": (W.dot20_fn(counts=[9, 9], nslice=20, beta=1.0, nlevel=2, node_temperature=0.5),
                 "const"),
    "heg10": (W.heg54(n=10, nslice=16, nlevel=2, t_over_tf=1.5), "grid"),
    "heg10_one_species": (dict(W.heg54(n=10, nslice=16, nlevel=2, t_over_tf=1.5),
                               node_kind=[2, 0]), "grid"),
    "heg10_uncached": (W.heg54(n=10, nslice=8, nlevel=2, t_over_tf=3.0), "grid"),
    "dot3_odd": (W.dot2(counts=[2, 1], nslice=37, beta=2.0, nlevel=2), "gauss"),
}


@pytest.mark.parametrize("nmoving,species", [(1, -1), (3, -1), (2, 0)])
@pytest.mark.parametrize("nrep", [1, 21, 170])
@pytest.mark.parametrize("case", list(DISPLACE))
def test_displacements_then_sections(pimc, case, nrep, nmoving, species):
    # One to eight CTAs a replica, one to three particles: particles, displacements and
    # decisions as the restatement's, action differences to the displacement bars of
    # the golden test; then the sections that follow, whose cached entries and
    # structure factors the accepted displacements updated.
    kw, kind = DISPLACE[case]
    tabs, ew = pimc.coulomb_tables(kw)
    box = [1.2, 1.2, 1.2]
    e = pimc.Engine(kw, nrep, tabs, ew, seed=99)
    x = [W.initial_path(O.make_config(**kw), kind, seed=7 + r) for r in range(nrep)]
    e.upload_paths(x)
    e.run_sections(12)
    start = e.download_paths()
    scales = [e.replica_state(r)["node_scale"] for r in (0, nrep - 1)]
    d = e.run_displace(9, box, nmoving, species, records=True)
    paths = e.download_paths()
    s = e.run_sections(25, records=True)
    for r in {0, nrep - 1}:
        port = O.PortOracle(O.make_config(**dict(kw, seed=99, replica=r)), tabs, ew)
        port.set_path(x[r])
        port.run(12)
        assert np.abs(port.get_path() - start[r]).max() <= 1e-12
        ref = port.run_displace(9, box, nmoving, species, first_attempt=12)
        assert np.array_equal(d["ipart"][r], ref["ipart"])
        assert np.array_equal(d["disp"][r], ref["disp"])
        assert np.array_equal(d["accepted"][r], ref["accepted"])
        for k, tol in (("ds", 1e-11), ("ds_node", 1e-9)):
            assert np.all(np.abs(d[k][r] - ref[k]) <= tol * np.maximum(np.abs(ref[k]), 1.0)), k
        assert np.abs(port.get_path() - paths[r]).max() <= 1e-12
        ref = port.run(25, first_attempt=21)
        for k in ("ifirst1", "ipart", "reject_level"):
            assert np.array_equal(s[k][r], ref[k]), k
        nl = kw["nlevel"] + 1
        for k, tol in (("ds", 1e-11), ("ds_node", 1e-9)):
            a, b = s[k][r][:, :nl], ref[k][:, :nl]
            assert np.all(np.abs(a - b) <= tol * np.maximum(np.abs(b), 1.0)), k


ESTIMATE = {
    "one": W.dot2(counts=[1], sho_omega=[1.0], nslice=37, beta=2.0, nlevel=2, coulomb=0),
    "dot3_odd": W.dot2(counts=[2, 1], nslice=37, beta=2.0, nlevel=2),
    "dot67": W.dot2(counts=[40, 27], sho_omega=[1.0, 0.5], nslice=70, beta=3.0, nlevel=3),
    "dot5_prim": W.dot2(counts=[3, 2], sho_omega=[0.0, 1.0], prim_a=[0.5, 0.0],
                        prim_b=[0.05, 0.0], nslice=64, beta=3.0, nlevel=3),
    # grid paths: image ties in every pair; Ewald with and without cached structure factors
    "heg8_ties": W.heg54(n=8, nslice=128, nlevel=3),
    "heg10_uncached": W.heg54(n=10, nslice=8, nlevel=2, t_over_tf=3.0),
}


@pytest.mark.parametrize("case", list(ESTIMATE))
def test_estimators_over_windows(pimc, case):
    # Windows that divide the path, that do not, and the whole path; sums of
    # M N^2 terms of mixed sign: 1e-11 of their absolute scale.
    kw = ESTIMATE[case]
    tabs, ew = pimc.coulomb_tables(kw)
    cfg = O.make_config(**kw)
    x = W.initial_path(cfg, "grid" if kw.get("mover") else "gauss", seed=5)
    if case == "heg10_uncached":
        x = x + 0.3 * np.random.default_rng(2).normal(size=x.shape)
    port = O.PortOracle(cfg, tabs, ew)
    port.set_path(x)
    e = pimc.Engine(kw, 3, tabs, ew)
    e.upload_paths([x] * 3)
    m = kw["nslice"]
    for w in (1, 4, 5, m // 2, m):
        ref = port.virial_energy(w)
        scale = max(1.0, abs(ref), abs(port.virial_energy(1)))
        assert np.all(np.abs(e.virial_energy(w) - ref) <= 1e-11 * scale), w
    if kw["coulomb"]:
        ref = port.coulomb_energy(1.0)
        assert np.all(np.abs(e.coulomb_energy(1.0) - ref) <= 1e-12 * abs(ref))
    if ew is not None:
        rcut = 0.5 * kw["cell"]
        est, vg = pimc.ewald_estimator_tables(kw, rcut, kw["ewald_kcut"])
        ref = port.ewald_coulomb_energy(1.0, rcut, est, vg)
        assert np.all(np.abs(e.ewald_coulomb_energy(1.0, rcut, est, vg) - ref) <= 1e-11 *
                      max(1.0, abs(ref)))
    ref = port.thermo_energy()
    assert np.all(np.abs(e.thermo_energy() - ref) <= 1e-12 * max(1.0, abs(ref)))


@pytest.mark.parametrize("n,heg", [(1, False), (8, False), (9, False), (16, False), (17, True),
                                   (27, True), (32, False)])
def test_node_evaluate_batches(pimc, n, heg):
    # Batches of one pair, part of a warp's lane groups, one wave and more than the
    # resident warps: each pair's results do not depend on the batch, bit for bit, and
    # are the restatement's.
    if heg:
        kw = W.heg54(n=2 * n, nslice=64, nlevel=3, beta=2.0, coulomb=0, ewald=0)
    else:
        kw = W.dot20_fn(counts=[n, 1], nslice=64, beta=4.0, nlevel=3, coulomb=0,
                        node_temperature=0.5)
    npart = sum(kw["counts"])
    rng = np.random.default_rng(n)
    nb = 3001
    side = kw["cell"] if heg else 3.0
    r1 = rng.uniform(-side / 2, side / 2, size=(nb, npart, 3))
    r2 = r1 + 0.1 * rng.normal(size=r1.shape)
    e = pimc.Engine(kw, 1)
    whole = e.node_evaluate(0, r1, r2)
    for b in (1, 2, 3, 31, 153, 913):
        part = e.node_evaluate(0, r1[:b], r2[:b])
        for x, y in zip(part, whole):
            assert np.array_equal(x, y[:b]), b
    port = O.PortOracle(O.make_config(**kw))
    for b in (0, nb - 1):
        perr, pdet, pd1, pd2 = port.node_eval(0, r1[b], r2[b], 0, False)
        assert whole[0][b] == perr
        assert abs(whole[1][b] - pdet) <= 1e-8 * abs(pdet)
        assert np.all(np.abs(whole[2][b] - pd1) <= 1e-8 * pd1)
        assert np.all(np.abs(whole[3][b] - pd2) <= 1e-8 * pd2)


@pytest.mark.parametrize("nbatch", [1, 3, 40, 400])
@pytest.mark.parametrize("case", ["heg10", "heg10_uncached", "dot3_odd"])
def test_action_difference_batches(pimc, case, nbatch):
    # The section's slices over many CTAs and few, every level.
    kw, _ = DISPLACE[case]
    tabs, ew = pimc.coulomb_tables(kw)
    cfg = O.make_config(**kw)
    port = O.PortOracle(cfg, tabs, ew)
    e = pimc.Engine(kw, 1, tabs, ew)
    rng = np.random.default_rng(4)
    nsec = (1 << kw["nlevel"]) + 1
    sec = rng.normal(size=(nbatch, nsec, cfg.npart, 3)) * 2.0
    ip = rng.integers(0, cfg.npart, nbatch)
    mov = sec[np.arange(nbatch), :, ip].copy()
    mov[:, 1:-1] += 0.3 * rng.normal(size=mov[:, 1:-1].shape)
    for level in range(kw["nlevel"] + 1):
        ds = e.action_difference(level, sec, mov, ip)
        for b in list(range(min(nbatch, 3))) + [nbatch - 1]:
            ref = port.action_diff(level, sec[b], mov[b], int(ip[b]))
            assert abs(ds[b] - ref) <= 1e-12 * max(abs(ref), 1.0), (level, b)


@pytest.mark.parametrize("rmin,rmax,ngpts", [(0.005, 20.0, 500), (1.0, 3.0, 2), (1e-4, 300.0, 97)])
def test_pair_table_grid_edges(pimc, rmin, rmax, ngpts):
    # Distances at the grid's points and ends, in every octave, below, beyond and far
    # beyond it, through the Action-level call at a diagonal level (u00 alone) and an
    # off-diagonal one.  One interpolation of two table values: 1e-12 of the largest.
    kw = W.dot2(nslice=64, nlevel=4, beta=2.0, sho_omega=[0.0, 0.0], spring=0)
    tabs, _ = pimc.coulomb_tables(kw, ngpts=ngpts, rmin=rmin, rmax=rmax)
    t = tabs[0]
    r = np.concatenate([1.0 / t["rgridinv"] * np.exp(np.arange(ngpts) / t["logrratioinv"]),
                        rmin * 2.0 ** np.arange(-3, 24), [rmax * (1 + 1e-15), rmax, rmin, 1e-9]])
    r = np.concatenate([r, r * (1 + 1e-14), r * (1 - 1e-14), r * 1.013])
    r = r[r < 490.0]  # inside half the cell
    cfg = O.make_config(**kw)
    port = O.PortOracle(cfg, tabs)
    e = pimc.Engine(kw, 1, tabs)
    sec = np.zeros((len(r), 17, 2, 3))
    sec[:, :, 0, 0] = r[:, None]
    sec[:, ::2, 0, 1] = 1e-3 * r[:, None]
    mov = sec[:, :, 0].copy()
    mov[:, 1:-1, 0] = np.roll(r, 7)[:, None]
    size = np.abs(np.asarray(t["ugrid"])[:, 0, 0]).max() * 16
    for level in (1, 3):
        ds = e.action_difference(level, sec, mov, np.zeros(len(r), np.int32))
        ref = np.array([port.action_diff(level, sec[b], mov[b], 0) for b in range(len(r))])
        assert np.all(np.abs(ds - ref) <= 1e-12 * size), level


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("counts", [[1, 2], [4, 3], [8, 7], [9, 10], [16, 5]])
def test_lane_group_widths(pimc, counts, mixed):
    # A launch of at most one CTA per SM evaluates Slater matrices with wider lane
    # groups than a fuller one: the same chains, bit for bit, and the oracle's.
    kw = W.dot20_fn(counts=counts, nslice=64, beta=64 / 25.6, nlevel=4)
    tabs, _ = pimc.coulomb_tables(kw)
    cfg = O.make_config(**kw)
    x = W.initial_path(cfg, "gauss", seed=3)
    nrep, natt = 700, 24
    few = pimc.Engine(kw, 2, tabs, seed=9, precision=mixed)
    many = pimc.Engine(kw, nrep, tabs, seed=9, precision=mixed)
    few.upload_paths([x] * 2)
    many.upload_paths([x] * nrep)
    a, b = few.run_sections(natt, records=True), many.run_sections(natt, records=True)
    for k in a:
        assert np.array_equal(a[k], b[k][:2], equal_nan=True), k
    assert np.array_equal(few.download_paths()[1], many.download_paths()[1])
    if not mixed:
        port = O.PortOracle(cfg, tabs)
        port.set_path(x)
        ref = port.run(natt)
        c = pimc.Engine(kw, 1, tabs)
        c.upload_paths([x])
        rec = c.run_sections(natt, records=True)
        assert np.array_equal(rec["reject_level"][0], ref["reject_level"])
        assert np.abs(c.download_paths()[0] - port.get_path()).max() <= 1e-10


@pytest.mark.parametrize("n", [3, 8, 9, 17])
def test_node_evaluate_widths(pimc, n):
    # Small batches take wider lane groups than large ones: the same values, bit for bit.
    kw = W.dot20_fn(counts=[n, 1], nslice=64, beta=64 / 25.6, nlevel=4)
    e = pimc.Engine(kw, 1, pimc.coulomb_tables(kw)[0])
    rng = np.random.default_rng(n)
    r1 = rng.normal(size=(5000, n + 1, 3))
    r2 = r1 + 0.05 * rng.normal(size=r1.shape)
    ref = e.node_evaluate(0, r1, r2)
    for b in (1, 3, 150, 700, 1300):
        for x, y in zip(e.node_evaluate(0, r1[:b], r2[:b]), ref):
            assert np.array_equal(x, y[:b])

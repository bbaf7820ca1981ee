"""What callers rely on beyond the values themselves: inputs that are accepted, and
results that do not depend on what else a call or an engine holds."""
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


@pytest.mark.parametrize("sign", [1, -1])
def test_infinite_table_entries(pimc, sign):
    # A hard core: the potential's rows below a radius are infinite.  A move into it
    # has an infinite action difference and is rejected, as with pi-qmc's
    # interpolation (1 - x) g0 + x g1 (which is NaN at x = 0, below the grid); an
    # infinite well at the Action-level call alone.
    kw = W.dot2(counts=[2, 1], nslice=64, nlevel=4, beta=4.0, sho_omega=[1.0, 1.0])
    tabs, _ = pimc.coulomb_tables(kw)
    for t in tabs:
        r = np.exp(np.arange(t["ngpts"]) / t["logrratioinv"]) / t["rgridinv"]
        t["ugrid"][r < 0.8, 0, 0] = sign * np.inf
    cfg = O.make_config(**kw)
    port = O.PortOracle(cfg, tabs)
    e = pimc.Engine(kw, 1, tabs)
    x = np.tile(np.array([[1.0, 0, 0], [-0.6, 0.9, 0], [-0.6, -0.9, 0.1]]), (64, 1, 1))
    if sign > 0:
        port.set_path(x)
        ref = port.run(400)
        e.upload_paths([x])
        rec = e.run_sections(400, records=True)
        assert np.isinf(ref["ds"]).any() and (ref["reject_level"] < 0).any()
        for k in ("ifirst1", "ipart", "reject_level"):
            assert np.array_equal(rec[k][0], ref[k]), k
        a, b = rec["ds"][0][:, :5], ref["ds"][:, :5]
        assert np.array_equal(np.isinf(a), np.isinf(b))
        assert np.abs(e.download_paths()[0] - port.get_path()).max() <= 1e-12
    sec = np.tile(x[:17], (3, 1, 1, 1))
    mov = sec[:, :, 0].copy()
    mov[0, 1:-1] = x[0, 1] + [0.3, 0, 0]
    mov[1, 1:-1] = x[0, 1] + [1e-4, 0, 0]  # below the grid
    mov[2, 1:-1] += 0.1
    for level in range(5):
        ds = e.action_difference(level, sec, mov, np.zeros(3, np.int32))
        ref = np.array([port.action_diff(level, sec[b], mov[b], 0) for b in range(3)])
        assert level > 2 or ref[0] == sign * np.inf  # (longer links end outside)
        assert np.isfinite(ref[2])
        np.testing.assert_allclose(ds, ref, rtol=1e-12, atol=1e-12)  # (infinities, NaN alike)


def test_several_tables_of_one_pair(pimc):
    # Two tables of the same species pair act together, in the virial estimator as in
    # the moves: a table split in two halves is the whole one.
    kw = W.dot2(counts=[3, 2], nslice=64, nlevel=3, beta=4.0)
    tabs, _ = pimc.coulomb_tables(kw)
    halves = [dict(t, ugrid=f * np.asarray(t["ugrid"])) for f in (0.25, 0.75) for t in tabs]
    x = W.initial_path(dict(kw), "gauss", seed=3)
    one, two = pimc.Engine(kw, 1, tabs), pimc.Engine(kw, 1, halves)
    for e in (one, two):
        e.upload_paths([x])
    port = O.PortOracle(O.make_config(**kw), halves)
    port.set_path(x)
    for w in (1, 16):
        a, b, ref = one.virial_energy(w)[0], two.virial_energy(w)[0], port.virial_energy(w)
        scale = 1e-11 * max(1.0, abs(ref), abs(one.virial_energy(1)[0]))
        assert abs(a - b) <= scale and abs(b - ref) <= scale, w
    ra, rb = (e.run_sections(50, records=True) for e in (one, two))
    assert np.array_equal(ra["reject_level"], rb["reject_level"])


@pytest.mark.parametrize("nmoving", [1, 3])
@pytest.mark.parametrize("nodes", [0, 2])
def test_displacements_in_long_boxes(pimc, nodes, nmoving):
    # A box ninety times as long as wide has wave vectors far up one axis: tables of a
    # displaced bead that do not fit shared memory for every warp.
    kw = W.heg54(n=10, cell=[10.0, 10.0, 900.0], nslice=16, nlevel=2, beta=1.6,
                 ewald_kcut=5 * 2 * np.pi / 10.0, node_kind=[nodes, nodes])
    tabs, ew = pimc.coulomb_tables(kw)
    assert ew["ikmax"][2] > 400
    rng = np.random.default_rng(3)
    site = rng.uniform(-0.5, 0.5, size=(1, 10, 3)) * [10.0, 10.0, 900.0]
    x = np.repeat(site, 16, axis=0)
    cfg = O.make_config(**dict(kw, seed=4, cell=10.0))
    cfg.cell[2] = 900.0
    port = O.PortOracle(cfg, tabs, ew)
    port.set_path(x)
    ref = port.run_displace(6, [1.0, 1.0, 5.0], nmoving, -1)
    e = pimc.Engine(kw, 1, tabs, ew, seed=4)
    e.upload_paths([x])
    d = e.run_displace(6, [1.0, 1.0, 5.0], nmoving, -1, records=True)
    assert np.array_equal(d["accepted"][0], ref["accepted"]) and ref["accepted"].any()
    for k, tol in (("ds", 1e-11), ("ds_node", 1e-9)):
        assert np.all(np.abs(d[k][0] - ref[k]) <= tol * np.maximum(np.abs(ref[k]), 1.0)), k
    assert np.abs(port.get_path() - e.download_paths()[0]).max() <= 1e-12
    # the structure factors that the moves left are those of the paths
    f = pimc.Engine(kw, 1, tabs, ew, seed=4)
    f.upload_paths([e.download_paths()[0]])
    assert e.thermo_energy()[0] == f.thermo_energy()[0]


@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("counts", [[1, 1], [4, 3], [20, 21]])
def test_mixed_sections_without_nodes(pimc, counts, block):
    # Without Slater matrices every warp takes action terms in both precision forms: on
    # the attempts that both chains make alike, ln T bit for bit and action
    # differences within the mixed form's 1e-4 of max(|dS|, 1).
    kw = W.dot2(counts=counts, nslice=64, beta=64 / 25.6, nlevel=4)
    tabs, _ = pimc.coulomb_tables(kw)
    x = W.initial_path(dict(kw), "gauss", seed=3)
    rec = []
    for precision in (0, 1):
        e = pimc.Engine(kw, 4, tabs, seed=5, precision=precision)
        e.configure(block, 0, 0, 2)
        e.upload_paths([x] * 4)
        rec.append(e.run_sections(40, records=True))
    f, m = rec
    alike = np.cumprod((f["reject_level"] == m["reject_level"]) & (f["ipart"] == m["ipart"]),
                       axis=1).astype(bool)
    assert alike.mean() > 0.5
    assert np.array_equal(f["lnt"][alike][:, :5], m["lnt"][alike][:, :5])
    a, b = m["ds"][alike][:, :5], f["ds"][alike][:, :5]
    assert np.all(np.abs(a - b) <= 1e-4 * np.maximum(np.abs(b), 1.0))


THERMO = {
    "dot4": W.dot2(counts=[2, 2], nslice=1024, beta=40.0),
    "dot8_odd": W.dot2(counts=[5, 3], nslice=333, beta=13.0, nlevel=3),
    "dot3_odd": W.dot2(counts=[2, 1], nslice=1237, beta=20.0, nlevel=2),
    "dot20": W.dot2(counts=[10, 10], nslice=300, beta=12.0, nlevel=3),
    "one": W.dot2(counts=[1], sho_omega=[1.0], nslice=9001, beta=90.0, nlevel=2, coulomb=0),
    "heg8": W.heg54(n=8, nslice=520, nlevel=3, node_kind=[0, 0]),
    "heg10_uncached": W.heg54(n=10, nslice=8, nlevel=2, t_over_tf=3.0, node_kind=[0, 0]),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", list(THERMO))
def test_thermo_energy_of_one_and_many(pimc, case, precision):
    # A replica's energy does not depend on how many are measured beside it, bit for
    # bit, and is the restatement's.
    kw = THERMO[case]
    tabs, ew = pimc.coulomb_tables(kw) if kw["coulomb"] else ((), None)
    rng = np.random.default_rng(1)
    x = [W.initial_path(dict(kw), "grid" if kw.get("mover") else "gauss", seed=r) for r in range(3)]
    x = [a + 0.2 * rng.normal(size=a.shape) for a in x]
    want = None
    for nrep in (1, 3, 40, 500):
        e = pimc.Engine(kw, nrep, tabs, ew, precision=precision)
        e.upload_paths([x[r % 3] for r in range(nrep)])
        got = e.thermo_energy()
        e.close()
        assert np.array_equal(got, np.tile(got[:3], -(-nrep // 3))[:nrep])
        if want is None:
            want = got[0]
            port = O.PortOracle(O.make_config(**kw), tabs, ew)
            port.set_path(x[0])
            ref = port.thermo_energy()
            assert abs(want - ref) <= (1e-5 if precision else 1e-12) * max(1.0, abs(ref))
        assert got[0] == want


def test_thermo_energy_in_a_long_box(pimc):
    # Wave vectors far up one axis: their tables fill the shared memory that the parts'
    # sums would take beside them.
    kw = W.heg54(n=13, cell=[10.0, 10.0, 936.0], nslice=128, nlevel=2, beta=12.8,
                 ewald_kcut=5 * 2 * np.pi / 10.0, node_kind=[0, 0])
    tabs, ew = pimc.coulomb_tables(kw)
    rng = np.random.default_rng(3)
    x = np.repeat(rng.uniform(-0.5, 0.5, size=(1, 13, 3)) * [10.0, 10.0, 936.0], 128, axis=0)
    x += 0.05 * rng.normal(size=x.shape)
    cfg = O.make_config(**dict(kw, cell=10.0))
    cfg.cell[2] = 936.0
    port = O.PortOracle(cfg, tabs, ew)
    port.set_path(x)
    e = pimc.Engine(kw, 1, tabs, ew)
    e.upload_paths([x])
    ref = port.thermo_energy()
    assert abs(e.thermo_energy()[0] - ref) <= 1e-12 * max(1.0, abs(ref))


FEW_AND_MANY = {
    # (system, paths, replicas of the larger engine): one warp a replica instead of two
    # from eight replicas an SM on; four warps instead of eight, two CTAs an SM, for
    # systems of which eight warps fill an SM, with more replicas than SMs
    "dot2": (W.dot2(nslice=64, beta=2.5), "gauss", 1300),
    "dot4_L3": (W.dot2(counts=[2, 2], nslice=64, beta=2.5, nlevel=3), "gauss", 1300),
    "one_L6": (W.dot2(counts=[1], sho_omega=[1.0], nslice=64, beta=2.5, nlevel=6, coulomb=0),
               "gauss", 1300),
    "dot2_dr": (W.dot2(nslice=64, beta=2.5, delayed_rejection=1), "gauss", 1300),
    "heg4": (W.heg54(n=4, nslice=1024, nlevel=4, node_kind=[0, 0]), "grid", 1300),
    "heg4_uncached": (W.heg54(n=4, nslice=16, nlevel=4, beta=0.4, node_kind=[0, 0]), "grid", 1300),
    "dot32_fn": (W.dot20_fn(counts=[16, 16], nslice=128, beta=5.0, node_temperature=0.25),
                 "const", 640),
    "heg54": (W.heg54(nslice=256, nlevel=3), "grid", 170),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", list(FEW_AND_MANY))
def test_chains_of_few_and_many_replicas(pimc, case, precision):
    # A replica's chain does not depend on how many replicas its engine has, bit for bit.
    kw, kind, nrep = FEW_AND_MANY[case]
    tabs, ew = pimc.coulomb_tables(kw) if kw["coulomb"] else ((), None)
    x = [W.initial_path(dict(kw), kind, seed=r) for r in range(2)]
    few = pimc.Engine(kw, 2, tabs, ew, seed=9, precision=precision)
    many = pimc.Engine(kw, nrep, tabs, ew, seed=9, precision=precision)
    few.upload_paths(x)
    many.upload_paths([x[r % 2] for r in range(nrep)])
    a, b = few.run_sections(30, records=True), many.run_sections(30, records=True)
    for k in a:
        assert np.array_equal(a[k], b[k][:2], equal_nan=True), k
    for p, q in zip(few.download_paths(), many.download_paths()):
        assert np.array_equal(p, q)
    blocks = few.launch_config()["block"], many.launch_config()["block"]
    assert blocks == ((64, 32) if nrep == 1300 else (256, 128))


FEW_AND_MANY_DISPLACED = {
    "dot2": (W.dot2(nslice=256, beta=10.0), "gauss"),
    "dot5_fn": (W.dot20_fn(counts=[3, 2], nslice=40, beta=2.0, nlevel=2, node_temperature=0.5),
                "const"),
    "dot20_fn": (W.dot20_fn(nslice=128, beta=5.0, nlevel=4, node_temperature=0.25), "const"),
    "heg10": (W.heg54(n=10, nslice=16, nlevel=2, t_over_tf=1.5), "grid"),
    "heg10_uncached": (W.heg54(n=10, nslice=8, nlevel=2, t_over_tf=3.0), "grid"),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", list(FEW_AND_MANY_DISPLACED))
def test_displacements_of_few_and_many_replicas(pimc, case, precision):
    # The CTAs that share a replica are as many as the replicas leave room for: the
    # decisions' sums do not depend on them, bit for bit.
    kw, kind = FEW_AND_MANY_DISPLACED[case]
    tabs, ew = pimc.coulomb_tables(kw)
    x = W.initial_path(dict(kw), kind, seed=3)
    want = None
    for nrep in (1, 21, 60, 170, 700):
        e = pimc.Engine(kw, nrep, tabs, ew, seed=99, precision=precision)
        e.upload_paths([x] * nrep)
        d = e.run_displace(12, [0.8, 0.8, 0.8], 1, -1, records=True)
        got = [d[k][0] for k in sorted(d)] + [e.download_paths()[0]]
        e.close()
        want = want or got
        for a, b in zip(got, want):
            assert np.array_equal(a, b), nrep


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [10, 54])
def test_action_difference_in_any_batch(pimc, n, precision):
    # An entry's value does not depend on how many entries there are, bit for bit.
    kw = W.heg54(n=n, nslice=512, nlevel=4)
    tabs, ew = pimc.coulomb_tables(kw)
    e = pimc.Engine(kw, 1, tabs, ew, precision=precision)
    rng = np.random.default_rng(n)
    nb = 300
    sec = rng.uniform(-0.5, 0.5, size=(nb, 17, n, 3)) * kw["cell"]
    ip = rng.integers(0, n, nb).astype(np.int32)
    mov = sec[np.arange(nb), :, ip].copy()
    mov[:, 1:-1] += 0.3 * rng.normal(size=mov[:, 1:-1].shape)
    for level in (0, 1):
        whole = e.action_difference(level, sec, mov, ip)
        for b in (1, 3, 17, 40, 120):
            assert np.array_equal(e.action_difference(level, sec[:b], mov[:b], ip[:b]), whole[:b]), b


@pytest.mark.parametrize("n", [10, 14, 22, 30])
def test_update_groups_of_few_and_many_replicas(pimc, n):
    # Mixed form, free-particle nodes: whether a matrix is updated or factorised does not
    # depend on how full the launch is, so neither does a replica's chain, bit for bit.
    # (a short ring: entries reach their last update at different times)
    kw = W.heg54(n=n, nslice=32, nlevel=3, t_over_tf=3.0, coulomb=0, ewald=0)
    x = W.initial_path(dict(kw), "grid", seed=1)
    # (the updates' rounding shows in few of the FP32 nodal terms)
    few = pimc.Engine(kw, 150, seed=9, precision=1)
    many = pimc.Engine(kw, 700, seed=9, precision=1)
    few.upload_paths([x] * 150)
    many.upload_paths([x] * 700)
    for _ in range(4):
        a, b = few.run_sections(100, records=True), many.run_sections(100, records=True)
        for k in a:
            assert np.array_equal(a[k], b[k][:150], equal_nan=True), k
    for p, q in zip(few.download_paths(), many.download_paths()):
        assert np.array_equal(p, q)


MIXED_DISPLACED = {
    "heg10": (W.heg54(n=10, nslice=32, nlevel=3, t_over_tf=3.0), "grid"),
    "heg26_free": (W.heg54(n=26, nslice=64, nlevel=3, t_over_tf=1.5, coulomb=0, ewald=0), "grid"),
    "heg16_one_species": (dict(W.heg54(n=16, nslice=32, nlevel=3, t_over_tf=1.5),
                               node_kind=[2, 0]), "grid"),
    "dot8_fn": (W.dot20_fn(counts=[5, 3], nslice=32, beta=1.6, nlevel=3, node_temperature=0.5),
                "const"),
}


@pytest.mark.parametrize("nmoving", [1, 2])
@pytest.mark.parametrize("nrep", [1, 40, 170])
@pytest.mark.parametrize("case", list(MIXED_DISPLACED))
def test_mixed_displacements_then_sections(pimc, case, nrep, nmoving):
    # Mixed form: after sections (whose matrices were updated) and displacements, the
    # cached elements, determinants, distances, inverses and structure factors are those
    # of the paths: the sections that follow are those of an engine that starts from
    # them.  (The bars of the mixed form against FP64, as inverses here have been
    # updated and there are fresh.)
    kw, kind = MIXED_DISPLACED[case]
    tabs, ew = pimc.coulomb_tables(kw) if kw["coulomb"] else ((), None)
    x = W.initial_path(dict(kw), kind, seed=7)
    a = pimc.Engine(kw, nrep, tabs, ew, seed=99, precision=1)
    a.upload_paths([x] * nrep)
    displaced = 0
    for _ in range(4):
        a.run_sections(25)
        displaced += a.run_displace(6, [0.6] * 3, nmoving, -1, records=True)["accepted"].sum()
        b = pimc.Engine(kw, nrep, tabs, ew, seed=99, precision=1)
        b.upload_paths(a.download_paths())
        for r in range(nrep):
            b.set_replica_state(r, a.replica_state(r))
        if ew is not None:
            assert np.array_equal(a.thermo_energy(), b.thermo_energy())
        ra, rb = a.run_sections(20, records=True), b.run_sections(20, records=True)
        b.close()
        alike = np.cumprod((ra["reject_level"] == rb["reject_level"]) & (ra["ipart"] == rb["ipart"]),
                           axis=1).astype(bool)
        assert alike.mean() > 0.95
        nl = kw["nlevel"] + 1
        for k in ("ds", "ds_node", "lnt"):
            p, q = ra[k][alike][:, :nl], rb[k][alike][:, :nl]
            assert np.array_equal(np.abs(p) >= 1e99, np.abs(q) >= 1e99)
            fin = np.abs(q) < 1e99
            tol = 1e-12 if k != "ds_node" else 1e-4
            assert np.all(np.abs(p - q)[fin] <= tol * np.maximum(np.abs(q[fin]), 1.0)), k
    assert displaced > 0


def test_virial_energy_beside_a_large_system(pimc):
    # A replica's value does not depend on the systems beside it (700 particles take fewer
    # warps than five), bit for bit.
    small = W.dot2(counts=[3, 2], nslice=6400, nlevel=1, beta=256.0)
    large = W.dot2(counts=[350, 350], nslice=16, nlevel=1, beta=0.64)
    tabs, _ = pimc.coulomb_tables(small)
    x = [W.initial_path(dict(small), "gauss", seed=r) for r in range(12)]
    y = W.initial_path(dict(large), "gauss", seed=3)
    alone = pimc.Engine(small, 12, tabs)
    alone.upload_paths(x)
    both = pimc.Engine.batch([small] * 12 + [large], [tabs] * 13)
    both.upload_paths(x + [y])
    for w in (1, 16):
        assert np.array_equal(alone.virial_energy(w), both.virial_energy(w)[:12])
    port = O.PortOracle(O.make_config(**large), tabs)
    port.set_path(y)
    ref = port.virial_energy(4)
    scale = max(1.0, abs(ref), abs(port.virial_energy(1)))
    assert abs(both.virial_energy(4)[12] - ref) <= 1e-11 * scale

"""Displacements on clusters of CTAs: what orders the CTAs' accesses to one another's
shared memory, and launches in close succession."""
import os
import re

import numpy as np
import pytest

import workloads as W

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pi-qmc_gb300",
                    "csrc")


def _kernels():
    """(file, name, body) of every __global__ function of the engine's sources."""
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        for m in re.finditer(r"__global__[^;{]*?(\w+)\(\w+ \w+\) \{\n(.*?)\n\}\n", text, re.S):
            yield f, m.group(1), re.sub(r"//[^\n]*", "", m.group(2))


def test_clusters_start_before_remote_access():
    # A CTA's shared memory may be accessed by another one only once the CTA has
    # started, which a barrier of the cluster guarantees and nothing else does.
    remote = [(f, name, body) for f, name, body in _kernels() if "map_shared_rank" in body]
    assert "displace_kernel" in [name for _, name, _ in remote]
    for f, name, body in remote:
        first = body.index("map_shared_rank")
        assert ".sync()" in body[:first], (f, name)


def test_tables_and_scratch_share_memory_in_turn():
    # The warps' Ewald tables and their Slater scratch are the same shared memory, split
    # at different strides: a barrier lies between the two uses, in either order.
    body = next(b for _, name, b in _kernels() if name == "displace_kernel")
    uses = [(m.start(), m.group(1)) for m in re.finditer(r"\b(displace_ewald|displace_nodes)\(", body)]
    assert [u for _, u in uses] == ["displace_ewald", "displace_nodes", "displace_nodes",
                                    "displace_ewald"]
    loop = uses + [(uses[0][0] + len(body), uses[0][1])]  # (and round to the next attempt)
    for (a, first), (b, second) in zip(loop, loop[1:]):
        if first != second:
            assert re.search(r"__syncthreads\(\)|cl\.sync\(\)", (body + body)[a:b]), (first, second)


@pytest.mark.gpu
@pytest.mark.parametrize("nrep,nmoving", [(1, 1), (21, 3), (320, 3)])
def test_warps_at_different_speeds(nrep, nmoving):
    # A short path leaves some warps without Ewald terms, which come to the Slater matrices
    # before the others: many attempts against the restatement.
    import oracle_lib as O
    import pimc_gb300 as pimc
    pimc.build.build()
    kw = W.heg54(n=8, nslice=198, nlevel=5, beta=7.92, cell=15.0, node_temperature=0.2,
                 ewald_kcut=3 * 2 * np.pi / 15.0)
    tabs, ew = pimc.coulomb_tables(kw)
    x = W.initial_path(dict(kw), "grid", seed=7)
    e = pimc.Engine(kw, nrep, tabs, ew, seed=99)
    e.upload_paths([x] * nrep)
    d = e.run_displace(20, [0.7] * 3, nmoving, -1, records=True)
    for r in {0, nrep - 1}:
        port = O.PortOracle(O.make_config(**dict(kw, seed=99, replica=r)), tabs, ew)
        port.set_path(x)
        ref = port.run_displace(20, [0.7] * 3, nmoving, -1)
        assert np.array_equal(d["accepted"][r], ref["accepted"])
        for k, tol in (("ds", 1e-11), ("ds_node", 1e-9)):
            assert np.all(np.abs(d[k][r] - ref[k]) <= tol * np.maximum(np.abs(ref[k]), 1.0)), k


@pytest.mark.gpu
@pytest.mark.parametrize("nrep", [1, 21, 60, 170])
def test_many_short_launches(nrep):
    # Every launch starts its clusters anew: 60 calls of one attempt are one call of 60.
    import pimc_gb300 as pimc
    pimc.build.build()
    kw = W.dot20_fn(counts=[3, 2], nslice=40, beta=2.0, nlevel=2, node_temperature=0.5)
    tabs, _ = pimc.coulomb_tables(kw)
    x = W.initial_path(dict(kw), "const", seed=7)
    a, b = (pimc.Engine(kw, nrep, tabs, seed=99) for _ in range(2))
    for e in (a, b):
        e.upload_paths([x] * nrep)
    one = a.run_displace(60, [1.2, 1.2, 1.2], 1, -1, records=True)
    parts = [b.run_displace(1, [1.2, 1.2, 1.2], 1, -1, records=True) for _ in range(60)]
    for k in one:
        assert np.array_equal(one[k], np.concatenate([p[k] for p in parts], axis=1)), k
    assert np.array_equal(a.download_paths(flat=True), b.download_paths(flat=True))


@pytest.mark.gpu
@pytest.mark.parametrize("nrep", [1, 40, 320])
@pytest.mark.parametrize("counts", [[5, 3], [13, 4], [2, 9, 4]])
def test_moves_in_species_of_different_size(counts, nrep):
    # Moved particles in several node species, whose matrices a warp takes one species
    # after the other without waiting for the other warps: against the restatement.
    import oracle_lib as O
    import pimc_gb300 as pimc
    pimc.build.build()
    ns = len(counts)
    kw = W.dot20_fn(counts=counts, nslice=128, beta=5.0, nlevel=3, node_temperature=0.5,
                    node_kind=[1] * ns, node_omega=[1.0] * ns, sho_omega=[1.0] * ns)
    tabs, _ = pimc.coulomb_tables(kw)
    x = W.initial_path(dict(kw), "const", seed=7)
    e = pimc.Engine(kw, nrep, tabs, seed=99)
    e.upload_paths([x] * nrep)
    d = e.run_displace(25, [0.6] * 3, 4, -1, records=True)
    for r in {0, nrep - 1}:
        port = O.PortOracle(O.make_config(**dict(kw, seed=99, replica=r)), tabs)
        port.set_path(x)
        ref = port.run_displace(25, [0.6] * 3, 4, -1)
        assert np.array_equal(d["accepted"][r], ref["accepted"])
        for k, tol in (("ds", 1e-11), ("ds_node", 1e-8)):
            assert np.all(np.abs(d[k][r] - ref[k]) <= tol * np.maximum(np.abs(ref[k]), 1.0)), k

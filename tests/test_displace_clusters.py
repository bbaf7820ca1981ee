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

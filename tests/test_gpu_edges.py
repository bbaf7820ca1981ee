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

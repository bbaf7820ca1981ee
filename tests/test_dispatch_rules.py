"""Rules that share out the work of a launch, on the host: who works, and on what."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "pi-qmc_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "kernels.cuh"
using namespace pimc;
int main() {
  for (int mixed = 0; mixed < 2; ++mixed)
    for (int nwarps = 1; nwarps <= 16; nwarps *= 2)
      for (int lanes = 0; lanes <= 32 * 40; lanes += 8)
        std::printf("action %d %d %d %d\n", mixed, nwarps, lanes,
                    first_action_warp(lanes, nwarps, mixed));
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    import pimc_gb300.build as B
    try:
        nvcc = B.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("rules")
    src, exe = d / "rules.cu", d / "rules"
    src.write_text(PROGRAM)
    subprocess.run([nvcc, *B.ARCH, "-std=c++17", "-O0", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return [line.split() for line in out.splitlines()]


def test_action_warps(rules):
    # The action terms' warps: every one where no Slater matrix is to be evaluated, else
    # those that the matrices leave, or all of them where those take over half.
    seen = set()
    for _, mixed, nwarps, lanes, a0 in (r for r in rules if r[0] == "action"):
        mixed, nwarps, lanes, a0 = int(mixed), int(nwarps), int(lanes), int(a0)
        busy = -(-lanes // 32)
        assert 0 <= a0 < nwarps
        if lanes == 0 or 2 * busy > nwarps:
            assert a0 == 0
        else:
            assert a0 >= busy
        seen.add((mixed, a0 > 0))
    assert len(seen) == 4

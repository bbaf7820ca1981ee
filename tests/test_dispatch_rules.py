"""Rules that share out the work of a launch, on the host: who works, and on what."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "pi-qmc_gb300", "csrc")

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "kernels.cuh"
using namespace pimc;
int main() {
  for (int mixed = 0; mixed < 2; ++mixed)
    for (int nwarps = 1; nwarps <= 16; nwarps *= 2)
      for (int lanes = 0; lanes <= 32 * 40; lanes += 8)
        std::printf("action %d %d %d %d\n", mixed, nwarps, lanes,
                    first_action_warp(lanes, nwarps, mixed));
  for (int sho : {0, 1, 16, 17, 32})
    for (int nrep : {1, 152, 153, 280, 300, 304, 305, 607, 608, 5000})
      for (int alike = 0; alike < 2; ++alike)
        std::printf("ctas %d %d %d %d\n", sho, nrep, alike,
                    prefers_two_ctas(nrep, 152, sho, alike));
  for (int nwarps = 1; nwarps <= 8; nwarps *= 2)
    for (int nshare = nwarps; nshare <= 2 * nwarps; nshare *= 2)
      for (int mixed = 0; mixed < 2; ++mixed)
        for (int lanes = 0; lanes <= 32 * 20; lanes += 8)
          std::printf("shares %d %d %d %d %d\n", nwarps, nshare,
                      nshare - first_action_warp(lanes, nshare, mixed),
                      nwarps - first_action_warp(lanes, nwarps, mixed),
                      action_shares_per_warp(nwarps, nshare));
  static DevSys s;  // (no node models, no Ewald sums, no delayed rejection)
  for (int kind : {PIMC_NODES_SHO, PIMC_NODES_FREE})
    for (int mixed = 0; mixed < 2; ++mixed)
      for (int n = 1; n <= 32; ++n)
        for (int wmin = 8; wmin <= 32; wmin *= 2) {
          s.node_kind[0] = kind;
          s.mixed = mixed;
          s.spec_count[0] = n;
          std::printf("width %d %d %d %d %d\n", kind == PIMC_NODES_FREE, mixed, n, wmin,
                      node_launch_width(s, 0, wmin));
        }
  s = DevSys();
  for (s.nlevel = 1; s.nlevel <= 6; ++s.nlevel)
    for (s.npart = 1; s.npart <= 200; ++s.npart)
      for (int mixed = 0; mixed < 2; ++mixed) {
        const int low = lowest_joint_level(s.nlevel, s.npart);
        int need = action_seps(0, s.nlevel - low);
        for (int l = low - 1; l >= 0; --l)
          need = std::max(need, action_seps(s.nlevel - l, s.nlevel - l));
        std::printf("levels %d %d %d %d %d\n", s.nlevel, s.npart, low, (mixed ? 2 : 4) * need,
                    action_buffer(s.nlevel, takes_single_levels(s), mixed));
      }
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


def test_joint_levels(rules):
    # Levels whose links fill more than a warp wait for the decisions above them in long
    # sections, and the buffers hold every evaluation that is made.
    for level, npart, low, need, room in (map(int, r[1:]) for r in rules if r[0] == "levels"):
        assert 0 <= low < level and need <= room
        assert low == 0 if level < 5 else level - low <= 5
        if level == 6 or (level == 5 and npart > 32):
            assert level - low == 4


def test_action_shares(rules):
    # The shares of a larger block's action terms all have a warp and a place in its buffer.
    for nwarps, nshare, shares, workers, most in (map(int, r[1:]) for r in rules
                                                  if r[0] == "shares"):
        assert 1 <= workers <= nwarps and 1 <= shares <= nshare
        assert -(-shares // workers) <= most
        assert nshare > nwarps or (shares == workers and most == 1)


def test_lane_group_widths(rules):
    # The groups that update matrices together are the same in every launch; the others
    # may be wider in a launch that asks for it.
    wider = 0
    for free, mixed, n, wmin, w in (map(int, r[1:]) for r in rules if r[0] == "width"):
        own = 8 if n <= 8 else 16 if n <= 16 else 32
        assert w >= own and w in (8, 16, 32)
        if free and mixed:
            assert w == own
        else:
            assert w <= max(own, wmin)
            wider += w > own
    assert wider


def test_two_ctas(rules):
    # Half as many warps a replica: with SHO nodes only where replicas are many and their
    # matrices share warps, with free-particle nodes wherever replicas wait for SMs.
    for sho, nrep, alike, two in (map(int, r[1:]) for r in rules if r[0] == "ctas"):
        many = nrep >= 608 or (alike and nrep in (300, 304))
        assert two == (many and sho <= 16 if sho else nrep > 152)

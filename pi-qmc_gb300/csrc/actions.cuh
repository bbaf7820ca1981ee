// The action differences of a bisection move: CompositeAction::getActionDifference
// for one moving particle (src/action/CompositeAction.cc:30-37) with SpringAction
// (src/action/SpringAction.cc:56-98), SHOAction (src/action/SHOAction.cc:19-65),
// PrimSHOAction (src/action/PrimSHOAction.cc:21-58) and PairAction per species pair
// (src/action/PairAction.cc:219-360), at one level or at all of them together.
//
// An FP64 warp instruction costs the SM 19 clocks whatever its active lanes, and
// the upper levels have one, two, four ... links, so the links of all levels
// share the lanes of a warp.  Slot n >= 1 of a binary heap is a link: its depth
// d = floor(log2 n) is level nlevel - d, its place n - 2^d there the link's number;
// the lanes' sums then split by depth with a few shuffles.  A warp takes one
// partner particle (several, where a level set is narrower than a warp): first
// the separations of the partner from the old path and the new beads, one lane per
// slice (2^(d+1) lanes' worth in all; every level's links use the same ones), then
// the links.  Level by level, every link formed its own four separations, on as
// many lanes as the level had links: 31 links of a two-electron dot took five
// passes of about 190 FP64 instructions, now one of 150 on full lanes.  With the
// movers' share of the same (mover_all) a step of 9728 such dots (32 attempts) went
// from 53.2 to 24.1 ms, of 304 fixed-node dots (N = 20, 640 attempts) from 191 to
// 159 ms.
#pragma once
#include <type_traits>

#include "section_kernel.cuh"

namespace pimc {

// The per-lane sum of one kind of term: FP64, or the mixed form's compensated FP32.
template <bool kMixed>
struct LaneSum {
  double v = 0.0;
  __device__ __forceinline__ void add(double t) { v += t; }
  __device__ __forceinline__ double value() const { return v; }
};
template <>
struct LaneSum<true> : FSum {};

// Separation of a partner from the moving particle at one slice, and its length.
struct Sep {
  double x, y, z, r;
};
struct SepF {
  float x, y, z, r;
};

// The number of (table, partner) combinations of a moving particle, and the p-th
// of them: its particle, its table in ti.
__device__ __forceinline__ int pair_partners(const DevSys& s, int ipart) {
  int n = 0;
  if (s.coulomb)
#pragma unroll 1
    for (int k = 0; k < s.ntab; ++k) {
      const DevTable& t = s.tab[k];
      if (ipart >= t.ifirst1 && ipart < t.ifirst1 + t.npart1)
        n += t.npart2;
      else if (ipart >= t.ifirst2 && ipart < t.ifirst2 + t.npart2)
        n += t.npart1;
    }
  return n;
}
__device__ __forceinline__ int pair_partner(const DevSys& s, int ipart, int p, int& ti) {
  ti = 0;
#pragma unroll 1
  for (int k = 0; k < s.ntab; ++k) {
    const DevTable& t = s.tab[k];
    int first, n;
    if (ipart >= t.ifirst1 && ipart < t.ifirst1 + t.npart1) {
      first = t.ifirst2;
      n = t.npart2;
    } else if (ipart >= t.ifirst2 && ipart < t.ifirst2 + t.npart2) {
      first = t.ifirst1;
      n = t.npart1;
    } else {
      continue;
    }
    if (p < n) {
      ti = k;
      return first + p;
    }
    p -= n;
  }
  return -1;
}

// Spring, harmonic and primitive terms (new - old) of the link that ends at slice
// t1 and starts at t0, at its level; the last link of a level has no PrimSHO term.
template <bool kMixed>
__device__ __forceinline__ void link_terms(const DevSys& s, const Smem& m, int ipart, int sp,
                                           int level, int t0, int t1, bool last,
                                           LaneSum<kMixed>& acc) {
  const int np = s.npart;
  const double n1x = m.mx[t1], n1y = m.my[t1], n1z = m.mz[t1];
  const double n0x = m.mx[t0], n0y = m.my[t0], n0z = m.mz[t0];
  const double o1x = m.s1x[t1 * np + ipart], o1y = m.s1y[t1 * np + ipart], o1z = m.s1z[t1 * np + ipart];
  const double o0x = m.s1x[t0 * np + ipart], o0y = m.s1y[t0 * np + ipart], o0z = m.s1z[t0 * np + ipart];
  const bool prim = (s.prim_a[sp] != 0 || s.prim_b[sp] != 0) && !last;
  if constexpr (kMixed) {
    // FP32 terms in which nothing cancels: spring (|d_new|^2 - |d_old|^2) / (4 lambda tau'),
    // the harmonic link action minus its free part as a (|d_new|^2 - |d_old|^2) +
    // b (r0.r1_new - r0.r1_old) (sho_a, sho_b), PrimSHO (a x^2 + b x^4) tau'
    if (s.spring) {
      float fx, fy, fz, gx, gy, gz;
      pbc_f(s, n1x - n0x, n1y - n0y, n1z - n0z, fx, fy, fz);
      pbc_f(s, o1x - o0x, o1y - o0y, o1z - o0z, gx, gy, gz);
      acc.add((float)s.spr_inv2s2[level][sp] * (norm2_move_f(fx, fy, fz) - norm2_move_f(gx, gy, gz)));
    }
    if (s.sho_omega[sp] > 0) {
      const float a0x = f32_rn(n0x), a0y = f32_rn(n0y), a0z = f32_rn(n0z);
      const float a1x = f32_rn(n1x), a1y = f32_rn(n1y), a1z = f32_rn(n1z);
      const float b0x = f32_rn(o0x), b0y = f32_rn(o0y), b0z = f32_rn(o0z);
      const float b1x = f32_rn(o1x), b1y = f32_rn(o1y), b1z = f32_rn(o1z);
      const float dnx = f32_rn(n1x - n0x), dny = f32_rn(n1y - n0y), dnz = f32_rn(n1z - n0z);
      const float dox = f32_rn(o1x - o0x), doy = f32_rn(o1y - o0y), doz = f32_rn(o1z - o0z);
      const float dd = norm2_move_f(dnx, dny, dnz) - norm2_move_f(dox, doy, doz);
      const float rr = dot_f(a0x, a0y, a0z, a1x, a1y, a1z) - dot_f(b0x, b0y, b0z, b1x, b1y, b1z);
      acc.add(__fmaf_rn(s.sho_b[level][sp], rr, __fmul_rn(s.sho_a[level][sp], dd)));
    }
    if (prim) {
      float xn, yn, zn, xo, yo, zo;
      pbc_f(s, n1x, n1y, n1z, xn, yn, zn);
      pbc_f(s, o1x, o1y, o1z, xo, yo, zo);
      const float pa = (float)s.prim_a[sp], pb = (float)s.prim_b[sp];
      const float r2n = norm2_move_f(xn, yn, zn), r2o = norm2_move_f(xo, yo, zo);
      const float d2 = r2n - r2o, d4 = __fmaf_rn(r2n, r2n, -__fmul_rn(r2o, r2o));
      acc.add(__fmaf_rn(pa, d2, __fmul_rn(pb, d4)) * (float)(s.tau * (1 << level)));
    }
  } else {
    // (the plain differences' squares serve the harmonic term and, but for an image,
    // the spring)
    const double dx = n1x - n0x, dy = n1y - n0y, dz = n1z - n0z;
    const double ex = o1x - o0x, ey = o1y - o0y, ez = o1z - o0z;
    const double dn = dx * dx + dy * dy + dz * dz, dold = ex * ex + ey * ey + ez * ez;
    if (s.spring) {
      double fx = dx, fy = dy, fz = dz, gx = ex, gy = ey, gz = ez, d2 = dn - dold;
      if (pbc(s, fx, fy, fz) | pbc(s, gx, gy, gz))
        d2 = (fx * fx + fy * fy + fz * fz) - (gx * gx + gy * gy + gz * gz);
      acc.add(s.spr_inv2s2[level][sp] * d2);
    }
    const double om = s.sho_omega[sp];
    if (om > 0) {
      const double coshwt = s.sho_cosh[level][sp], div1 = s.sho_div1[level][sp];
      const double div2 = s.sho_div2[level], msho = s.mass[sp];
      double r0r0 = n0x * n0x + n0y * n0y + n0z * n0z;
      double r1r1 = n1x * n1x + n1y * n1y + n1z * n1z;
      double r0r1 = n0x * n1x + n0y * n1y + n0z * n1z;
      const double nw = msho * om * ((r1r1 + r0r0) * coshwt - 2.0 * r0r1) * div1 - msho * dn * div2;
      r0r0 = o0x * o0x + o0y * o0y + o0z * o0z;
      r1r1 = o1x * o1x + o1y * o1y + o1z * o1z;
      r0r1 = o0x * o1x + o0y * o1y + o0z * o1z;
      const double od = msho * om * ((r1r1 + r0r0) * coshwt - 2.0 * r0r1) * div1 - msho * dold * div2;
      acc.add(nw - od);
    }
    if (prim) {
      double x = n1x, y = n1y, z = n1z;
      pbc(s, x, y, z);
      double x2 = x * x + y * y + z * z;
        const double kt = s.tau * pow2(level);
      const double nw = (s.prim_a[sp] * x2 + s.prim_b[sp] * x2 * x2) * kt;
      x = o1x;
      y = o1y;
      z = o1z;
      pbc(s, x, y, z);
      x2 = x * x + y * y + z * z;
      acc.add(nw - (s.prim_a[sp] * x2 + s.prim_b[sp] * x2 * x2) * kt);
    }
  }
}

// PairAction of one link from its two separations, times its length in slices (2^shift).
__device__ __forceinline__ double pair_term(const DevTable& t, const Sep& a, const Sep& b,
                                            bool offdiag, int shift) {
  const double qq = 0.5 * (a.r + b.r);
  if (!offdiag) return tab_u00(t, qq) * pow2(shift);
  const double sx = a.x - b.x, sy = a.y - b.y, sz = a.z - b.z;
  const double qi = reciprocal(qq);
  return tab_uk0(t, qq, dot3(sx, sy, sz, sx, sy, sz) * (qi * qi)) * pow2(shift);
}
__device__ __forceinline__ float pair_term(const DevTable& t, const SepF& a, const SepF& b,
                                           bool offdiag, int shift) {
  const float qq = 0.5f * (a.r + b.r);
  const float s2 =
      offdiag ? __fdividef(norm2_move_f(a.x - b.x, a.y - b.y, a.z - b.z), __fmul_rn(qq, qq)) : 0.f;
  return tab_uk0_f(t, qq, s2, offdiag ? t.norder : 0) * __uint_as_float((127u + shift) << 23);
}

// Separations a warp holds at once (levels dmin .. dmax of the heap, below).
__host__ __device__ __forceinline__ int action_seps(int dmin, int dmax) {
  const int nl = dmin ? 1 << dmax : 2 << dmax;
  return (nl < 32 ? 32 / nl : 1) * (2 << dmax);
}
// Doubles of a share's lane sums, and of a warp's separations.
__host__ __device__ __forceinline__ int action_sum_words(int nlevel) {
  return 32 * (nlevel >= 6 ? 3 : (nlevel >= 5 ? 2 : 1));
}
__host__ __device__ __forceinline__ int action_sep_words(int nlevel, bool single_levels, bool mixed) {
  int e = action_seps(0, nlevel);
  if (single_levels && e < 64) e = 64;
  return mixed ? 2 * e : 4 * e;
}
// Doubles of a warp's work buffer: its separations, then its lanes' sums over them; or
// the sums of several shares after them.
__host__ __device__ __forceinline__ int action_buffer(int nlevel, bool single_levels, bool mixed,
                                                      int shares = 1) {
  const int seps = action_sep_words(nlevel, single_levels, mixed), sums = action_sum_words(nlevel);
  return shares > 1 ? seps + shares * sums : (seps > sums ? seps : sums);
}

// The lowest level that is evaluated with those above it where an attempt has neither
// Slater matrices nor Ewald sums: all together while their links fit a warp's lanes.  The
// 32 and 64 links of the lowest levels of longer sections wait for the decisions above
// them, which few attempts pass (32 attempts of 304 dots of 10 electrons, L = 6, 1 %
// accepted: 2740 us together, 1270 so; of 100 electrons, L = 5, 14 % accepted: 6300
// and 4280); but for up to 32 particles at L = 5, where they cost little and many
// pass (152 dots of two, 60 % accepted: 734 us together, 811 apart).
__host__ __device__ __forceinline__ int lowest_joint_level(int nlevel, int npart) {
  return nlevel > 5 || (nlevel == 5 && npart > 32) ? nlevel - 4 : 0;
}
// Whether a system takes levels singly (the size of its action buffers).
__host__ __device__ __forceinline__ bool takes_single_levels(const DevSys& s) {
  return s.fixed_node || s.dr || s.ewald || lowest_joint_level(s.nlevel, s.npart) > 0;
}

// The first of a CTA's warps that take action terms beside the Slater matrices of
// `lanes` lanes: the others, or half of them in the mixed form, whose terms are cheap;
// every warp, after its matrices, where those take more than half of the warps, and where
// there are none (half of the warps left without work: a step of 152 mixed dots of 40
// electrons without nodes, L = 4, 32 attempts: 1148 us, 862 with all).
__host__ __device__ __forceinline__ int first_action_warp(int lanes, int nwarps, bool mixed) {
  const int busy = (lanes + 31) / 32;
  return lanes == 0 || 2 * busy > nwarps ? 0 : (mixed ? nwarps / 2 : busy);
}

// The most shares of nshare warps' action terms that one of nwarps warps takes.
__host__ __device__ __forceinline__ int action_shares_per_warp(int nwarps, int nshare) {
  int most = 1;
  for (int busy = 0; nwarps < nshare && busy <= nshare; ++busy)
    for (int mixed = 0; mixed < 2; ++mixed) {
      const int n = nshare - first_action_warp(32 * busy, nshare, mixed);
      const int w = nwarps - first_action_warp(32 * busy, nwarps, mixed);
      if ((n + w - 1) / w > most) most = (n + w - 1) / w;
    }
  return most;
}

// Share w of the nw of the work: the terms of heap depths 0 .. dmax (dmin = 0) or of
// depth dmax alone (dmin = dmax), on the calling warp with its buffer.  The lanes'
// sums go to sums (the buffer itself, or beyond its separations):
// [0] slots 0 .. 31, or the one depth's; [32] depth 5; [64] depth 6.
template <bool kMixed>
static __device__ __noinline__ void action_warp(const DevSys& s, const Smem& m, int ipart,
                                                int dmin, int dmax, int w, int nw, double* buf,
                                                double* sums) {
  using S = typename std::conditional<kMixed, SepF, Sep>::type;
  const int lane = threadIdx.x & 31, L = s.nlevel, np = s.npart;
  const int sh = L - dmax, nI = 2 << dmax, mid = 1 << dmax;
  const int nl = dmin ? mid : nI, base = dmin ? mid : 0;
  LaneSum<kMixed> a0, a1, a2;
  auto add = [&](int it, auto term) {
    if (dmin || it == 0)
      a0.add(term);
    else if (it == 1)
      a1.add(term);
    else
      a2.add(term);
  };
  const int total = pair_partners(s, ipart);
  const int P = nl < 32 ? 32 / nl : 1;  // partners a warp takes at once
  S* sep = (S*)buf;
#pragma unroll 1
  for (int pc = w; pc * P < total; pc += nw) {
    __syncwarp();
    // the partners' separations: entry i <= mid the old path at slice i << sh, entry
    // mid + i the new bead there (the end slices do not move)
#pragma unroll 1
    for (int e = lane; e < P * nI; e += 32) {
      const int g = e >> (dmax + 1), i = e & (nI - 1);
      int ti;
      const int j = pc * P + g < total ? pair_partner(s, ipart, pc * P + g, ti) : -1;
      if (j < 0 || j == ipart) continue;
      const bool moved = i > mid;
      const int t = (moved ? i - mid : i) << sh;
      const double ax = moved ? m.mx[t] : m.s1x[t * np + ipart];
      const double ay = moved ? m.my[t] : m.s1y[t * np + ipart];
      const double az = moved ? m.mz[t] : m.s1z[t * np + ipart];
      double dx = ax - m.s1x[t * np + j], dy = ay - m.s1y[t * np + j], dz = az - m.s1z[t * np + j];
      if constexpr (kMixed) {
        float fx, fy, fz;
        pbc_f(s, dx, dy, dz, fx, fy, fz);
        sep[e] = SepF{fx, fy, fz, sqrtf(norm2_move_f(fx, fy, fz))};
      } else {
        pbc(s, dx, dy, dz);
        sep[e] = Sep{dx, dy, dz, square_root(dot3(dx, dy, dz, dx, dy, dz))};
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int it = 0; it * 32 < P * nl; ++it) {
      const int li = it * 32 + lane, g = nl < 32 ? li / nl : 0, slot = base + li - g * nl;
      int ti;
      const int j = pc * P + g < total ? pair_partner(s, ipart, pc * P + g, ti) : -1;
      if (j < 0 || j == ipart || slot == 0) continue;
      const int d = 31 - __clz(slot), k = slot - (1 << d);
      const int i0 = k << (dmax - d), i1 = (k + 1) << (dmax - d);
      const DevTable& t = s.tab[ti];
      const bool offdiag = L - d < 3 && t.norder > 0;
      const S* sg = sep + g * nI;
      const S& b1 = sg[i1];
      const S& b0 = sg[i0];
      const S& n1 = sg[i1 == mid ? i1 : mid + i1];
      const S& n0 = sg[i0 == 0 ? 0 : mid + i0];
      decltype(pair_term(t, n1, n0, offdiag, 1)) v[2];
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {  // (one copy of the lookup's code)
        const auto x = pair_term(t, pass ? b1 : n1, pass ? b0 : n0, offdiag, L - d);
        v[1] = pass ? x : v[1];
        v[0] = pass ? v[0] : x;
      }
      add(P > 1 ? 0 : it, v[0] - v[1]);
    }
  }
  // the links' own terms, on the warp after the last one with a partner
  if (w == ((total + P - 1) / P) % nw) {
    const int sp = species_of(s, ipart);
#pragma unroll 1
    for (int it = 0; it * 32 < nl; ++it) {
      const int li = it * 32 + lane, slot = base + li;
      if (li >= nl || slot == 0) continue;
      const int d = 31 - __clz(slot), k = slot - (1 << d), level = L - d;
      LaneSum<kMixed>& a = (dmin || it == 0) ? a0 : (it == 1 ? a1 : a2);
      link_terms<kMixed>(s, m, ipart, sp, level, k << level, (k + 1) << level, k + 1 == (1 << d), a);
    }
  }
  __syncwarp();
  sums[lane] = a0.value();
  if (!dmin && dmax >= 5) sums[32 + lane] = a1.value();
  if (!dmin && dmax >= 6) sums[64 + lane] = a2.value();
}

// A heap's lane values (slot n of nI <= 32 on every lane congruent to it) folded by
// depth: lane 2^d holds depth d's sum.  Five shuffles for all depths.
__device__ __forceinline__ double fold_by_depth(double x, int nI) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int o = 16; o >= nI; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  const int slot = lane & (nI - 1);
#pragma unroll 1
  for (int o = nI / 4; o > 0; o >>= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, x, o);
    if (slot >= 2 * o) x += y;
  }
  return x;
}
__device__ __forceinline__ double fold_warp(double x) {
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// The action differences of action_warp's nshare shares, per level into lds[level]: share
// k's sums are the k / nw-th (of `words`) from buf0 on in the buffer of the k % nw-th
// of the nw warps.  Called by every warp after a barrier; the first ones work.
__device__ __forceinline__ void action_reduce(const DevSys& s, const double* buf0, int stride,
                                              int dmin, int dmax, int nshare, int nw, int words,
                                              double* lds) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int chunks = (dmin || dmax < 5) ? 1 : dmax - 3;
#pragma unroll 1
  for (int c = warp; c < chunks; c += nwarps) {
    double x = 0.0;
#pragma unroll 1
    for (int k = 0, w = 0, at = 32 * c + lane; k < nshare; ++k) {
      x += buf0[(size_t)w * stride + at];
      if (++w == nw) {
        w = 0;
        at += words;
      }
    }
    if (dmin || c > 0) {
      x = fold_warp(x);
      if (lane == 0) lds[s.nlevel - (dmin ? dmax : 4 + c)] = x;
    } else {
      const int nI = min(32, 2 << dmax);
      x = fold_by_depth(x, nI);
      const int d = 31 - __clz(max(lane, 1));
      if (lane < nI && lane == (1 << d)) lds[s.nlevel - d] = x;
    }
  }
}

}  // namespace pimc

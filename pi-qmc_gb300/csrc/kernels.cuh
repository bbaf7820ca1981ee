// The section-move sampler: shared-memory layout, section staging, mover,
// fixed-node set-up and levels, and the persistent kernel itself.
#pragma once
#include "../../include/pimc_gb300.h"
#include "actions.cuh"

namespace pimc {

// Offsets (in doubles) of the shared-memory working set; computed on the host
// for the largest replica of a launch.
struct Layout {
  int s1, s2, mv, red, q, dm, ndm, dist, ndist, ewt, nodescr, ictl, ecache, ncol;
  int ncol_stride;
  int nrm;  // the attempt's normals, 3 per movable slice
  int old;  // the mover's terms of the old beads
  int act, act_stride, act_global;  // per-warp buffers of the action differences: offset
                                    // (-1: the warps' Slater scratch, or the CTA's global area)
  int nodescr_in_smem;  // the node scratch (its hot parts when split) in shared memory
  int nodescr_stride;   // doubles per warp of that scratch
  int split;            // cold parts apart, in the CTA's global area
  int nodecold_stride;  // doubles per warp of the cold parts
  int cold_follows;     // each group's cold part follows its hot part
  int ncol_global;      // the new-column buffer in the CTA's global area
  int gcta;             // doubles of global scratch per CTA
  int ewt_cols;         // bead columns of the Ewald tables area
  int ewt_words;        // doubles of the tables area
  int ewxy;             // their (kx, ky) products (estimators; 0: none)
  int sums;             // the thermodynamic estimator's sums by part and thread
  int total;  // doubles
};

// Whether systems of which a CTA of eight warps fills an SM run as two CTAs of four, which
// hide each other's barriers and serial parts, but leave a replica half of the warps.
// Free-particle nodes: where there are more replicas than SMs (12 attempts of 48
// electrons, L = 3, mixed: 160 replicas 3.20 -> 2.66 ms, 608 7.46 -> 5.49).  SHO nodes,
// whose matrices keep the warps busy: where the shorter chain of a replica does not
// count, from four replicas an SM on (1024 uneven dots of up to 32 particles 7.73 -> 6.31 ms,
// 608 4.68 -> 4.04, but 456 3.62 -> 3.91 and 240 2.38 -> 3.90), or where replicas of
// one kind fill two CTAs an SM and no more (dots of 32: 304 replicas 5.60 -> 5.17, but
// 240 4.86 -> 5.10 and 360 6.74 -> 7.42); and not for species that take a warp a
// matrix (36 particles, 1000 replicas: 17.9 -> 18.9).
// largest_sho: the largest species with SHO nodes (0: none).
inline bool prefers_two_ctas(int nreplica, int nsm, int largest_sho, bool alike) {
  if (!largest_sho) return nreplica > nsm;
  const bool filled = alike && nreplica <= 2 * nsm && 10 * nreplica >= 19 * nsm;
  return largest_sho <= 16 && (nreplica >= 4 * nsm || filled);
}

struct RunParams {
  const DevSys* sys;
  DevState* state;
  double* paths;
  double* nodecache;  // per-replica Slater-result cache pool (null: none)
  double* nodescr_g;  // global per-warp node scratch when it does not fit in smem
  pimc_move_record* rec;
  const int* order;  // replicas in decreasing cost (longest first)
  int* next;         // work-queue head, zeroed before each launch
  int nattempt;
  const int* nattempt_r;  // per-replica attempts (null: nattempt for every replica)
  long long* ekcache;     // structure-factor cache pool (null: none)
  long long* ekstage;     // per-CTA staging of an attempt's new structure factors
  int ekstage_stride;     // int64 words per CTA
  double* xstage;         // mixed form: per-CTA staging of changed slices' inverses (null: none)
  long long xstage_cta;   // doubles per CTA
  int nrep;
  int wide;  // at most one CTA per SM
  int nshare;  // warps that sums are shared out to, at least the block's
  uint64_t seed;
  Layout lay;
};

__device__ __forceinline__ Smem carve(double* base, const Layout& L, const DevSys& s,
                                      double* nodescr_g, double* xstage = nullptr, bool wide = false,
                                      int nshare = 0) {
  Smem m;
  // mixed form: this CTA's staging of the inverse blocks of an attempt's changed
  // slices ([nsec][2 + ns_max^2], global memory), committed to the cache on accept
  m.xstage = xstage;
  m.xstage_stride = s.ns_max * s.ns_max + 2;
  const int ss = s.nsec * s.npart;
  m.s1x = base + L.s1;
  m.s1y = m.s1x + ss;
  m.s1z = m.s1y + ss;
  m.s2x = base + L.s2;
  m.s2y = m.s2x + ss;
  m.s2z = m.s2y + ss;
  m.mx = base + L.mv;
  m.my = m.mx + s.nsec;
  m.mz = m.my + s.nsec;
  m.red = base + L.red;
  m.old = base + L.old;
  m.qpart = base + L.q;
  m.dm = base + L.dm;
  m.ndm = base + L.ndm;
  m.dist = base + L.dist;
  m.ndist = base + L.ndist;
  m.ewt = base + L.ewt;
  m.ictl = (int*)(base + L.ictl);
  m.ecache = L.ecache >= 0 ? base + L.ecache : nullptr;
  // the CTA's global area: per-warp node scratch (all of it, or the cold parts),
  // then the new-column buffer when it is not in shared memory
  double* gbase = nodescr_g ? nodescr_g + (size_t)blockIdx.x * L.gcta : nullptr;
  const int nw = blockDim.x >> 5;
  const int gwarp = L.split ? L.nodecold_stride : (L.nodescr_in_smem ? 0 : L.nodescr_stride);
  m.ncol = L.ncol >= 0 ? base + L.ncol
                       : ((L.ncol_global && gbase) ? gbase + (size_t)nw * gwarp : nullptr);
  m.nodecold = (L.split && gbase) ? gbase : nullptr;
  m.nodecold_stride = L.nodecold_stride;
  m.node_cold_follows = L.cold_follows;
  m.ewt_cols = L.ewt_cols;
  m.ewxy = L.ewxy ? base + L.ewxy : nullptr;
  m.nrm = base + L.nrm;
  m.ncol_stride = L.ncol_stride;
  m.nodescr_stride = L.nodescr_stride;
  m.nodescr = L.nodescr_in_smem ? base + L.nodescr : gbase;
  m.wide = wide;
  // the level-0 Ewald term's tables: their own area, or the Slater scratch
  m.ewx = m.ewt;
  m.ewx_words = L.ewt_words;
  if (L.nodescr_in_smem && nw * L.nodescr_stride > L.ewt_words) {
    m.ewx = m.nodescr;
    m.ewx_words = nw * L.nodescr_stride;
  }
  m.act = L.act >= 0 ? base + L.act
                     : (L.act_global ? gbase + (L.gcta - nw * L.act_stride) : m.nodescr);
  m.act_stride = L.act_stride;
  m.nshare = nshare ? nshare : nw;
  return m;
}

// Section slice k of a section starting at ifirst, in path slice numbering with
// the identity permutation (SerialPaths::getBeads, src/base/SerialPaths.cc:119-136).
__device__ __forceinline__ int wrap_slice(int islice, int M) {
  return islice < 0 ? islice + M : (islice < M ? islice : islice - M);
}

// The level-0 Ewald term of CoulombAction::getActionDifference
// (src/action/CoulombAction.cc:107-119: evalLongRange of the new minus the old
// configuration on section slices 1 .. 2^L-1, times tau/epsilon) from the
// slices' cached structure factors: only the moving particle's term changes,
// rho'_k = rho_k + q (e^{ik.r'} - e^{ik.r}), exact on the fixed-point grid, and
// evalLongRange's difference is sum_k 2 v_k (|rho'_k|^2 - |rho_k|^2) / (2V)
// (the self energy cancels).  O(totk) per slice instead of O(totk N) for each
// of the two configurations.  rho'_k goes to `stage` for the accept step.
// FP64 bound: 15 instructions and eight conversions per slice and k-vector with the
// products q e^{i(kx x + ky y)} tabulated beside the axes' tables, over the Slater
// scratch, which is free by then (53 without the products, in four passes: N = 54,
// totk = 257, 314,000 -> 158,000 clocks an attempt).
static __device__ __noinline__ double ewald_level0_cached(const DevSys& s, const Smem& m, int ipart,
                                             int ifirst1, const long long* ek, long long* stage) {
  const int np = s.npart, nsec = s.nsec, M = s.nslice, totk = s.totk;
  const int ky0 = s.ikmax[1], kz0 = s.ikmax[2];
  const int nx = s.ikmax[0] + 1, ny = 2 * ky0 + 1, per = nx + ny + 2 * kz0 + 1;
  // columns: a slice's old and new bead.  As many as the area holds of the three axes'
  // tables and their (kx, ky) products (an odd row length against bank conflicts);
  // where that is not one slice, the tables alone.
  int w = m.ewx_words / (2 * (per + nx * ny));
  const bool xy = w >= 3;
  if (!xy) w = m.ewx_words / (2 * per);
  w = w < 3 ? 2 : (min(w, 2 * (nsec - 2) + 1) - 1) | 1;
  const int chunk = w / 2;  // slices per pass
  double2* X = (double2*)m.ewx;
  double2* Y = X + nx * w;
  double2* Z = Y + ny * w;
  double2* XY = X + per * w;
  const double qs = __dmul_rn(m.qpart[ipart], s.ek_scale);  // (exact: a power of two)
  // (a term's place among all slices' decides whose share it is in: the sum does not
  // depend on the passes or on the block)
  const int nthr = 32 * m.nshare;
  double acc[2] = {0.0, 0.0};
#pragma unroll 1
  for (int t0 = 1; t0 < nsec - 1; t0 += chunk) {
    const int nc = 2 * min(chunk, nsec - 1 - t0);
    __syncthreads();
#pragma unroll 1
    for (int it = threadIdx.x; it < 3 * nc; it += blockDim.x) {
      const int a = it / nc, c = it - a * nc, t = t0 + (c >> 1), o = t * np + ipart;
      const double* bead = c & 1 ? (a == 0 ? m.mx : (a == 1 ? m.my : m.mz)) + t
                                 : (a == 0 ? m.s1x : (a == 1 ? m.s1y : m.s1z)) + o;
      ewald_axis_table(s, (a == 0 ? X : (a == 1 ? Y : Z)) + c, w, a, *bead);
    }
    __syncthreads();
    if (xy) {
#pragma unroll 1
      for (int it = threadIdx.x; it < nx * ny * nc; it += blockDim.x) {
        const int p = it / nc, c = it - p * nc, kx = p / ny;
        const double2 a = X[kx * w + c];
        XY[p * w + c] = cmul_rn(make_double2(__dmul_rn(qs, a.x), __dmul_rn(qs, a.y)),
                                Y[(p - kx * ny) * w + c]);
      }
      __syncthreads();
    }
    const int first = (threadIdx.x - (t0 - 1) * totk) & (blockDim.x - 1);
#pragma unroll 1
    for (int it = first; 2 * it < nc * totk; it += blockDim.x) {
      const int tt = it / totk, k = it - tt * totk, t = t0 + tt;
      const longlong2 o =
          *(const longlong2*)(ek + ((size_t)wrap_slice(ifirst1 + t, M) * totk + k) * 2);
      const double vk = __ldg(s.vk + k);
      const int kx = __ldg(s.kvec + 3 * k), ky = __ldg(s.kvec + 3 * k + 1) + ky0,
                kz = __ldg(s.kvec + 3 * k + 2) + kz0;
      longlong2 d = make_longlong2(0, 0);  // new - old
#pragma unroll
      for (int c = 2 * tt; c < 2 * tt + 2; ++c) {
        double2 p;
        if (xy) {
          p = XY[(kx * ny + ky) * w + c];
        } else {
          const double2 a = X[kx * w + c];
          p = cmul_rn(make_double2(__dmul_rn(qs, a.x), __dmul_rn(qs, a.y)), Y[ky * w + c]);
        }
        const double2 v = cmul_rn(p, Z[kz * w + c]);
        d.x = __double2ll_rn(v.x) - d.x;
        d.y = __double2ll_rn(v.y) - d.y;
      }
      const longlong2 n = make_longlong2(o.x + d.x, o.y + d.y);
      *(longlong2*)(stage + ((size_t)(t - 1) * totk + k) * 2) = n;
      // |rho'|^2 - |rho|^2 = (rho' - rho) . (rho' + rho)
      const bool second = ((t0 - 1) * totk + it) & (nthr - 1) & blockDim.x;
      const double a = __fma_rn(vk,
                                __fma_rn(__ll2double_rn(d.x), __ll2double_rn(o.x + n.x),
                                         __dmul_rn(__ll2double_rn(d.y), __ll2double_rn(o.y + n.y))),
                                second ? acc[1] : acc[0]);
      acc[0] = second ? acc[0] : a;
      acc[1] = second ? a : acc[1];
    }
  }
  const double is = 1.0 / s.ek_scale;
  const double sum =
      share_sum(m.nshare, m.red, [&](int h) { return h ? acc[1] : acc[0]; }) * (2 * is * is);
  return sum * s.one_over_2v * s.tau / s.epsilon;
}

static __device__ __noinline__ void load_section(const DevSys& s, const double* path, int ifirst, double* sx,
                             double* sy, double* sz) {
  const int np = s.npart, n = s.nsec * np;
#pragma unroll 1
  for (int i0 = threadIdx.x; i0 < n; i0 += 4 * blockDim.x) {  // (four beads' loads in flight)
    double x[4], y[4], z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = min(i0 + q * (int)blockDim.x, n - 1);
      const int k = idx / np, p = idx - k * np;
      const double* src = path + ((size_t)wrap_slice(ifirst + k, s.nslice) * np + p) * 3;
      x[q] = src[0];
      y[q] = src[1];
      z[q] = src[2];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = i0 + q * blockDim.x;
      if (idx < n) {
        sx[idx] = x[q];
        sy[idx] = y[q];
        sz[idx] = z[q];
      }
    }
  }
}

// SerialPaths::putBeads (src/base/SerialPaths.cc:143-185) with the identity permutation.
static __device__ __noinline__ void store_section(const DevSys& s, double* path, int ifirst, const double* sx,
                              const double* sy, const double* sz) {
  const int np = s.npart, n = s.nsec * np;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < n; idx += blockDim.x) {
    const int k = idx / np, p = idx - k * np;
    const int islice = ifirst + k;
    if (islice < 0) continue;
    const int t = islice < s.nslice ? islice : islice % s.nslice;
    double* dst = path + ((size_t)t * np + p) * 3;
    dst[0] = sx[idx];
    dst[1] = sy[idx];
    dst[2] = sz[idx];
  }
}

// Every normal the attempt's mover can use, drawn in parallel before the
// levels: moved slice `ord` (0 .. 2^L - 2 in FreeMover's order) takes Box-Muller
// pairs 2 ord and 2 ord + 1 and uses the first three values.  Both precision
// forms draw the same FP64 normals, so a mixed-form chain makes the FP64
// chain's proposals and its action differences can be compared with the FP64
// form's on identical moves.
static __device__ __noinline__ void attempt_normals(const DevSys& s, const Smem& m, uint64_t seed,
                                       uint32_t rep, uint32_t att) {
  // (with delayed rejection one more: the second proposal at level nlevel - 1
  // takes order 1, the slices after it one order later)
  // (the second pairs start on a half-warp: up to 16 slices' pairs take one warp)
  const int nord = (1 << s.nlevel) - 1 + (s.dr ? 1 : 0), pad = (nord + 15) & ~15;
#pragma unroll 1
  for (int it = threadIdx.x; it < 2 * pad; it += blockDim.x) {
    const int second = it >= pad, o = it - second * pad;
    if (o >= nord) continue;
    double z0, z1;
    stream_normal_pair(seed, rep, att, 2u * o + second, &z0, &z1);
    if (second) {
      m.nrm[3 * o + 2] = z0;
    } else {
      m.nrm[3 * o] = z0;
      m.nrm[3 * o + 1] = z1;
    }
  }
}

// The uniform-stream index of the first uniform consumed at `level`
// (image choices of FreeMoverPBC, then the Metropolis uniform).
__device__ __forceinline__ uint32_t level_uniform_base(const DevSys& s, int level) {
  uint32_t u = (s.fixed_node ? 2u : 1u) + 1u;  // section choice + particle choice
  const uint32_t pbcu = s.mover == PIMC_MOVER_FREE_PBC ? 3u : 0u;
#pragma unroll 1
  for (int l = s.nlevel; l > level; --l) {
    const uint32_t nmov = (l == s.nlevel) ? 0u : (1u << (s.nlevel - l - 1));
    u += pbcu * nmov + 1u;
  }
  return u;
}

// FreeMoverPBC's image choice of a midpoint offset md (half the separation of the
// neighbouring beads): md or md + L/2 with probabilities w1 = exp(-md^2 / 2 sigma^2)
// against w2.  |md + L/2| >= L/2 - |md|, so when ((L/2 - |md|)^2 - md^2) / 2 sigma^2
// > 40 on every axis w2 is below 2^-57 w1, w1 / (w1 + w2) rounds to 1 (or is 0/0)
// and no uniform exceeds it: the exponentials and uniforms are left out.  That is
// every choice in a box much wider than the level's sigma.
static __device__ __noinline__ void mover_image(const DevSys& s, double md[3], double inv2Sigma2,
                                            uint64_t seed, uint32_t rep, uint32_t att,
                                            uint32_t u0) {
  const float w = (float)inv2Sigma2;
  bool sure = true;
  for (int d = 0; d < 3; ++d) {
    const float c = (float)s.cell[d], a = abs_f32_trunc(md[d]) * 1.000002f;
    sure &= w * (c * (0.25f * c - a)) > 40.f * 1.0001f;
  }
  if (sure) return;
  double m2[3] = {md[0] + 0.5 * s.cell[0], md[1] + 0.5 * s.cell[1], md[2] + 0.5 * s.cell[2]};
  pbc(s, m2[0], m2[1], m2[2]);
  for (int d = 0; d < 3; ++d) {
    // No periodic Gaussian on the mover path (the engine rejects boxes that need one).
    const double w1 = exp(-inv2Sigma2 * md[d] * md[d]);
    const double w2 = exp(-inv2Sigma2 * m2[d] * m2[d]);
    const double u = stream_uniform(seed, rep, att, u0 + d);
    if (u > w1 / (w1 + w2)) md[d] = m2[d];
  }
}

// FreeMover::makeMove (src/advancer/mover/FreeMover.cc:59-124) and
// FreeMoverPBC::makeMove (src/advancer/mover/FreeMoverPBC.cc:59-152) for one moving
// particle at every level.  Moved slices are the nodes of a binary heap: slot n >= 1
// of depth d = floor(log2 n) is moved at level nlevel - 1 - d, and takes normals
// n - 1.  What does not depend on the new beads (the old beads' terms here, the
// proposals' own in mover_all) runs on one lane per slice of every level; only the
// midpoints go level by level.  (Level by level with everything in it, each level
// cost the FP64 pipe the same 55 instructions for its 1, 2, 4 ... slices.)
__device__ __forceinline__ void moved_slice(int L, int slot, int& level, int& t, int& k) {
  const int d = 31 - __clz(slot);
  level = L - 1 - d;
  k = slot - (1 << d);
  t = (2 * k + 1) << level;
}

// The old beads' part of ln(T_old / T_new), per moved slice into m.old.  One warp.
static __device__ __noinline__ void mover_old(const DevSys& s, const Smem& m, int ipart) {
  const int np = s.npart, sp = species_of(s, ipart);
#pragma unroll 1
  for (int slot = threadIdx.x & 31; slot < (1 << s.nlevel); slot += 32) {
    if (slot == 0) continue;
    int level, t, k;
    moved_slice(s.nlevel, slot, level, t, k);
    const int tp = t - (1 << level), tn = t + (1 << level);
    const double inv2Sigma2 = s.mov_inv2s2[level][sp];
    const double ox = m.s1x[t * np + ipart], oy = m.s1y[t * np + ipart], oz = m.s1z[t * np + ipart];
    const double opx = m.s1x[tp * np + ipart], opy = m.s1y[tp * np + ipart], opz = m.s1z[tp * np + ipart];
    const double onx = m.s1x[tn * np + ipart], ony = m.s1y[tn * np + ipart], onz = m.s1z[tn * np + ipart];
    double acc = 0.0;
    if (s.mover == PIMC_MOVER_FREE) {
      double ax = onx - opx, ay = ony - opy, az = onz - opz;
      pbc(s, ax, ay, az);
      ax = __fma_rn(ax, 0.5, opx);  // (halving is exact)
      ay = __fma_rn(ay, 0.5, opy);
      az = __fma_rn(az, 0.5, opz);
      pbc(s, ax, ay, az);
      double ex = ox - ax, ey = oy - ay, ez = oz - az;
      pbc(s, ex, ey, ez);
      acc -= ex * ex * inv2Sigma2;
      acc -= ey * ey * inv2Sigma2;
      acc -= ez * ez * inv2Sigma2;
    } else {
      double po[3] = {ox - opx, oy - opy, oz - opz}, no[3] = {ox - onx, oy - ony, oz - onz};
      double dol[3] = {onx - opx, ony - opy, onz - opz};
      pbc(s, po[0], po[1], po[2]);
      pbc(s, no[0], no[1], no[2]);
      pbc(s, dol[0], dol[1], dol[2]);
      for (int d = 0; d < 3; ++d) {
        acc -= po[d] * po[d] * inv2Sigma2 * 0.5;
        acc -= no[d] * no[d] * inv2Sigma2 * 0.5;
        acc += dol[d] * dol[d] * inv2Sigma2 * 0.25;
      }
    }
    m.old[slot] = acc;
  }
}

// The new beads of every level, and ln(T_old / T_new) per level into llt.  One
// warp; reads the section's end beads in m.mx, m.nrm and m.old.
static __device__ __noinline__ void mover_all(const DevSys& s, const Smem& m, int ipart,
                                              uint64_t seed, uint32_t att, double* llt) {
  const int L = s.nlevel, lane = threadIdx.x & 31, sp = species_of(s, ipart);
  if (lane == 0) llt[L] = 0.0;  // the top level moves nothing
#pragma unroll 1
  for (int c = 0; 32 * c < (1 << L); ++c) {
    const int slot = 32 * c + lane;
    const bool on = slot > 0 && slot < (1 << L);
    int level, t, k;
    moved_slice(L, on ? slot : 1, level, t, k);
    const int tp = t - (1 << level), tn = t + (1 << level), ord = on ? slot - 1 : 0;
    const double sigma = s.mov_sigma[level][sp], inv2Sigma2 = s.mov_inv2s2[level][sp];
    const double z0 = m.nrm[3 * ord], z1 = m.nrm[3 * ord + 1], z2 = m.nrm[3 * ord + 2];
    double acc = 0.0;
    const int dlo = c ? 5 : 0, dhi = c ? 5 : min(4, L - 1);
    if (s.mover == PIMC_MOVER_FREE) {
      double dx = __dmul_rn(z0, sigma), dy = __dmul_rn(z1, sigma), dz = __dmul_rn(z2, sigma);
      pbc(s, dx, dy, dz);
      acc += dx * dx * inv2Sigma2;
      acc += dy * dy * inv2Sigma2;
      acc += dz * dz * inv2Sigma2;
#pragma unroll 1
      for (int d = dlo; d <= dhi; ++d) {
        if (on && level == L - 1 - d) {
          const double mpx = m.mx[tp], mpy = m.my[tp], mpz = m.mz[tp];
          double x = m.mx[tn] - mpx, y = m.my[tn] - mpy, z = m.mz[tn] - mpz;
          pbc(s, x, y, z);
          x = __fma_rn(x, 0.5, mpx);
          y = __fma_rn(y, 0.5, mpy);
          z = __fma_rn(z, 0.5, mpz);
          pbc(s, x, y, z);
          x = __dadd_rn(x, dx);
          y = __dadd_rn(y, dy);
          z = __dadd_rn(z, dz);
          pbc(s, x, y, z);
          m.mx[t] = x;
          m.my[t] = y;
          m.mz[t] = z;
        }
        __syncwarp();
      }
    } else {
#pragma unroll 1
      for (int d = dlo; d <= dhi; ++d) {
        if (on && level == L - 1 - d) {
          const double mpx = m.mx[tp], mpy = m.my[tp], mpz = m.mz[tp];
          double md[3] = {m.mx[tn] - mpx, m.my[tn] - mpy, m.mz[tn] - mpz};
          pbc(s, md[0], md[1], md[2]);
          md[0] *= 0.5; md[1] *= 0.5; md[2] *= 0.5;
          mover_image(s, md, inv2Sigma2, seed, s.stream_id, att,
                      level_uniform_base(s, level) + 3u * k);
          double x = __fma_rn(z0, sigma, __dadd_rn(md[0], mpx));
          double y = __fma_rn(z1, sigma, __dadd_rn(md[1], mpy));
          double z = __fma_rn(z2, sigma, __dadd_rn(md[2], mpz));
          pbc(s, x, y, z);
          m.mx[t] = x;
          m.my[t] = y;
          m.mz[t] = z;
        }
        __syncwarp();
      }
      if (on) {
        const double nx = m.mx[t], ny = m.my[t], nz = m.mz[t];
        const double mpx = m.mx[tp], mpy = m.my[tp], mpz = m.mz[tp];
        const double mnx = m.mx[tn], mny = m.my[tn], mnz = m.mz[tn];
        double pn[3] = {nx - mpx, ny - mpy, nz - mpz}, nn[3] = {nx - mnx, ny - mny, nz - mnz};
        double dn[3] = {mnx - mpx, mny - mpy, mnz - mpz};
        pbc(s, pn[0], pn[1], pn[2]);
        pbc(s, nn[0], nn[1], nn[2]);
        pbc(s, dn[0], dn[1], dn[2]);
        for (int d = 0; d < 3; ++d) {
          acc += pn[d] * pn[d] * inv2Sigma2 * 0.5;
          acc += nn[d] * nn[d] * inv2Sigma2 * 0.5;
          acc -= dn[d] * dn[d] * inv2Sigma2 * 0.25;
        }
      }
    }
    double x = on ? acc + m.old[slot] : 0.0;
    if (c == 0) {
      x = fold_by_depth(x, min(32, 1 << L));
      const int d = 31 - __clz(max(lane, 1));
      if (on && lane == (1 << d)) llt[L - 1 - d] = x;
    } else {
      x = fold_warp(x);
      if (lane == 0) llt[L - 6] = x;
    }
  }
  __syncwarp();
}

// The movers' makeMove for one moving particle at one level (delayed rejection,
// whose second proposal shifts the normals and uniforms of the levels under it);
// threads own moved slices.  Returns ln(T_old/T_new).
// oshift: moved-slice orders taken by a delayed-rejection proposal before
// this level; second: the delayed-rejection proposal itself (its width).
static __device__ __noinline__ double mover_level_part(const DevSys& s, const Smem& m, int ipart, int level,
                              int oshift, bool second) {
  const int L = s.nlevel, np = s.npart;
  const int nStride = 1 << level;
  const int nmov = (level == L) ? 0 : (1 << (L - level - 1));
  const int ord0 = ((level == L) ? 0 : (1 << (L - level - 1)) - 1) + oshift;
  const int sp = species_of(s, ipart);
  const double sigma = second ? s.dr_sigma[sp] : s.mov_sigma[level][sp];
  const double inv2Sigma2 = second ? s.dr_inv2s2[sp] : s.mov_inv2s2[level][sp];
  double part = 0.0;
#pragma unroll 1
  for (int k = threadIdx.x; k < nmov; k += blockDim.x) {
    const int t = nStride * (2 * k + 1), tp = t - nStride, tn = t + nStride;
    // the attempt's normals were drawn up front (attempt_normals)
    const double z0 = m.nrm[3 * (ord0 + k)], z1 = m.nrm[3 * (ord0 + k) + 1];
    const double z2 = m.nrm[3 * (ord0 + k) + 2];
    const double ox = m.s1x[t * np + ipart], oy = m.s1y[t * np + ipart], oz = m.s1z[t * np + ipart];
    const double opx = m.s1x[tp * np + ipart], opy = m.s1y[tp * np + ipart], opz = m.s1z[tp * np + ipart];
    const double onx = m.s1x[tn * np + ipart], ony = m.s1y[tn * np + ipart], onz = m.s1z[tn * np + ipart];
    const double mpx = m.mx[tp], mpy = m.my[tp], mpz = m.mz[tp];
    const double mnx = m.mx[tn], mny = m.my[tn], mnz = m.mz[tn];
    double acc = 0.0;
    double mdx = mnx - mpx, mdy = mny - mpy, mdz = mnz - mpz;
    pbc(s, mdx, mdy, mdz);
    mdx *= 0.5; mdy *= 0.5; mdz *= 0.5;
    mdx += mpx; mdy += mpy; mdz += mpz;
    pbc(s, mdx, mdy, mdz);
    double dx = z0 * sigma, dy = z1 * sigma, dz = z2 * sigma;
    pbc(s, dx, dy, dz);
    double nx = mdx + dx, ny = mdy + dy, nz = mdz + dz;
    pbc(s, nx, ny, nz);
    m.mx[t] = nx;
    m.my[t] = ny;
    m.mz[t] = nz;
    acc += dx * dx * inv2Sigma2;
    acc += dy * dy * inv2Sigma2;
    acc += dz * dz * inv2Sigma2;
    double ax = onx - opx, ay = ony - opy, az = onz - opz;
    pbc(s, ax, ay, az);
    ax *= 0.5; ay *= 0.5; az *= 0.5;
    ax += opx; ay += opy; az += opz;
    pbc(s, ax, ay, az);
    double ex = ox - ax, ey = oy - ay, ez = oz - az;
    pbc(s, ex, ey, ez);
    acc -= ex * ex * inv2Sigma2;
    acc -= ey * ey * inv2Sigma2;
    acc -= ez * ez * inv2Sigma2;
    part += acc;
  }
  return part;
}

// FreeMover::makeMove for one level: the beads, and ln(T_old/T_new) summed over the block.
static __device__ double mover_level(const DevSys& s, const Smem& m, int ipart, int level,
                                     int oshift = 0, bool second = false) {
  return block_sum(mover_level_part(s, m, ipart, level, oshift, second), m.red);
}

// Evaluates one slice pair per lane group of width W.
static __device__ __noinline__ void node_eval_dispatch(int W, const DevSys& s, int sp,
                                                   const SliceView& v1, const SliceView& v2,
                                                   double scale, double* scr, int full,
                                                   double* ecache, unsigned cols, bool write,
                                                   double& det, int& err, double* d1,
                                                   double* d2, double* newcol = nullptr,
                                                   unsigned rowmask = 0xffffffffu,
                                                   double* cold = nullptr,
                                                   const double* xin = nullptr,
                                                   double det_in = 0.0, double* xout = nullptr,
                                                   double xepoch = 0.0) {
  // (xin and xout are the same for every lane of a warp)
  const auto run = [&](auto w, auto sho, auto sm) {
    node_eval_group<decltype(w)::value, decltype(sho)::value, decltype(sm)::value>(
        s, sp, v1, v2, scale, scr, full, ecache, cols, write, det, err, d1, d2, newcol, rowmask,
        cold, xin, det_in, xout, xepoch);
  };
  const std::integral_constant<int, 8> w8;
  const std::integral_constant<int, 16> w16;
  const std::integral_constant<int, 32> w32;
  const std::true_type yes;
  const std::false_type no;
  if (s.node_kind[sp] == PIMC_NODES_SHO) {
    if (W == 8) run(w8, yes, no);
    else if (W == 16) run(w16, yes, no);
    else run(w32, yes, no);
  } else if (xin || xout) {
    if (W == 8) run(w8, no, yes);
    else if (W == 16) run(w16, no, yes);
    else run(w32, no, yes);
  } else {
    if (W == 8) run(w8, no, no);
    else if (W == 16) run(w16, no, no);
    else run(w32, no, no);
  }
}

// Index of the entry's stale-row word (after the element matrices): bit r set
// = row r (r2 particle r) moved since the matrix was cached; bit 63 = the
// cached matrix is not usable at all.
__device__ __forceinline__ int cache_mask_slot(const DevSys& s, int sp) {
  const int n = s.spec_count[sp];
  return 2 + 2 * n + n * n * (s.node_kind[sp] == PIMC_NODES_FREE ? 4 : 1);
}
// Whether a species' cached Slater entries carry the inverse block that the
// mixed form's Sherman-Morrison updates work on: FreeParticleNodes species.
// (The SHONodes matrices of the cold dots are ill-conditioned by
// construction, cond 1e12..1e14 at omega/T = 20, where every factorisation
// fails the updates' conditioning gate: the block would only cost them.)
__host__ __device__ __forceinline__ bool sm_species(const DevSys& s, int sp) {
  return s.mixed && s.node_kind[sp] == PIMC_NODES_FREE;
}
// Lane-group width of a species' evaluations in a launch that asks for wmin lanes at
// least: that of its size where it takes updates, which the matrices of a warp take
// together or not at all (one matrix a warp instead of four would update others, and a
// chain depend on the launch it runs in).
__host__ __device__ __forceinline__ int node_launch_width(const DevSys& s, int sp, int wmin) {
  const int n = s.spec_count[sp], w = node_group_width(n), most = node_group_widest(n);
  return sm_species(s, sp) || wmin < w ? w : (wmin < most ? wmin : most);
}
// Mixed form: index of the entry's inverse block [epoch of its scale, updates
// since the last factorisation, inverse (n*n, X layout)], after the stale-row word.
__device__ __forceinline__ int cache_x_slot(const DevSys& s, int sp) {
  return cache_mask_slot(s, sp) + 1;
}
__device__ __forceinline__ unsigned cache_rowmask(const double* e, int slot) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(e[slot]);
  return (b >> 63) ? 0xffffffffu : (unsigned)(b & 0xffffffffull);
}

// Slater-result cache entry of species sp for path slice t1 (r1 at t1, r2 at
// t1 + M/2): [0] epoch (NaN = invalid), [1] determinant, [2..2+n) d1,
// [2+n..2+2n) d2, [2+2n..) exp matrix (SHONodes).  An entry is valid while
// neither slice's particles of that species have moved and the species'
// scale epoch is unchanged; evaluate() of the same inputs at the same scale
// returns exactly these values, so a hit replaces the evaluation bit for bit.
__device__ __forceinline__ double* cache_entry(const DevSys& s, double* cache, int sp, int t1) {
  return cache + ((size_t)sp * s.nslice + t1) * s.nc_stride;
}

// One pass of the set-up over slices [start, nsec) of one node species (only_sp)
// or of all of them (only_sp < 0): cached results are copied, the others are
// evaluated, the species' warps side by side.  Determinants go to dm[sp][t],
// error flags to errs[sp][t], the moving species' distances to dist.  With llt,
// the last warp makes the attempt's proposals beside it (mover_all).
static __device__ __noinline__ void node_init_pass(const DevSys& s, const Smem& m, const double* scale,
                                      const int* epoch, int msp, double* cache, int ifirst1,
                                      int only_sp, int start, int ipart, uint64_t seed,
                                      uint32_t att, double* llt) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int nsec = s.nsec, M = s.nslice, nsm = s.ns_max;
  int* errs = m.ictl + C_NCTL;                 // [kMaxSpecies][nsec]
  int* miss = errs + kMaxSpecies * nsec;       // [kMaxSpecies][nsec] slices to evaluate
  int* nmiss = m.ictl + C_NMISS;               // [kMaxSpecies] (C_NMISS .. C_NMISS + 3)
  const double NaN = __longlong_as_double(0x7ff8000000000000LL);
  const int nt = nsec - start;
  // A warp lists a species' misses in the order of their slices: matrices that share a
  // warp below are updated together or not at all, so a chain would follow the order.
#pragma unroll 1
  for (int sp = warp; sp < s.nspecies; sp += nwarps) {
    const bool on = s.node_kind[sp] && (only_sp < 0 || sp == only_sp);
    int count = 0;
#pragma unroll 1
    for (int t0 = start; on && t0 < nsec; t0 += 64) {  // (two slices' loads in flight)
      double ep[2], det[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = min(t0 + 32 * q + lane, nsec - 1);
        const double* e = cache ? cache_entry(s, cache, sp, wrap_slice(ifirst1 + t, M)) : nullptr;
        ep[q] = e ? e[0] : NaN;
        det[q] = e ? e[1] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int t = t0 + 32 * q + lane;
        const bool hit = ep[q] == (double)epoch[sp], in = t < nsec;
        if (in && hit) {
          m.dm[sp * nsec + t] = det[q];
          errs[sp * nsec + t] = 0;
        }
        const unsigned lost = __ballot_sync(0xffffffffu, in && !hit);
        if (in && !hit) miss[sp * nsec + count + __popc(lost & ((1u << lane) - 1u))] = t;
        count += __popc(lost);
      }
    }
    if (lane == 0) nmiss[sp] = count;
  }
  // the moving species' distances where the entry is valid (a particle per thread:
  // as a loop of the slice's own thread this took 8,000-21,000 clocks of load latency)
  if (cache && msp >= 0 && s.node_kind[msp] && (only_sp < 0 || only_sp == msp)) {
    const int n = s.spec_count[msp];
#pragma unroll 1
    for (int it = threadIdx.x; it < nt * n; it += blockDim.x) {
      const int t = start + it / n, j = it - (t - start) * n;
      const double* e = cache_entry(s, cache, msp, wrap_slice(ifirst1 + t, M));
      const double ep = e[0], a = e[2 + j], b = e[2 + n + j];
      if (ep == (double)epoch[msp]) {
        m.dist[(t * 2) * nsm + j] = a;
        m.dist[(t * 2 + 1) * nsm + j] = b;
      }
    }
  }
  __syncthreads();
  // warp tasks: each warp takes up to G misses of one species (lane groups of
  // a warp must run the same species so that they stay converged)
  int ntask = 0, first[kMaxSpecies + 1], wmin = m.wide ? 32 : 8;
  const unsigned narrow = s.node_widths, widest = s.node_widest;
  const auto width = [&](int sp) {
    return min(max(wmin, (int)((narrow >> (8 * sp)) & 63u)), (int)((widest >> (8 * sp)) & 63u));
  };
#pragma unroll 1
  for (;; wmin >>= 1) {  // (wide: the widest groups that take no further round)
    ntask = 0;
#pragma unroll 1
    for (int sp = 0; sp < s.nspecies; ++sp) {
      const int shift = 6 - __ffs(width(sp));  // 32 / width groups a warp
      first[sp] = ntask;
      ntask += (nmiss[sp] + (1 << shift) - 1) >> shift;
    }
    first[s.nspecies] = ntask;
    if (wmin == 8 || ntask <= nwarps) break;
  }
  if (llt && warp == nwarps - 1) mover_all(s, m, ipart, seed, att, llt);
#pragma unroll 1
  for (int wt = warp; wt < ntask; wt += nwarps) {
    int sp = 0;
    while (wt >= first[sp + 1]) ++sp;
    const int n = s.spec_count[sp];
    const bool sho = s.node_kind[sp] == PIMC_NODES_SHO, mine = sp == msp;
    const int W = width(sp);
    const int G = 32 / W, gm = lane / W, glm = lane & (W - 1);
    const int base = (wt - first[sp]) * G;
    const int task = base + gm;
    const bool act = task < nmiss[sp];
    const int t = miss[sp * nsec + (act ? task : base)];
    double* scrm = group_scr(m, warp * G + gm, G, n, !sho);
    double* coldm = group_cold(m, warp * G + gm, G, n, !sho);
    double* e = cache ? cache_entry(s, cache, sp, wrap_slice(ifirst1 + t, M)) : nullptr;
    SliceView v1{m.s1x, m.s1y, m.s1z, s.npart, t, -1, 0, 0, 0};
    SliceView v2{m.s2x, m.s2y, m.s2z, s.npart, t, -1, 0, 0, 0};
    double det = 0;
    int err = 0;
    double* ec = e ? e + 2 + 2 * n
                   : ((sho && mine && m.ecache) ? m.ecache + (size_t)t * n * n : nullptr);
    // with a cache every miss is evaluated in full so that its entry is complete
    const int full = (mine || e) ? 1 : 0;
    double* d1 = mine ? m.dist + (t * 2) * nsm : (e ? e + 2 : nullptr);
    double* d2 = mine ? m.dist + (t * 2 + 1) * nsm : (e ? e + 2 + n : nullptr);
    const unsigned rmask = e ? cache_rowmask(e, cache_mask_slot(s, sp)) : 0xffffffffu;
    // mixed form: the entry's inverse, updated for its changed rows when it can be
    double* xb = (e && sm_species(s, sp)) ? e + cache_x_slot(s, sp) : nullptr;
    node_eval_dispatch(W, s, sp, v1, v2, scale[sp], scrm, full, ec, 0u, act, det, err, d1, d2,
                       nullptr, rmask, coldm, xb, e ? e[1] : 0.0, xb, (double)epoch[sp]);
    if (act) {
      if (e && mine && glm < n) {
        e[2 + glm] = d1[glm];
        e[2 + n + glm] = d2[glm];
      }
      if (glm == 0) {
        m.dm[sp * nsec + t] = det;
        errs[sp * nsec + t] = err;
        if (e) {
          e[1] = det;
          e[0] = err ? NaN : (double)epoch[sp];
          e[cache_mask_slot(s, sp)] = 0.0;  // the element matrix is whole again
        }
      }
    }
  }
  __syncthreads();
}

// |x| < lo or |x| > hi (both normal; never for a NaN), on the integer pipe
__device__ __forceinline__ bool outside_magnitudes(double x, double lo, double hi) {
  const long long a = __double_as_longlong(x) & 0x7fffffffffffffffLL;
  return a < __double_as_longlong(lo) || (a > __double_as_longlong(hi) && a <= 0x7ff0000000000000LL);
}

// FixedNodeAction::initialize (src/fixednode/FixedNodeAction.cc:331-357) for every
// species with a node model, reproducing NodeModel::evaluate's rescaling loop
// (src/fixednode/SHONodes.cc:112-126): every species' slices are evaluated in
// parallel at the current scales (pi-qmc sets the species up one after the
// other; they are independent); at a species' first slice whose determinant
// leaves [1e-50, 1e50] its loop is replayed sequentially, and its later
// slices are re-evaluated.
static __device__ __noinline__ void node_initialize(const DevSys& s, const Smem& m, double* scale, int* epoch,
                                int msp, uint32_t* status, double* cache, int ifirst1, int ipart,
                                uint64_t seed, uint32_t att, double* llt) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsec = s.nsec, M = s.nslice;
  const int nsm = s.ns_max;
  int* errs = m.ictl + C_NCTL;  // [kMaxSpecies][nsec]
  const double NaN = __longlong_as_double(0x7ff8000000000000LL);
  node_init_pass(s, m, scale, epoch, msp, cache, ifirst1, -1, 0, ipart, seed, att, llt);
#pragma unroll 1
  for (int sp = 0; sp < s.nspecies; ++sp) {
    if (!s.node_kind[sp]) continue;
    const int n = s.spec_count[sp];
    const int W = node_group_width(n), g = lane / W;
    const bool sho = s.node_kind[sp] == PIMC_NODES_SHO;
    const bool mine = sp == msp;
    double* dm = m.dm + sp * nsec;
    int* er = errs + sp * nsec;
    int start = 0;
    for (int round = 0; round < 64; ++round) {
      if (round > 0)
        node_init_pass(s, m, scale, epoch, msp, cache, ifirst1, sp, start, ipart, seed, att, nullptr);
      // (every warp looks for itself, a slice per lane)
      int k = -1;
#pragma unroll 1
      for (int t0 = start; k < 0 && t0 < nsec; t0 += 32) {
        const int t = t0 + lane;
        const unsigned bad = __ballot_sync(
            0xffffffffu, t < nsec && (er[t] || outside_magnitudes(dm[t], 1e-50, 1e50)));
        if (bad) k = t0 + __ffs(bad) - 1;
      }
      if (k < 0) break;
      __syncthreads();  // (warp 0 changes what the others have read)
      if (warp == 0) {
        // pi-qmc's do-while rescale loop on slice k, by group 0 of warp 0
        // (the other groups repeat it without storing).
        double det = dm[k];
        int err = er[k];
        double sc2 = scale[sp];
        int guard = 0;
        double* dsc = group_scr(m, g, 32 / W, n, !sho);
        double* dcold = group_cold(m, g, 32 / W, n, !sho);
        // (the elements do not depend on the scale: those of the slice's entry, whole
        // since the pass above)
        double* ec = cache ? cache_entry(s, cache, sp, wrap_slice(ifirst1 + k, M)) + 2 + 2 * n
                           : nullptr;
        while (err || fabs(det) < 1e-50 || fabs(det) > 1e50) {
          if (err || ++guard > 2000) {
            if (lane == 0) *status |= err ? (PIMC_STATUS_SINGULAR | PIMC_STATUS_RESCALE_LIMIT)
                                          : PIMC_STATUS_RESCALE_LIMIT;
            break;
          }
          if (fabs(det) < 1e-250)
            sc2 *= 2;
          else
            sc2 *= pow(fabs(det), -1. / n);
          SliceView v1{m.s1x, m.s1y, m.s1z, s.npart, k, -1, 0, 0, 0};
          SliceView v2{m.s2x, m.s2y, m.s2z, s.npart, k, -1, 0, 0, 0};
          double d = 0;
          int e2 = 0;
          node_eval_dispatch(W, s, sp, v1, v2, sc2, dsc, mine ? 1 : 0, ec, 0u, g == 0, d, e2,
                             m.dist + (k * 2) * nsm, m.dist + (k * 2 + 1) * nsm, nullptr, 0u,
                             dcold);
          det = __shfl_sync(0xffffffffu, d, 0);
          err = __shfl_sync(0xffffffffu, e2, 0);
        }
        if (lane == 0) {
          dm[k] = det;
          er[k] = err;
          if (sc2 != scale[sp]) epoch[sp] += 1;
          scale[sp] = sc2;
          if (cache) cache_entry(s, cache, sp, wrap_slice(ifirst1 + k, M))[0] = NaN;
        }
      }
      __syncthreads();
      start = k + 1;
      if (start >= nsec) break;
    }
    // crossing check, as the reference counts errors at set-up
    if (warp == 0) {
      bool crossed = false;
#pragma unroll 1
      for (int t = lane; t < nsec; t += 32) crossed = crossed || er[t] || dm[t] * dm[0] <= 1e-200;
      if (__any_sync(0xffffffffu, crossed) && lane == 0) *status |= PIMC_STATUS_INIT_CROSSING;
    }
  }
  if (msp >= 0 && s.node_kind[msp]) {
    // newDist(0) = dist(0)
#pragma unroll 1
    for (int i = threadIdx.x; i < 2 * nsm; i += blockDim.x) m.ndist[i] = m.dist[i];
  }
  __syncthreads();
}

// FixedNodeAction::getActionDifference's nodal action over the section
// (src/fixednode/FixedNodeAction.cc:96-131), after level 0's evaluations.
static __device__ __noinline__ double nodal_action(const DevSys& s, const Smem& m, int n) {
  const int nsec = s.nsec, nsm = s.ns_max;
  return share_sum(m.nshare, m.red, [&](int h) {
    double part = 0.0;
    FSum fpart;
#pragma unroll 1
    for (int it = threadIdx.x + h * blockDim.x; it < (nsec - 1) * n; it += 32 * m.nshare) {
      const int t = 1 + it / n, p = it - (t - 1) * n;
      double num = 1.0, den = 1.0;
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {  // d1, then d2
        const double* D = m.dist + (t * 2 + side) * nsm + p;
        const double* N = m.ndist + (t * 2 + side) * nsm + p;
        const double d = D[0] * D[-2 * nsm], e = N[0] * N[-2 * nsm];
        if (s.mixed) {
          // FP32 terms (1 - e^-x through expm1 keeps them accurate near the node),
          // their sum compensated
          const float a = -expm1f(-f32_rn(d)), b = -expm1f(-f32_rn(e));
          fpart.add(logf(a) - logf(b));
        } else {  // (one logarithm for both sides)
          num *= 1 - exp(-d);
          den *= 1 - exp(-e);
        }
      }
      if (!s.mixed) part += log(num / den);
    }
    return s.mixed ? fpart.value() : part;
  });
}

// Bisection levels lo .. hi of the attempt at once, after its proposals (a
// level's proposal does not depend on the decisions above it).  The changed
// slices of the levels go to the first warps, side by side; the other warps
// take the action differences of levels alo .. ahi (all of them together down from
// the top, ahi = nlevel, or one; none with alo > ahi), or every warp does after
// its node work when that takes more than half of them.  Per level l: lds[l] the
// action difference, lnd[l] the fixed-node difference
// (FixedNodeAction::getActionDifference, src/fixednode/FixedNodeAction.cc:39-131:
// 2e100 when a changed slice crosses a node; on level 0, alone, the nodal action).
// The caller applies pi-qmc's level-by-level decisions to them.
static __device__ __noinline__ void eval_levels(const DevSys& s, const Smem& m, double scale, int msp,
                                  int ipart, int lo, int hi, int alo, int ahi, bool mynode,
                                  double* cache, int ifirst1, int ep, double* lds, double* lnd) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int nsec = s.nsec, nsm = s.ns_max, L = s.nlevel;
  const int n = mynode ? s.spec_count[msp] : 1;
  const int top = hi == L ? L - 1 : hi;
  int ntask = 0;
  if (mynode)
#pragma unroll 1
    for (int l = top; l >= lo; --l) ntask += (nsec - 1 - (1 << l)) / (1 << (l + 1)) + 1;
  // lane groups of the species' width, packed (32 / W matrices a warp): the
  // SM's narrow FP64 pipe, shared by every resident warp, is the limit, and a
  // packed warp instruction serves several matrices
  int W = node_group_width(n);
  // (of the narrowest groups: the sums' shares do not depend on the launch)
  const int dmax = L - alo, dmin = ahi == L ? 0 : dmax;
  const int shares = m.nshare - first_action_warp(ntask * W, m.nshare, s.mixed);
  const int a0 = first_action_warp(ntask * W, nwarps, s.mixed);
  // A CTA that has its SM to itself is bound by the chain of each matrix's operations,
  // not by the pipe: it takes the widest groups that need no further round of the
  // warps without action terms (128 mixed dots, one a CTA: 50.9 -> 44.9 ms a round, and
  // 41.1 with half of the warps on the action; two CTAs per SM share the pipe, where
  // narrow groups' fewer instructions count).
  if (m.wide && mynode) {
    const int most = a0 == 0 || alo > ahi ? nwarps : a0;
    const int widest = (s.node_widest >> (8 * msp)) & 63u;
    while (W < widest && ntask * W <= 16 * most) W *= 2;
  }
  const int G = 32 / W, g = lane / W, nodeW = min(nwarps, (ntask + G - 1) / G);
  if (mynode) {
    if (threadIdx.x == 0) m.ictl[C_FLAG] = 0;
    if (hi == L) {
      // the top level's only slice is the section's fixed end: copied from the set-up
      const int t = nsec - 1;
#pragma unroll 1
      for (int i = threadIdx.x; i < 2 * nsm; i += blockDim.x) m.ndist[t * 2 * nsm + i] = m.dist[t * 2 * nsm + i];
    }
    __syncthreads();
    if (hi == L && threadIdx.x == 0) {
      const int t = nsec - 1;
      m.ndm[t] = m.dm[msp * nsec + t];
      if (m.ndm[t] * m.dm[msp * nsec + 0] <= 1e-200) atomicOr(&m.ictl[C_FLAG], 1 << L);
    }
    if (warp < nodeW) {
      const bool sho = s.node_kind[msp] == PIMC_NODES_SHO;
      double* scr = group_scr(m, warp * G + g, G, n, !sho);
      double* cold = group_cold(m, warp * G + g, G, n, !sho);
      const int jcol = ipart - s.spec_first[msp];
#pragma unroll 1
      for (int base = warp * G; base < ntask; base += nodeW * G) {
        const int task = base + g;
        const bool act = task < ntask;
        int k = act ? task : base, l = top;  // task -> (level, slice)
#pragma unroll 1
        for (;;) {
          const int nl = (nsec - 1 - (1 << l)) / (1 << (l + 1)) + 1;
          if (k < nl || l == lo) break;
          k -= nl;
          --l;
        }
        const int t = (1 << l) + k * (1 << (l + 1));
        SliceView v1{m.s1x, m.s1y, m.s1z, s.npart, t, ipart, m.mx[t], m.my[t], m.mz[t]};
        SliceView v2{m.s2x, m.s2y, m.s2z, s.npart, t, -1, 0, 0, 0};
        double det = 0;
        int err = 0;
        double* ec = nullptr;
        const double* xb = nullptr;  // mixed form: the entry's inverse block
        double det_in = 0.0;
        if (cache) {
          double* e = cache_entry(s, cache, msp, wrap_slice(ifirst1 + t, s.nslice));
          ec = e + 2 + 2 * n;
          if (sm_species(s, msp) && m.xstage) {
            xb = e + cache_x_slot(s, msp);
            det_in = e[1];
          }
        } else if (sho && m.ecache) {
          ec = m.ecache + (size_t)t * n * n;
        }
        node_eval_dispatch(W, s, msp, v1, v2, scale, scr, 1, ec, 1u << jcol, act, det, err,
                           m.ndist + (t * 2) * nsm, m.ndist + (t * 2 + 1) * nsm,
                           cache ? m.ncol + t * m.ncol_stride : nullptr, 0u, cold, xb, det_in,
                           xb ? m.xstage + (size_t)t * m.xstage_stride : nullptr, (double)ep);
        if (act && (lane & (W - 1)) == 0) {
          m.ndm[t] = det;
          if (err || det * m.dm[msp * nsec + 0] <= 1e-200) atomicOr(&m.ictl[C_FLAG], 1 << l);
        }
      }
    }
  }
  if (alo <= ahi) {
    // (the sums' shares are those of m.nshare warps, several to a warp here if need be)
    const bool apart = m.nshare > nwarps;
    const int words = apart ? action_sum_words(L) : 0;
    const int off = apart ? action_sep_words(L, takes_single_levels(s), s.mixed) : 0;
    if (warp >= a0) {
      double* buf = m.act + (size_t)warp * m.act_stride;
      double* sums = buf + off;
#pragma unroll 1
      for (int w = warp - a0; w < shares; w += nwarps - a0) {
        if (s.mixed)
          action_warp<true>(s, m, ipart, dmin, dmax, w, shares, buf, sums);
        else
          action_warp<false>(s, m, ipart, dmin, dmax, w, shares, buf, sums);
        sums += words;
      }
    }
    __syncthreads();
    action_reduce(s, m.act + (size_t)a0 * m.act_stride + off, m.act_stride, dmin, dmax, shares,
                  nwarps - a0, words, lds);
  }
  __syncthreads();
  const int flags = mynode ? m.ictl[C_FLAG] : 0;
  double nodal = 0.0;
  if (mynode && lo == 0 && !(flags & 1)) nodal = nodal_action(s, m, n);
  if (threadIdx.x == 0)
#pragma unroll 1
    for (int level = lo; level <= hi; ++level)
      lnd[level] = ((flags >> level) & 1) ? 2e100 : (level == 0 ? nodal : 0.0);
  __syncthreads();
}


// MultiLevelSampler::tryMove's delayed rejection (src/advancer/MultiLevelSampler.cc:114-148;
// DoubleMLSampler.cc:148-204 with the node term) after the first proposal B at
// level L - 1 was rejected: the second proposal C (width newSigmaFactor, the
// next normals), its action difference, FreeMover::makeDelayedMove
// (src/advancer/mover/FreeMover.cc:127-185) for the forward C->B and reverse
// B->C probabilities, and the combined acceptance with the next uniform.
// Thread 0 holds piRatioBoA and the acceptance of B in red[kWarps + 3, 4];
// returns the level-(L - 1) rejection (C_REJECT) and, when C is accepted, the
// modified action difference in red[kWarps + 2].
static __device__ __noinline__ void delayed_rejection(const DevSys& s, const Smem& m, double scale,
                                                     int msp, int ipart, bool mynode,
                                                     double* cache, int ifirst1, int ep,
                                                     uint64_t seed, uint32_t att, uint32_t uacc,
                                                     double oldDS, long long* ek,
                                                     long long* ekstage, pimc_move_record* rec,
                                                     uint32_t* status) {
  const int L = s.nlevel, level = L - 1, nsec = s.nsec;
  const int t = 1 << level, tp = 0, tn = nsec - 1;
  const int sp = species_of(s, ipart);
  double* bead = m.red + kWarps + 5;  // the rejected bead B
  if (threadIdx.x == 0) {
    bead[0] = m.mx[t];
    bead[1] = m.my[t];
    bead[2] = m.mz[t];
  }
  __syncthreads();
  // C: FreeMover::makeMove with factor = newFactor and the next normals
  const double lnTC = mover_level(s, m, ipart, level, 1, true);
  double* lds = m.red + kWarps + 8;
  double* lnd = lds + 2 * kMaxLevels;
  eval_levels(s, m, scale, msp, ipart, level, level, level, level, mynode, cache, ifirst1, ep, lds,
              lnd);
  double dsC = lds[level];
  if (s.ewald && s.coulomb && level == 0) {
    if (ek)
      dsC += ewald_level0_cached(s, m, ipart, ifirst1, ek, ekstage);
    else
#pragma unroll 1
      for (int k = 1; k < nsec - 1; ++k) dsC += ewald_slice_diff(s, m, ipart, k);
  }
  const double dsnC = lnd[level];
  if (threadIdx.x == 0) {
    const double piRatioBoA = m.red[kWarps + 3], accRatioA2B = m.red[kWarps + 4];
    const double sigma = s.mov_sigma[level][sp], inv2Sigma2 = s.mov_inv2s2[level][sp];
    // transA2B = B's forward probability: its Gaussian step, as makeMove drew it
    double dx = m.nrm[0] * sigma, dy = m.nrm[1] * sigma, dz = m.nrm[2] * sigma;
    pbc(s, dx, dy, dz);
    double transA2B = 0.0;
    transA2B += dx * dx * inv2Sigma2;
    transA2B += dy * dy * inv2Sigma2;
    transA2B += dz * dz * inv2Sigma2;
    transA2B += log(1.0);
    const double deltaC = s.fixed_node ? dsC + dsnC : dsC;
    const double piRatioCoA = -deltaC + oldDS;
    const double accRatioA2C = exp(lnTC + piRatioCoA);
    // makeDelayedMove with factor = defaultFactor: the midpoint of the level's
    // neighbours (the section ends, the same for B and C), B and C about it
    double mx = m.mx[tn] - m.mx[tp], my = m.my[tn] - m.my[tp], mz = m.mz[tn] - m.mz[tp];
    pbc(s, mx, my, mz);
    mx *= 0.5; my *= 0.5; mz *= 0.5;
    mx += m.mx[tp]; my += m.my[tp]; mz += m.mz[tp];
    pbc(s, mx, my, mz);
    double bx = bead[0] - mx, by = bead[1] - my, bz = bead[2] - mz;
    pbc(s, bx, by, bz);
    double forwardProb = 0.0, toldOverTnew = 0.0, tmp;
    tmp = bx * bx * inv2Sigma2; forwardProb -= tmp; toldOverTnew += tmp;
    tmp = by * by * inv2Sigma2; forwardProb -= tmp; toldOverTnew += tmp;
    tmp = bz * bz * inv2Sigma2; forwardProb -= tmp; toldOverTnew += tmp;
    forwardProb += log(1.0);
    double cx = m.mx[t] - mx, cy = m.my[t] - my, cz = m.mz[t] - mz;
    pbc(s, cx, cy, cz);
    toldOverTnew -= cx * cx * inv2Sigma2;
    toldOverTnew -= cy * cy * inv2Sigma2;
    toldOverTnew -= cz * cz * inv2Sigma2;
    toldOverTnew += log(1.0);
    const double transC2B = forwardProb;
    double accRatioC2B = exp(toldOverTnew - piRatioCoA + piRatioBoA);
    accRatioC2B = (accRatioC2B >= 1) ? 1 : accRatioC2B;
    const double accRatioA2B2C = accRatioA2C * exp(transC2B + transA2B) * (1 - accRatioC2B) /
                                 (1 - accRatioA2B);
    const double delta =
        deltaC - transC2B - transA2B - log((1 - accRatioC2B) / (1 - accRatioA2B));
    if (rec) {
      rec->ds[level] = dsC;
      rec->ds_node[level] = dsnC;
      rec->lnt[level] = lnTC;
    }
    if (!(isfinite(lnTC) && isfinite(dsC))) *status |= PIMC_STATUS_NONFINITE;
    const double u = stream_uniform(seed, s.stream_id, att, uacc + 1u);
    m.ictl[C_REJECT] = (u > accRatioA2B2C) ? level : -1;
    m.red[kWarps + 2] = delta;
  }
  __syncthreads();
}


// n values by a warp, eight loads in flight a lane
template <class T>
__device__ __forceinline__ void copy_warp(T* dst, const T* src, int n) {
#pragma unroll 1
  for (int k0 = threadIdx.x & 31; k0 < n; k0 += 256) {
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = src[min(k0 + 32 * q, n - 1)];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (k0 + 32 * q < n) dst[k0 + 32 * q] = v[q];
  }
}

// NT (largest block) and MINB set the register budget, 65536 / (NT * MINB)
// per thread; the variants are compiled in separate translation units
// (section_variants.cu) and chosen at run time by the launch configuration.
// kNodes = false: the variant for launches without node models, whose code
// leaves the fixed-node phases out (a smaller kernel: fewer instruction-fetch
// stalls when thousands of one-warp CTAs run different phases).
template <int NT, int MINB, bool kNodes = true>
__global__ void __launch_bounds__(NT, MINB) section_moves_kernel(RunParams P) {
  extern __shared__ double smem[];
  __shared__ DevSys S;
  __shared__ double scale[kMaxSpecies];
  __shared__ int epoch[kMaxSpecies];
  __shared__ uint32_t status;
  __shared__ long long nacc;
  __shared__ int rnext;
  // The carved pointers live in shared memory: the called phases take them
  // by reference, which would otherwise place them in each thread's stack.
  __shared__ Smem M_;
  // Persistent CTAs take replicas from a queue ordered longest-first, so that
  // uneven replicas (different N, M, L) balance across the SMs.
#pragma unroll 1
  for (;;) {
    if (threadIdx.x == 0) {
      const int k = atomicAdd(P.next, 1);
      rnext = (k < P.nrep) ? P.order[k] : -1;
    }
    __syncthreads();
    const int r = rnext;
    if (r < 0) break;
    {
      const int* src = (const int*)(P.sys + r);
      int* dst = (int*)&S;
#pragma unroll 1
      for (int i = threadIdx.x; i < (int)(sizeof(DevSys) / sizeof(int)); i += blockDim.x)
        dst[i] = src[i];
    }
    if (threadIdx.x == 0) {
      M_ = carve(smem, P.lay, P.sys[r], P.nodescr_g,
                 P.xstage ? P.xstage + (size_t)blockIdx.x * P.xstage_cta : nullptr, P.wide,
                 P.nshare);
      status = P.state[r].status;
      nacc = 0;
#pragma unroll 1
      for (int k = 0; k < kMaxSpecies; ++k) {
        scale[k] = P.state[r].node_scale[k];
        epoch[k] = P.state[r].epoch[k];
      }
    }
    __syncthreads();
    const DevSys& s = S;
    const Smem& m = M_;
    double* path = P.paths + s.path_offset;
    const uint32_t att0 = P.state[r].attempt;
    double* cache = (P.nodecache && s.nc_offset >= 0) ? P.nodecache + s.nc_offset : nullptr;
    long long* ek = (P.ekcache && s.ek_offset >= 0) ? P.ekcache + s.ek_offset : nullptr;
    long long* ekstage = ek ? P.ekstage + (size_t)blockIdx.x * P.ekstage_stride : nullptr;
    const int np = s.npart, nsec = s.nsec, M = s.nslice, L = s.nlevel;
    const bool fixed = kNodes && s.fixed_node;
#pragma unroll 1
    for (int i = threadIdx.x; i < np; i += blockDim.x) m.qpart[i] = s.charge[species_of(s, i)];
    const int nat = P.nattempt_r ? P.nattempt_r[r] : P.nattempt;
#pragma unroll 1
    for (int a = 0; a < nat; ++a) {
      const uint32_t att = att0 + (uint32_t)a;
      // ---- section choice and moving particle
      if (threadIdx.x < 32) {  // (a uniform per lane)
        int i1, i2 = -2;
        const double u = stream_uniform(P.seed, s.stream_id, att, min(threadIdx.x, 2));
        const double u1 = __shfl_sync(0xffffffffu, u, 1), u2 = __shfl_sync(0xffffffffu, u, 2);
        const double x = __shfl_sync(0xffffffffu, u, 0) * (1 - 1e-8);
        if (!fixed) {
          const int ilo = -1, ihi = M - 1;
          i1 = ilo + (int)((ihi + 1 - ilo) * x);
          if (i1 > ihi) i1 = ihi;
        } else {
          const int ilo = -1, ihi = M / 2 - 1;
          i1 = ilo + (int)((ihi + 1 - ilo) * x);
          if (i1 > ihi) i1 = ihi;
          if (u1 >= 0.5) i1 = (i1 + M / 2 + 1) % M - 1;
          i2 = (i1 + M / 2 + 1) % M - 1;
        }
        int ip = (int)(np * (fixed ? u2 : u1));
        if (ip >= np) ip = np - 1;
        if (threadIdx.x == 0) {
          m.ictl[C_IFIRST1] = i1;
          m.ictl[C_IFIRST2] = i2;
          m.ictl[C_IPART] = ip;
          m.ictl[C_REJECT] = -1;
        }
      }
      __syncthreads();
      const int ifirst1 = m.ictl[C_IFIRST1], ifirst2 = m.ictl[C_IFIRST2];
      const int ipart = m.ictl[C_IPART];
      load_section(s, path, ifirst1, m.s1x, m.s1y, m.s1z);
      if (fixed) load_section(s, path, ifirst2, m.s2x, m.s2y, m.s2z);
      attempt_normals(s, m, P.seed, s.stream_id, att);
      __syncthreads();
      double* lds = m.red + kWarps + 8;  // [kMaxLevels] per level: action difference,
      double* llt = lds + kMaxLevels;     // mover ln T,
      double* lnd = llt + kMaxLevels;     // fixed-node difference
#pragma unroll 1
      for (int t = threadIdx.x; t < nsec; t += blockDim.x) {
        m.mx[t] = m.s1x[t * np + ipart];
        m.my[t] = m.s1y[t * np + ipart];
        m.mz[t] = m.s1z[t * np + ipart];
      }
      if (!s.dr && (threadIdx.x >> 5) == (blockDim.x >> 5) - 1) mover_old(s, m, ipart);
      const int msp = species_of(s, ipart);
      const bool mynode = fixed && s.node_kind[msp];
      // the proposals of every level: beside the node set-up, or now
      if (fixed) {
        node_initialize(s, m, scale, epoch, mynode ? msp : -1, &status, cache, ifirst1, ipart,
                        P.seed, att, s.dr ? nullptr : llt);
      } else {
        __syncthreads();
        if (!s.dr && threadIdx.x < 32) mover_all(s, m, ipart, P.seed, att, llt);
      }
      __syncthreads();
      pimc_move_record* rec = P.rec ? P.rec + (size_t)r * P.nattempt + a : nullptr;
      double oldDS = 0.0;
      int reject = -1;
      // The top levels (L down to lb) are evaluated together, their Slater
      // matrices side by side; the decisions then follow level by level exactly as
      // below.  Work done for levels under a rejection is discarded.  Without node
      // work or Ewald sums that is every level, or what fits a warp
      // (lowest_joint_level); else the lower levels, whose
      // slices make up most of the work, wait for the decisions above them (the
      // mixed form's FP32 action terms are cheap and all come with the top ones).
      // (with delayed rejection every level is taken in turn: a second proposal
      // at level L - 1 changes the normals and uniforms of the levels under it)
      const bool longr = s.ewald && s.coulomb, waits = mynode || longr;
      const int lb = s.dr ? L + 1 : (waits ? max(1, L - 3) : lowest_joint_level(L, np));
      const int alb = s.mixed && waits ? 0 : lb;  // the lowest level whose action comes with them
      if (lb <= L) {
        eval_levels(s, m, scale[msp], msp, ipart, lb, L, alb, L, mynode, cache, ifirst1,
                    epoch[msp], lds, lnd);
        if (threadIdx.x < 32) {
          // Lane i takes level L - i: every level's acceptance probability
          // exp(lnT - total + total of the level above) and uniform at once
          // (the same operations as one level after the other); the first
          // rejecting level from the top decides, and only the levels down to
          // it count as evaluated.
          const int lane = threadIdx.x, level = L - lane;
          const bool mine = level >= lb;
          double total = 0.0, ds = 0.0, dsn = 0.0, lnT = 0.0;
          bool rej = false;
          if (mine) {
            ds = lds[level];
            dsn = lnd[level];
            lnT = llt[level];
            total = fixed ? ds + dsn : ds;
            const double old =
                level == L ? 0.0 : (fixed ? lds[level + 1] + lnd[level + 1] : lds[level + 1]);
            const uint32_t ubase = level_uniform_base(s, level);
            const uint32_t nmov = (level == L) ? 0u : (1u << (L - level - 1));
            const uint32_t uacc = ubase + (s.mover == PIMC_MOVER_FREE_PBC ? 3u * nmov : 0u);
            const double p = exp(lnT + (-total + old));
            const double u = stream_uniform(P.seed, s.stream_id, att, uacc);
            rej = u > p;
          }
          const unsigned rmask = __ballot_sync(0xffffffffu, rej);
          const int last = rmask ? __ffs(rmask) - 1 : L - lb;  // lowest evaluated lane's index
          const bool evaluated = mine && lane <= last;
          if (evaluated && rec) {
            rec->ds[level] = ds;
            rec->ds_node[level] = dsn;
            rec->lnt[level] = lnT;
          }
          const bool bad = evaluated && !(isfinite(lnT) && isfinite(ds));
          if (__ballot_sync(0xffffffffu, bad) && lane == 0) status |= PIMC_STATUS_NONFINITE;
          if (lane == last) {
            if (rmask) m.ictl[C_REJECT] = level;
            m.red[kWarps + 2] = total;
          }
        }
        __syncthreads();
        reject = m.ictl[C_REJECT];
        oldDS = m.red[kWarps + 2];
      }
      int oshift = 0;   // moved-slice orders and uniforms a delayed-rejection
      uint32_t ushift = 0;  // proposal took before the level
#pragma unroll 1
      for (int level = min(L, lb - 1); level >= 0 && reject < 0; --level) {
        const uint32_t ubase = level_uniform_base(s, level) + ushift;
        const double lnT = s.dr ? mover_level(s, m, ipart, level, oshift) : llt[level];
        const bool done = level >= alb && lb <= L;
        eval_levels(s, m, scale[msp], msp, ipart, level, level, done ? 1 : level, done ? 0 : level,
                    mynode, cache, ifirst1, epoch[msp], lds, lnd);
        double ds = lds[level];
        if (longr && level == 0) {
          if (ek)
            ds += ewald_level0_cached(s, m, ipart, ifirst1, ek, ekstage);
          else
#pragma unroll 1
            for (int t = 1; t < nsec - 1; ++t) ds += ewald_slice_diff(s, m, ipart, t);
        }
        const double dsn = lnd[level];
        if (threadIdx.x == 0) {
          const double total = fixed ? ds + dsn : ds;
          const uint32_t nmov = (level == L) ? 0u : (1u << (L - level - 1));
          const uint32_t uacc =
              ubase + (s.mover == PIMC_MOVER_FREE_PBC ? 3u * nmov : 0u);
          const double p = exp(lnT + (-total + oldDS));
          const double u = stream_uniform(P.seed, s.stream_id, att, uacc);
          if (rec) {
            rec->ds[level] = ds;
            rec->ds_node[level] = dsn;
            rec->lnt[level] = lnT;
          }
          if (!(isfinite(lnT) && isfinite(ds))) status |= PIMC_STATUS_NONFINITE;
          if (u > p) m.ictl[C_REJECT] = level;
          m.red[kWarps + 2] = total;
          m.red[kWarps + 3] = -total + oldDS;  // piRatioBoA
          m.red[kWarps + 4] = p;               // accRatioA2B
        }
        __syncthreads();
        reject = m.ictl[C_REJECT];
        if (reject == L - 1 && s.dr) {
          const uint32_t nmov = 1u << (L - level - 1);
          const uint32_t uacc = ubase + (s.mover == PIMC_MOVER_FREE_PBC ? 3u * nmov : 0u);
          delayed_rejection(s, m, scale[msp], msp, ipart, mynode, cache, ifirst1, epoch[msp],
                            P.seed, att, uacc, oldDS, ek, ekstage, rec, &status);
          reject = m.ictl[C_REJECT];
          oshift = 1;
          ushift = 1;
        }
        if (reject >= 0) break;
        oldDS = m.red[kWarps + 2];
      }
      if (reject < 0) {
#pragma unroll 1
        for (int t = threadIdx.x; t < nsec; t += blockDim.x) {
          m.s1x[t * np + ipart] = m.mx[t];
          m.s1y[t * np + ipart] = m.my[t];
          m.s1z[t * np + ipart] = m.mz[t];
        }
        if (threadIdx.x == 0) ++nacc;
        if (ek) {  // the moved slices' structure factors: the staged level-0 values
          const int totk = s.totk;
#pragma unroll 1
          for (int tt = threadIdx.x >> 5; tt < nsec - 2; tt += blockDim.x >> 5)
            copy_warp((longlong2*)ek + (size_t)wrap_slice(ifirst1 + 1 + tt, M) * totk,
                      (const longlong2*)ekstage + (size_t)tt * totk, totk);
        }
        if (cache && mynode) {
          // The moved slices now hold the level evaluations; the entries that
          // pair them the other way round (r2 on a moved slice) are stale.
          const int n = s.spec_count[msp], jcol = ipart - s.spec_first[msp];
          const int nsm = s.ns_max;
          const double NaN = __longlong_as_double(0x7ff8000000000000LL);
          const bool sho = s.node_kind[msp] == PIMC_NODES_SHO;
#pragma unroll 1
          for (int it = threadIdx.x; it < (nsec - 2) * n; it += blockDim.x) {
            const int k = 1 + it / n, j = it - (k - 1) * n;
            const int t1 = wrap_slice(ifirst1 + k, M);
            double* e = cache_entry(s, cache, msp, t1);
            const double* nc = m.ncol + k * m.ncol_stride + j;
            double c[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) c[q] = sho && q ? 0.0 : nc[q * n];
            e[2 + j] = m.ndist[(k * 2) * nsm + j];
            e[2 + n + j] = m.ndist[(k * 2 + 1) * nsm + j];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (!sho || q == 0) e[2 + 2 * n + q * n * n + jcol * n + j] = c[q];
          }
          if (sm_species(s, msp) && m.xstage) {
            // the moved slices' inverse blocks, as the level evaluations left them
            const int xw = n * n + 2, xs = cache_x_slot(s, msp);
#pragma unroll 1
            for (int k = 1 + (threadIdx.x >> 5); k < nsec - 1; k += blockDim.x >> 5)
              copy_warp(cache_entry(s, cache, msp, wrap_slice(ifirst1 + k, M)) + xs,
                        m.xstage + (size_t)k * m.xstage_stride, xw);
          }
          __syncthreads();
#pragma unroll 1
          for (int k = 1 + threadIdx.x; k < nsec - 1; k += blockDim.x) {
            const int t1 = wrap_slice(ifirst1 + k, M);
            double* e = cache_entry(s, cache, msp, t1);
            e[1] = m.ndm[k];
            e[0] = (double)epoch[msp];
            double* o = cache_entry(s, cache, msp, (t1 + M / 2) % M);
            o[0] = NaN;
            const int ms = cache_mask_slot(s, msp);
            o[ms] = __longlong_as_double(__double_as_longlong(o[ms]) | (1ll << jcol));
          }
        }
      }
      if (threadIdx.x == 0 && rec) {
        rec->ifirst1 = ifirst1;
        rec->ifirst2 = ifirst2;
        rec->ipart = ipart;
        rec->reject_level = reject;
      }
      __syncthreads();
      // SerialPaths::putBeads / putDoubleBeads (src/base/SerialPaths.cc:143-205).
      // The sections come back unchanged but for the moving particle's interior
      // beads of section 1 when the move was accepted, so only those are
      // written, unless the two sections overlap beyond their end slices
      // (2^L > M/2), where pi-qmc's put order decides which copy a shared
      // slice keeps and both sections are written in that order.
      if (fixed && (1 << L) > M / 2) {
        if (ifirst1 < M / 2 - 1) {
          store_section(s, path, ifirst1, m.s1x, m.s1y, m.s1z);
          __syncthreads();
          store_section(s, path, ifirst2, m.s2x, m.s2y, m.s2z);
        } else {
          store_section(s, path, ifirst2, m.s2x, m.s2y, m.s2z);
          __syncthreads();
          store_section(s, path, ifirst1, m.s1x, m.s1y, m.s1z);
        }
      } else if (reject < 0) {
#pragma unroll 1
        for (int k = 1 + threadIdx.x; k < nsec - 1; k += blockDim.x) {
          const int islice = ifirst1 + k;
          if (islice < 0) continue;
          const int t = islice < M ? islice : islice % M;
          double* dst = path + ((size_t)t * np + ipart) * 3;
          dst[0] = m.s1x[k * np + ipart];
          dst[1] = m.s1y[k * np + ipart];
          dst[2] = m.s1z[k * np + ipart];
        }
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      P.state[r].attempt = att0 + (uint32_t)nat;
      P.state[r].status = status;
      P.state[r].accepted += nacc;
      P.state[r].attempted += nat;
#pragma unroll 1
      for (int k = 0; k < kMaxSpecies; ++k) {
        P.state[r].node_scale[k] = scale[k];
        P.state[r].epoch[k] = epoch[k];
      }
    }
    __syncthreads();
  }
}

}  // namespace pimc

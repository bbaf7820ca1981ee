// The bisection section-move kernel: one CTA advances one replica through a
// sequence of section-move attempts, entirely on the device.
//
// Per attempt (pi-qmc order: SectionChooser.cc:30-48, DoubleSectionChooser.cc:33-65):
//   SectionChooser::run / DoubleSectionChooser::run   -> choose section(s), stage in smem
//   FixedNodeAction::initialize                        -> det + distances on every slice
//   SimpleParticleChooser::chooseParticles             -> moving particle
//   MultiLevelSampler::tryMove / DoubleMLSampler::tryMove, levels L..0:
//       FreeMover(PBC)::makeMove, CompositeAction::getActionDifference,
//       FixedNodeAction::getActionDifference, Metropolis test
//   SerialPaths::putBeads / putDoubleBeads             -> section(s) back to HBM
//
// Random numbers come from the counter-addressed streams of pimc_rng.h, so the
// CPU checkers can replay exactly the numbers a replica consumed.
#pragma once
#include "pimc_device.cuh"

namespace pimc {

// Shared-memory working set of one CTA (carved from dynamic shared memory).
struct Smem {
  double *s1x, *s1y, *s1z;  // section 1: [nsec][npart]
  double *s2x, *s2y, *s2z;  // section 2 (fixed node)
  double *mx, *my, *mz;     // moving beads [nsec]
  double* red;              // reduction scratch
  double* old;              // [2^L] the mover's terms of the old beads, by moved slice
  double* act;              // per-warp buffers of the action differences (actions.cuh)
  int act_stride;           // doubles per warp
  int nshare;               // warps that sums are shared out to: the block's, or of a larger
                            // block, whose shares this one takes several at a time
  double* dm;               // [nspecies][nsec] determinants at section set-up
  double* ndm;              // [nsec] determinants of the moving species' new slices
  double* dist;             // [nsec][2][ns_max] distances at set-up (moving species)
  double* ndist;            // [nsec][2][ns_max] distances of the new path
  double* ewt;              // Ewald exp(ik.r) tables: [kx, ky, kz rows][ewt_cols]
  double* ewx;              // the level-0 Ewald term's tables,
  int ewx_words;            // and their room
  double* ewxy;             // estimators: [kx, ky][npart] products of the tables, or null
  double* qpart;            // [npart] charges
  int* ictl;                // control words
  double* nodescr;          // per-warp node scratch (smem or global)
  double* ecache;           // [nsec][n*n] exp matrices of the moving species (SHONodes)
  double* ncol;             // [nsec][ncol_stride] recomputed column of each changed slice
  int ncol_stride;          // ns_max (SHO exp column) or 4 ns_max (free-particle values + gradients)
  double* nrm;              // [2^L - 1][3] the attempt's proposal normals
  int nodescr_stride;       // doubles per warp
  bool wide;                // wider lane groups where warps would idle
  double* nodecold;         // cold parts of the node scratch when apart (global), or null
  int nodecold_stride;      // doubles per warp
  int node_cold_follows;    // each group's cold part follows its hot part
  int ewt_cols;             // bead columns of the Ewald tables area
  double* xstage;           // mixed form: [nsec][xstage_stride] inverse blocks (global), or null
  int xstage_stride;
};


enum {
  C_IFIRST1 = 0, C_IFIRST2, C_IPART, C_REJECT, C_FLAG, C_NMISS, C_NCTL = 16
};

// Positions of particle p on section slice t, with the moving bead substituted.
struct SliceView {
  const double *sx, *sy, *sz;
  int npart;
  int t;
  int imov;  // substituted particle or -1
  double mxv, myv, mzv;
  __device__ __forceinline__ void get(int p, double& x, double& y, double& z) const {
    if (p == imov) {
      x = mxv;
      y = myv;
      z = mzv;
    } else {
      const int o = t * npart + p;
      x = sx[o];
      y = sy[o];
      z = sz[o];
    }
  }
};

// a / m for 0 <= a < 2048, 1 <= m <= 32 (an integer division takes some 25 instructions)
struct SmallReciprocals {
  unsigned v[33];
  constexpr SmallReciprocals() : v{} {
    for (unsigned m = 1; m <= 32; ++m) v[m] = (65536u + m - 1u) / m;
  }
};
static __constant__ SmallReciprocals kSmallReciprocals;
__device__ __forceinline__ int small_div(int a, int m) {
  return (int)(((unsigned)a * kSmallReciprocals.v[m]) >> 16);
}

// ------------------------------------------------------------------ node model
// The mixed form's Sherman-Morrison updates of cached inverses: at most
// kSmRefresh updates between two factorisations of a slice pair's matrix, and
// none whose determinant ratio is below kSmMinRatio in magnitude.
// A factorisation whose conditioning estimate n max|a| max|inv| exceeds
// kSmMaxCond starts no updates: an update's relative error grows with the
// condition number (the SHONodes matrices of a cold dot reach 1e13 and more).
constexpr double kSmRefresh = 16.0;
constexpr double kSmMinRatio = 0.05;
constexpr double kSmMaxCond = 1e7;
// Scratch doubles one lane group needs for an n-particle species: a hot part
// (the LU and the inverse, rewritten at every elimination step (the inverse's place
// later takes 8 n sums), the reciprocal pivots and the row order), and, for evaluations whose elements are not in a cache
// entry, a cold part (the SHO exp matrix, or the free-particle gradient matrices:
// written once, read once).
__host__ __device__ constexpr int node_group_inverse(int n) { return (n < 8 ? 8 : n) * n; }
__host__ __device__ constexpr int node_group_hot(int n) {
  return n * n + node_group_inverse(n) + n + (n + 1) / 2 + 1;
}
__host__ __device__ constexpr int node_group_cold(int n, bool free_nodes = true) {
  return n * n + (free_nodes ? 3 * n * n : 0);
}
__host__ __device__ constexpr int node_group_scratch(int n, bool free_nodes = true) {
  return node_group_hot(n) + node_group_cold(n, free_nodes);
}

// Slater scratch of a lane group: the hot part (with the cold part after it where
// the layout has one there) and the cold part.  slot counts the groups of every
// warp, G to a warp.
__device__ __forceinline__ double* group_scr(const Smem& m, int slot, int G, int n, bool free_nodes) {
  return m.nodescr + (size_t)(slot / G) * m.nodescr_stride +
         (slot % G) * (m.node_cold_follows ? node_group_scratch(n, free_nodes) : node_group_hot(n));
}
__device__ __forceinline__ double* group_cold(const Smem& m, int slot, int G, int n, bool free_nodes) {
  return m.nodecold ? m.nodecold + (size_t)(slot / G) * m.nodecold_stride +
                          (slot % G) * node_group_cold(n, free_nodes)
                    : nullptr;
}

// *dst = *src, asynchronously where the hardware can (global to shared); complete
// for the lane after copy_wait, for the others after a barrier too.
__device__ __forceinline__ void copy_async(double* dst, const double* src) {
#ifdef __CUDA_ARCH__
  if (__isShared(dst) && __isGlobal(src)) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(__cvta_generic_to_global(src))
                 : "memory");
    return;
  }
#endif
  *dst = *src;
}
__device__ __forceinline__ void copy_wait() {
#ifdef __CUDA_ARCH__
  asm volatile("cp.async.wait_all;" ::: "memory");
#endif
}

__device__ __forceinline__ bool in_shared(const double* p) {
#ifdef __CUDA_ARCH__
  return __isShared(p);
#else
  return true;
#endif
}
__device__ __forceinline__ void prefetch_l2(const double* p) {
#ifdef __CUDA_ARCH__
  asm volatile("prefetch.global.L2 [%0];" ::"l"(__cvta_generic_to_global(p)));
#endif
}

// One element rho(r1_j, r2_i) of a species' Slater matrix (unscaled), and for
// free-particle nodes its gradient with respect to r1_j.  Rounded operations: the
// same bits wherever it is computed.
struct NodeElement {
  double v, gx, gy, gz;
};
__device__ __forceinline__ double sho_element(const DevSys& s, int sp, double rix, double riy,
                                              double riz, double rjx, double rjy, double rjz) {
  const double ri2 = dot3(rix, riy, riz, rix, riy, riz);
  const double rj2 = dot3(rjx, rjy, rjz, rjx, rjy, rjz);
  const double rirj = dot3(rix, riy, riz, rjx, rjy, rjz);
  const double q = __dsub_rn(__dmul_rn(__dadd_rn(ri2, rj2), s.node_cosh[sp]),
                             __dmul_rn(2.0, rirj));
  return exp(__dmul_rn(-s.node_c[sp], q));
}
// (a call: boxes too small for pg_images_eval)
static __device__ __noinline__ NodeElement pg_series_element(const DevSys& s, int sp, double dx,
                                                             double dy, double dz) {
  double v[3], g[3];
  const double d[3] = {dx, dy, dz};
#pragma unroll 1
  for (int a = 0; a < 3; ++a)
    v[a] = pg_eval(s.pg_nome[sp][a], s.pg_pref[sp][a], s.pg_k[sp][a], s.pg_nmax[sp][a], d[a], &g[a]);
  NodeElement r;
  r.v = v[0] * v[1] * v[2];
  r.gx = g[0] / (v[0] + 1e-300) * v[0] * v[1] * v[2];
  r.gy = g[1] / (v[1] + 1e-300) * v[0] * v[1] * v[2];
  r.gz = g[2] / (v[2] + 1e-300) * v[0] * v[1] * v[2];
  return r;
}
__device__ __forceinline__ NodeElement free_element(const DevSys& s, int sp, double dx, double dy,
                                                    double dz) {
  pbc(s, dx, dy, dz);
  if (!s.pg_images[sp]) return pg_series_element(s, sp, dx, dy, dz);
  NodeElement r;
  r.v = pg_images_eval(s, sp, dx, dy, dz, r.gx, r.gy, r.gz);
  return r;
}
template <bool kSho>
__device__ __forceinline__ NodeElement node_element(const DevSys& s, int sp, const SliceView& v1,
                                                    const SliceView& v2, int i, int j) {
  const int f = s.spec_first[sp];
  double rix, riy, riz, rjx, rjy, rjz;
  v2.get(f + i, rix, riy, riz);
  v1.get(f + j, rjx, rjy, rjz);
  if constexpr (kSho)
    return NodeElement{sho_element(s, sp, rix, riy, riz, rjx, rjy, rjz), 0.0, 0.0, 0.0};
  else
    return free_element(s, sp, rjx - rix, rjy - riy, rjz - riz);
}

// NodeModel::evaluate (+ evaluateDistance) for one species on one slice pair,
// executed by a group of W >= n lanes (W = 8, 16 or 32; 32/W groups per warp each
// take their own slice pair).  LU with
// partial pivoting (first largest |pivot|, LAPACK dgetrf semantics), determinant from
// the U diagonal and pivots, inverse (dgetri semantics: the forward substitution runs
// with the elimination, on the columns of the identity its row interchanges have
// reached), then the log-gradient nodal distances
// (src/fixednode/SHONodes.cc:51-170, src/fixednode/FreeParticleNodes.cc:72-234).
// full = 0: determinant only.  Every lane of the warp must call this (the
// shuffles span the warp); a group with write = false computes but stores
// nothing.  ecache (or null) holds the slice pair's element matrix: the rows of
// rowmask are recomputed, and the columns of `cols` in the other rows (their
// other inputs are unchanged, so the values are bit-identical); without columns
// what is recomputed is stored there, a single column goes to newcol.
// kSho: SHONodes (else FreeParticleNodes).  kSm: the variant with the mixed form's
// Sherman-Morrison updates and inverse blocks (xin / xout); without it those
// arguments are ignored and the evaluation is the plain factorisation.
//
// FP64 bound: every step deals single elements to the lanes, so that a warp
// instruction, which costs the SM the same whatever its lanes, has few idle ones.
// Cached elements are read where they are used, straight from the entry, in
// coalesced order; only a factorisation copies them (scaled).  The loops are not
// unrolled and the models are apart: left to the compiler, one instance was 209 KB of
// code, and warps in different phases waited for instructions.  A step of 304
// fixed-node dots 157 -> 139 ms, of 152 electron gases 84 -> 62 ms.  (Two particles'
// rows to a lane, four 10 x 10 matrices a warp on half the warps, would take 20 % fewer
// FP64 instructions and measured 6 % more time.)
template <int W, bool kSho, bool kSm = false>
static __device__ __noinline__ void node_eval_group(const DevSys& s, int sp, const SliceView& v1,
                                const SliceView& v2, double scale, double* scr, int full,
                                double* ecache, unsigned cols, bool write, double& det_out,
                                int& err_out, double* d1, double* d2,
                                double* newcol = nullptr, unsigned rowmask = 0xffffffffu,
                                double* cold = nullptr, const double* xin = nullptr,
                                double det_in = 0.0, double* xout = nullptr,
                                double xepoch = 0.0) {
  constexpr unsigned FULL = 0xffffffffu;
  const int gl = threadIdx.x & (W - 1);
  const int n = s.spec_count[sp];
  const int f = s.spec_first[sp];
  // hot part at scr; the cold part follows it unless given apart
  double* A = scr;          // n*n column-major, LU; after the inverse: work space
  double* X = A + n * n;    // n*n inverse, column-major
  double* R = X + node_group_inverse(n);  // n reciprocals of the U diagonal
  int* order = (int*)(R + n + 1);  // the matrix row at each position; then its inverse
  double* E = cold ? cold : scr + node_group_hot(n);  // elements (and gradients) without a place
  constexpr bool sho = kSho;
  const int nn = n * n;
  const unsigned nmask = n >= 32 ? 0xffffffffu : ((1u << n) - 1u);
  const unsigned rows_new = !ecache ? nmask : (rowmask & nmask);
  // --- build the Slater matrix: A(i,j) = scale * rho(r1_j, r2_i).  The new elements
  // are computed, one per lane and step (whole rows, then the new columns of the
  // other rows); the others follow when the matrix is factorised.  Every element is
  // the same rounded arithmetic wherever it is computed, so cached and recomputed
  // values agree bit for bit.
  const bool to_cache = ecache && !cols, to_col = ecache && cols && newcol;
  // component c (0: value, 1 .. 3: gradient) of element (i, j), k = j n + i
  auto elem = [&](int c, int i, int j, int k) -> double {
    if (!ecache) return E[c * nn + k];
    if (cols && (((cols >> j) | (rows_new >> i)) & 1u)) return newcol ? newcol[c * n + i] : E[c * nn + k];
    return ecache[c * nn + k];
  };
  auto element = [&](int i, int j) {
    const NodeElement v = node_element<kSho>(s, sp, v1, v2, i, j);
    double* at = to_cache ? ecache + j * n + i : (to_col ? newcol + i : E + j * n + i);
    const int step = to_col ? n : nn;
    if (!to_cache || write) {
      at[0] = v.v;
      if (!sho) {
        at[step] = v.gx;
        at[2 * step] = v.gy;
        at[3 * step] = v.gz;
      }
    }
    A[j * n + i] = scale * v.v;
  };
  // (mixed form: the cached inverse is on its way to X meanwhile, the gradients to L2)
  bool good = false;
  if (kSm && xin) {
    good = xin[0] == xepoch && xin[1] < kSmRefresh;
#pragma unroll 4
    for (int k = gl; k < nn; k += W) copy_async(X + k, xin + 2 + k);
    if (!sho && ecache)
#pragma unroll 1
      for (int k = 16 * gl; k < 3 * nn; k += 16 * W) prefetch_l2(ecache + nn + k);
  }
  {
    const int nrows = __popc(rows_new), ncols = ecache ? __popc(cols & nmask) : 0;
#pragma unroll 1
    for (int e = gl; e < (nrows + ncols) * n; e += W) {
      // the q-th new row's element in column x, then the new columns' in row x
      int q = small_div(e, n);
      const int x = e - q * n;
      const bool row = q < nrows;
      unsigned bits = row ? rows_new : cols & nmask;
#pragma unroll 1
      for (q = row ? q : q - nrows; q > 0; --q) bits &= bits - 1u;  // drop the first q
      const int b = __ffs(bits) - 1;
      if (row || !((rows_new >> x) & 1u)) element(row ? b : x, row ? x : b);
    }
  }
  __syncwarp();
  int info = 0;
  // --- the mixed form: Sherman-Morrison updates of the cached inverse (xin:
  // its [epoch, updates, inverse] block) instead of a factorisation, for the
  // new column jcol of a level evaluation or each changed row of a refresh.
  // A group updates when its block is of the current scale (epoch), has had
  // fewer than kSmRefresh updates since its last factorisation, and every
  // determinant ratio is at least kSmMinRatio in magnitude (a refresh: at most
  // n/2 rows); otherwise, or when another writing group of the warp cannot,
  // the warp factorises as below.  Every lane takes part in the shuffles.
  bool use_sm = false;
  // (a warp none of whose writing groups can update factorises at once)
  if (kSm && __any_sync(FULL, good && write) && __all_sync(FULL, good || !write)) {
    copy_wait();
    __syncwarp();
    double det = det_in;
    if (cols) {
      const int jcol = __ffs(cols) - 1;  // (a level evaluation: one column)
      // column jcol replaced by u = A(:, jcol): w = inv u, ratio = w_jcol,
      // inv'(a, b) = inv(a, b) - (w_a - [a = jcol]) inv(jcol, b) / ratio
      double w = 0.0;
      if (gl < n)
#pragma unroll 1
        for (int i = 0; i < n; ++i) w = __fma_rn(X[i * n + gl], A[jcol * n + i], w);
      const double ratio = __shfl_sync(FULL, w, jcol, W);
      good = good && fabs(ratio) >= kSmMinRatio;
      use_sm = __all_sync(FULL, good || !write);
      if (use_sm) {
        const double rj = gl < n ? X[gl * n + jcol] : 0.0;  // inv(jcol, b), b = gl
        const double f = gl < n ? (w - (gl == jcol ? 1.0 : 0.0)) / ratio : 0.0;
        __syncwarp();
#pragma unroll 1
        for (int e0 = 0; e0 < nn; e0 += W) {
          const int e = e0 + gl;
          const bool on = e < nn;
          const int b = on ? small_div(e, n) : 0, a = on ? e - b * n : 0;
          const double fa = __shfl_sync(FULL, f, a, W);
          const double rb = __shfl_sync(FULL, rj, b, W);
          if (on) X[b * n + a] = __fma_rn(-fa, rb, X[b * n + a]);
        }
        det = __dmul_rn(det_in, ratio);
      }
    } else {
      // each changed row i in turn, v = A(i, :): z = v inv, ratio = z_i,
      // inv'(a, b) = inv(a, b) - inv(a, i) (z_b - [b = i]) / ratio
      const int nr = __popc(rows_new);
      good = good && nr > 0 && 2 * nr <= n;
      const unsigned nrmax = __reduce_max_sync(FULL, good ? (unsigned)nr : 0u);
      unsigned rm = good ? rows_new : 0u;
#pragma unroll 1
      for (unsigned k = 0; k < nrmax; ++k) {
        const bool live = rm != 0u;
        const int i = live ? __ffs(rm) - 1 : 0;
        rm &= rm - 1u;
        double z = 0.0;
        if (gl < n)
#pragma unroll 1
          for (int j = 0; j < n; ++j) z = __fma_rn(A[j * n + i], X[gl * n + j], z);
        const double ratio = __shfl_sync(FULL, z, i, W);
        const double ci = gl < n ? X[i * n + gl] : 0.0;  // inv(a, i), a = gl
        const double g = gl < n ? (z - (gl == i ? 1.0 : 0.0)) / ratio : 0.0;
        __syncwarp();
#pragma unroll 1
        for (int e0 = 0; e0 < nn; e0 += W) {
          const int e = e0 + gl;
          const bool on = e < nn && live;
          const int b = e < nn ? small_div(e, n) : 0, a = e < nn ? e - b * n : 0;
          const double ca = __shfl_sync(FULL, ci, a, W);
          const double gb = __shfl_sync(FULL, g, b, W);
          if (on) X[b * n + a] = __fma_rn(-ca, gb, X[b * n + a]);
        }
        __syncwarp();
        if (live) {
          det = __dmul_rn(det, ratio);
          good = good && fabs(ratio) >= kSmMinRatio;
        }
      }
      use_sm = __all_sync(FULL, good || !write);
    }
    if (use_sm && write) {
      det_out = det;
      err_out = 0;
    }
  }
  if (kSm && !use_sm) {  // (X is about to be overwritten)
    copy_wait();
    __syncwarp();
  }
  double amax = 0.0;  // max |a| of the matrix, for the conditioning estimate (mixed form)
  // every lane takes part in the shuffles
  const bool xany = kSm && __any_sync(FULL, xout != nullptr);
  if (!use_sm) {
  if (ecache) {
    // the cached elements (four loads in flight a lane)
    int j = small_div(gl, n), i = gl - j * n;
    const int dj = small_div(W, n), di = W - dj * n;
#pragma unroll 1
    for (int k0 = gl; k0 < nn; k0 += 4 * W) {
      double v[4];
      unsigned have = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (k0 + q * W < nn && !(((cols >> j) | (rows_new >> i)) & 1u)) {
          v[q] = ecache[k0 + q * W];
          have |= 1u << q;
        }
        i += di;
        j += dj;
        if (i >= n) {
          i -= n;
          ++j;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if ((have >> q) & 1u) A[k0 + q * W] = scale * v[q];
    }
  }
#pragma unroll 1
  for (int k = gl; k < nn; k += W) X[k] = 0.0;
  if (gl < n) order[gl] = gl;
  __syncwarp();
  if (xany) {
#pragma unroll 1
    for (int k = gl; k < nn; k += W) amax = fmax(amax, fabs(A[k]));
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(FULL, amax, o, W));
  }
  // --- LU with partial pivoting (the pivot is the first largest |a|), the identity's
  // columns beside the matrix: X holds one column per position, in the order in
  // which the row interchanges bring the rows up, so that step j works on the n
  // consecutive columns j + 1 .. j + n of [A | X].
  unsigned pivbits = 0;  // parity of the interchanges
#pragma unroll 1
  for (int j = 0; j < n; ++j) {
    // the largest |a| on the integer pipe: bit patterns of non-negative doubles are
    // ordered like them.  First the upper 26 bits with the row below them (the
    // smallest row wins a tie); where two rows share those, the whole patterns.
    const bool live = gl >= j && gl < n;
    const double aj = live ? A[j * n + gl] : 0.0;
    const unsigned mine =
        live ? (((unsigned)__double2hiint(aj) << 1) & ~63u) | (unsigned)(32 - gl) : 0u;
    unsigned key = mine;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) key = max(key, __shfl_xor_sync(FULL, key, o, W));
    int p = 32 - (int)(key & 63u);
    if (__any_sync(FULL, live && gl != p && ((mine ^ key) >> 6) == 0)) {
      long long av = live ? (__double_as_longlong(aj) & 0x7fffffffffffffffLL) : -1LL;
      p = gl;
#pragma unroll
      for (int o = W / 2; o > 0; o >>= 1) {
        const long long ov = __shfl_xor_sync(FULL, av, o, W);
        const int oi = __shfl_xor_sync(FULL, p, o, W);
        if (ov > av || (ov == av && oi < p)) {
          av = ov;
          p = oi;
        }
      }
    }
    const double apj = A[j * n + p];
    const bool regular = (__double_as_longlong(apj) & 0x7fffffffffffffffLL) != 0;  // apj != 0
    __syncwarp();  // (every lane has it: the interchange moves it)
    if (regular) {
      // (the reciprocal starts on its way beside the interchange)
      const double rinv = reciprocal(apj);
      if (p != j) {
        pivbits ^= 1u;
        if (gl < n) {  // rows j and p of columns j .. j + n - 1
          double* col = A + (j + gl) * n;
          const double t = col[j];
          col[j] = col[p];
          col[p] = t;
        }
      }
      if (gl == 0) {
        const int t = order[j];
        order[j] = order[p];
        order[p] = t;
        X[j * n + j] = 1.0;
        R[j] = rinv;
      }
      __syncwarp();
      if (gl > j && gl < n) A[j * n + gl] *= rinv;
    } else {
      if (info == 0) info = j + 1;
      __syncwarp();
    }
    __syncwarp();
    // elimination, one element per lane and step, the operands of two steps loaded at
    // a time: a(i,k) -= l(i,j) u(j,k).  Each element takes the same FMAs in the same
    // order as a factorisation and a solve per column.
    const int m = n - j - 1, cnt = full ? m * n : m * m;
    if (m > 0) {
      const double* l = A + j * n + j + 1;
      double* c0 = A + (j + 1) * n + j;  // row j of the first column
      const int dk = small_div(W, m), di = W - dk * m, step = dk * n + di;
      int k0 = small_div(gl, m), ii = gl - k0 * m, at = k0 * n + ii;
#pragma unroll 1
      for (int e = gl; e < cnt; e += 2 * W) {
        const bool two = e + W < cnt;
        const int i0 = ii, a0 = at;
        ii += di;
        at += step;
        if (ii >= m) {
          ii -= m;
          at += n - m;
        }
        const double l0 = l[i0], u0 = c0[a0 - i0], x0 = c0[a0 + 1];
        if (two) {
          const double l1 = l[ii], u1 = c0[at - ii], x1 = c0[at + 1];
          c0[at + 1] = __fma_rn(-l1, u1, x1);
        }
        c0[a0 + 1] = __fma_rn(-l0, u0, x0);
        ii += di;
        at += step;
        if (ii >= m) {
          ii -= m;
          at += n - m;
        }
      }
    }
    __syncwarp();
  }
  // --- determinant (sequential product, as the reference; the interchanges' signs
  // are exact wherever they come in)
  double det = 1.0;
#pragma unroll 4
  for (int i = 0; i < n; ++i) det = __dmul_rn(det, A[i * n + i]);
  if (pivbits) det = __longlong_as_double(__double_as_longlong(det) ^ (long long)0x8000000000000000ULL);
  if (write) {
    det_out = det;
    err_out = info != 0;
  }
  if (!full) return;  // the same for every group of the warp
#pragma unroll 1
  for (int j = n - 1; j >= 0; --j) {  // back: x(j) *= 1/u(j,j); x(i) -= u(i,j) x(j), i < j
    const double rj = R[j];
    if (gl < n) X[gl * n + j] *= rj;
    __syncwarp();
    if (j > 0) {
      const int dc = small_div(W, j), di = W - dc * j, step = dc * n + di, cnt = n * j;
      int c0 = small_div(gl, j), ii = gl - c0 * j, at = c0 * n + ii;
      const double* u = A + j * n;
#pragma unroll 1
      for (int e = gl; e < cnt; e += 2 * W) {
        const bool two = e + W < cnt;
        const int i0 = ii, a0 = at;
        ii += di;
        at += step;
        if (ii >= j) {
          ii -= j;
          at += n - j;
        }
        const double u0 = u[i0], t0 = X[a0 - i0 + j], x0 = X[a0];
        if (two) {
          const double u1 = u[ii], t1 = X[at - ii + j], x1 = X[at];
          X[at] = __fma_rn(-u1, t1, x1);
        }
        X[a0] = __fma_rn(-u0, t0, x0);
        ii += di;
        at += step;
        if (ii >= j) {
          ii -= j;
          at += n - j;
        }
      }
    }
    __syncwarp();
  }
  // X's columns are solutions for the unit vectors order[0], order[1], ...: turned
  // into the position of each (SHONodes, whose weights follow it), or sorted
  // through A (free-particle nodes, which read the inverse more than once)
  if constexpr (kSho) {
    const int o = gl < n ? order[gl] : 0;
    __syncwarp();
    if (gl < n) order[o] = gl;
  } else {
#pragma unroll 1
    for (int c = 0; c < n; ++c)
      if (gl < n) A[order[c] * n + gl] = X[c * n + gl];
    __syncwarp();
#pragma unroll 1
    for (int k = gl; k < nn; k += W) X[k] = A[k];
  }
  __syncwarp();
  }  // factorisation
  // the inverse and its update count for the cache (mixed form); a fresh
  // factorisation that is too ill-conditioned is marked as used up
  if (xany) {
    double xmax = 0.0;
    if (!use_sm) {
#pragma unroll 1
      for (int k = gl; k < nn; k += W) xmax = fmax(xmax, fabs(X[k]));
#pragma unroll
      for (int o = W / 2; o > 0; o >>= 1) xmax = fmax(xmax, __shfl_xor_sync(FULL, xmax, o, W));
    }
    if (write && xout) {
#pragma unroll 1
      for (int k = gl; k < nn; k += W) xout[2 + k] = X[k];
      if (gl == 0) {
        xout[0] = info == 0 ? xepoch : __longlong_as_double(0x7ff8000000000000LL);
        xout[1] = use_sm ? xin[1] + 1.0
                         : (n * amax * xmax <= kSmMaxCond ? 0.0 : kSmRefresh);
      }
    }
  }
  // --- nodal distances: d = sqrt(2m / (tau |grad ln det|^2)), the gradient
  // with respect to r1_j (d1) and r2_i (d2); inv(j,i) = X[i*n + j].  (No early
  // exit: a singular group simply skips them, so the warp stays converged.)
  const double dk = s.node_dk[sp];
  const bool ok = info == 0;
  if constexpr (kSho) {
    // weights w(i,j) = inv(j,i) rho(i,j), shared by both gradients
    if (ok) {
      int j = small_div(gl, n), i = gl - j * n;
      const int dj = small_div(W, n), di = W - dj * n;
#pragma unroll 1
      for (int e0 = gl; e0 < nn; e0 += 4 * W) {  // (four loads in flight a lane)
        double v[4], x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (e0 + q * W < nn) {
            v[q] = elem(0, i, j, e0 + q * W);
            x[q] = X[order[i] * n + j];
          }
          i += di;
          j += dj;
          if (i >= n) {
            i -= n;
            ++j;
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (e0 + q * W < nn) A[e0 + q * W] = __dmul_rn(x[q], v[q]);
      }
    }
    __syncwarp();
    // d1: sum_i w(i,j) 2c (r2_i - ch r1_j), d2: sum_j w(i,j) 2c (r1_j - ch r2_i): with S the
    // sum of w r and T that of w, S - ch r T
    const double c = s.node_c[sp], ch = s.node_cosh[sp];
    const double fac = 2 * c * scale;
    double* S = X;
    // (X, spent, takes the sums, one of the 8 n per lane and step, three steps at once)
    if (ok)
#pragma unroll 1
      for (int q0 = gl; q0 < 8 * n; q0 += 3 * W) {
        const double *w[3], *x[3];
        double xm[3], sum[3];
        int dw[3], im[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int q = min(q0 + k * W, 8 * n - 1), c = q & 3, o = q >> 2;
          const bool first = o < n;
          const SliceView& v = first ? v2 : v1;
          w[k] = A + (first ? o * n : o - n);
          dw[k] = first ? 1 : n;
          // (c = 3: the sum of the weights alone, a factor of one)
          x[k] = (c == 0 ? v.sx : (c == 1 ? v.sy : v.sz)) + v.t * v.npart + f;
          xm[k] = c == 0 ? v.mxv : (c == 1 ? v.myv : (c == 2 ? v.mzv : 1.0));
          im[k] = c == 3 ? -1 : v.imov - f;
          sum[k] = 0;
        }
        const bool one = (gl & 3) == 3;  // (W and q0 - gl are multiples of 4)
#pragma unroll 1
        for (int i = 0; i < n; ++i)
#pragma unroll
          for (int k = 0; k < 3; ++k)
            if (q0 + k * W < 8 * n) {
              sum[k] = __fma_rn(*w[k], one || i == im[k] ? xm[k] : x[k][i], sum[k]);
              w[k] += dw[k];
            }
#pragma unroll
        for (int k = 0; k < 3; ++k)
          if (q0 + k * W < 8 * n) S[q0 + k * W] = sum[k];
      }
    __syncwarp();
    if (ok)
#pragma unroll 1
      for (int q = gl; q < 2 * n; q += W) {
        const bool first = q < n;
        const int p = first ? q : q - n;
        double rx, ry, rz;
        (first ? v1 : v2).get(f + p, rx, ry, rz);
        const double ct = __dmul_rn(ch, S[4 * q + 3]);
        const double lx = __dmul_rn(fac, __fma_rn(-ct, rx, S[4 * q]));
        const double ly = __dmul_rn(fac, __fma_rn(-ct, ry, S[4 * q + 1]));
        const double lz = __dmul_rn(fac, __fma_rn(-ct, rz, S[4 * q + 2]));
        const double d = __dmul_rn(dk, rsqrt(__dadd_rn(dot3(lx, ly, lz, lx, ly, lz), 1e-15)));
        if (write) (first ? d1 : d2)[p] = d;
      }
  } else {
    // The gradient matrices pass once through A (spent) in tiles of n/3 columns, read
    // coalesced: lane i adds its row for d2 (sum_j inv(j,i) dA(i,j)/dr2_i, with
    // dA/dr2_i = -dA/dr1_j), and lanes (component, j) the tile's columns for d1 (sum_i
    // inv(j,i) dA(i,j)/dr1_j), each kept by its lane until all tiles are done.
    double l2[3] = {0, 0, 0}, lx = 0, ly = 0, lz = 0;
    if (n < 3) {  // (no room for a tile: straight from the elements)
      if (gl < n)
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
          const double w1 = X[k * n + gl], w2 = X[gl * n + k];
          lx = __fma_rn(w1, elem(1, k, gl, gl * n + k), lx);
          ly = __fma_rn(w1, elem(2, k, gl, gl * n + k), ly);
          lz = __fma_rn(w1, elem(3, k, gl, gl * n + k), lz);
#pragma unroll
          for (int c = 0; c < 3; ++c) l2[c] = __fma_rn(w2, elem(1 + c, gl, k, k * n + gl), l2[c]);
        }
    } else {
      const int tw = small_div(n, 3), nt = small_div(n + tw - 1, tw);  // 3 to 5 tiles of 3 tw <= W rows
      double l1[5] = {0, 0, 0, 0, 0};
      const bool async = ecache && in_shared(A);
#pragma unroll 1
      for (int t = 0; t < nt; ++t) {
        const int j0 = t * tw, wd = min(tw, n - j0);
        __syncwarp();
        // row r = component * wd + column of the tile, element i on lane i: all rows'
        // loads in flight, or four rows' where the scratch is not in shared memory
        const int i = min(gl, n - 1);
        auto source = [&](int r) {
          const int c = 1 + (r >= wd) + (r >= 2 * wd), j = j0 + r - (c - 1) * wd;
          const double* from = (ecache ? ecache : E) + c * nn + j * n;
          if (cols && (((cols >> j) | (rows_new >> i)) & 1u))
            from = newcol ? newcol + c * n : E + c * nn + j * n;
          return from + i;
        };
        if (async) {
          if (gl < n)
#pragma unroll 1
            for (int r = 0; r < 3 * wd; ++r) copy_async(A + r * n + gl, source(r));
          copy_wait();
        } else {
#pragma unroll 1
          for (int r0 = 0; r0 < 3 * wd; r0 += 4) {
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) v[q] = *source(min(r0 + q, 3 * wd - 1));
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (r0 + q < 3 * wd && gl < n) A[(r0 + q) * n + gl] = v[q];
          }
        }
        __syncwarp();
        if (gl < n)
#pragma unroll 1
          for (int jj = 0; jj < wd; ++jj) {
            const double w = X[gl * n + j0 + jj];
#pragma unroll
            for (int c = 0; c < 3; ++c) l2[c] = __fma_rn(w, A[(c * wd + jj) * n + gl], l2[c]);
          }
        if (gl < 3 * wd) {
          const int j = j0 + gl - (gl >= wd) * wd - (gl >= 2 * wd) * wd;
          double sum = 0.0;
#pragma unroll 1
          for (int k = 0; k < n; ++k) sum = __fma_rn(X[k * n + j], A[gl * n + k], sum);
#pragma unroll
          for (int q = 0; q < 5; ++q)
            if (q == t) l1[q] = sum;
        }
      }
      // lane j takes its column's three sums from the lanes that hold them
      const int mine = min(gl, n - 1), mt = small_div(mine, tw), jj = mine - mt * tw;
#pragma unroll
      for (int t = 0; t < 5; ++t) {
        const int wd = max(1, min(tw, n - t * tw));
        const double a = __shfl_sync(FULL, l1[t], min(jj, W - 1), W);
        const double b = __shfl_sync(FULL, l1[t], min(wd + jj, W - 1), W);
        const double c = __shfl_sync(FULL, l1[t], min(2 * wd + jj, W - 1), W);
        if (t == mt) {
          lx = a;
          ly = b;
          lz = c;
        }
      }
    }
    if (ok && gl < n) {
      lx *= scale;
      ly *= scale;
      lz *= scale;
      if (write) d1[gl] = dk * rsqrt(dot3(lx, ly, lz, lx, ly, lz) + 1e-15);
      lx = l2[0] * scale;
      ly = l2[1] * scale;
      lz = l2[2] * scale;
      if (write) d2[gl] = dk * rsqrt(dot3(lx, ly, lz, lx, ly, lz) + 1e-15);
    }
  }
  __syncwarp();
}


// Group width for an n-particle species.
__host__ __device__ __forceinline__ int node_group_width(int n) {
  return n <= 8 ? 8 : (n <= 16 ? 16 : 32);
}
// The widest lane group worth its longer reductions: one that n x n elements fill.
__host__ __device__ __forceinline__ int node_group_widest(int n) {
  int w = node_group_width(n);
  while (w < 32 && n * n > 2 * w) w *= 2;
  return w;
}

// One warp evaluates one slice pair (the entry-point kernels).
static __device__ void node_eval_warp(const DevSys& s, int sp, const SliceView& v1, const SliceView& v2,
                               double scale, double* scr, int full, double& det_out,
                               int& err_out, double* d1, double* d2) {
  if (s.node_kind[sp] == 1)
    node_eval_group<32, true>(s, sp, v1, v2, scale, scr, full, nullptr, 0u, true, det_out, err_out,
                              d1, d2);
  else
    node_eval_group<32, false>(s, sp, v1, v2, scale, scr, full, nullptr, 0u, true, det_out,
                               err_out, d1, d2);
}

__device__ __forceinline__ int species_of(const DevSys& s, int p) {
  int r = 0;
  for (int k = 0; k < s.nspecies; ++k)
    if (p >= s.spec_first[k] && p < s.spec_first[k] + s.spec_count[k]) r = k;
  return r;
}

// ------------------------------------------------------------------ Ewald sums
// e^{ik.r} factor tables of one bead, column `col` of X [nx][w], Y [ny][w] and
// Z [nz][w] (Y and Z rows offset by ikmax): EwaldSum's recurrence over
// multiples of the first wave vector (src/util/EwaldSum.cc:110-150), in
// individually rounded operations, so every kernel that builds a bead's tables
// gets the same bits.
static __device__ __forceinline__ double2 cmul_rn(double2 a, double2 b) {
  return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                      __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}

static __device__ __noinline__ void ewald_axis_table(const DevSys& s, double2* T, int w, int a,
                                                     double x) {
  const int k0 = s.ikmax[a];
  if (a > 0) T += k0 * w;
  T[0] = make_double2(1.0, 0.0);
  if (k0 <= 0) return;
  double sn, cs;
  sincos(__dmul_rn(s.deltak[a], x), &sn, &cs);
  // the negative multiples of y and z are the conjugates: the recurrence of the
  // conjugate gives exactly those
  const double2 t1 = make_double2(cs, sn);
  double2 t = t1;
#pragma unroll 1
  for (int k = 1; k <= k0; ++k) {
    T[k * w] = t;
    if (a > 0) T[-k * w] = make_double2(t.x, -t.y);
    t = cmul_rn(t, t1);
  }
}

static __device__ __forceinline__ void ewald_bead_tables(const DevSys& s, double2* X, double2* Y,
                                                         double2* Z, int w, int col, double x,
                                                         double y, double z) {
#pragma unroll 1
  for (int a = 0; a < 3; ++a)
    ewald_axis_table(s, (a == 0 ? X : (a == 1 ? Y : Z)) + col, w, a, a == 0 ? x : (a == 1 ? y : z));
}

// q e^{ik.r} of table column col for k-vector k, on the fixed-point grid of the
// structure-factor cache (rounded to the nearest multiple of 1/ek_scale; qs = q ek_scale,
// exact, as the scale is a power of two).
static __device__ __forceinline__ void ewald_term_fixed(const DevSys& s, const double2* X,
                                                        const double2* Y, const double2* Z,
                                                        int w, int col, int kx, int ky, int kz,
                                                        double qs, long long& re, long long& im) {
  const double2 a = X[kx * w + col];
  const double2 t = make_double2(__dmul_rn(qs, a.x), __dmul_rn(qs, a.y));
  const double2 v = cmul_rn(cmul_rn(t, Y[ky * w + col]), Z[kz * w + col]);
  re = __double2ll_rn(v.x);
  im = __double2ll_rn(v.y);
}

// EwaldSum::evalLongRange (src/util/EwaldSum.cc:103-181) for the old and the
// new configuration of one slice (the new one has particle ipart at the moving
// bead), as CoulombAction::getActionDifference uses them at level 0
// (src/action/CoulombAction.cc:107-119).  Returns both evalLongRange values.
static __device__ void ewald_slice_sums(const DevSys& s, const Smem& m, int ipart, int t, double& eold,
                                 double& enew) {
  const int np = s.npart;
  const int kx0 = s.ikmax[0], ky0 = s.ikmax[1], kz0 = s.ikmax[2];
  const int nx = kx0 + 1, ny = 2 * ky0 + 1;
  const int w = m.ewt_cols;            // >= np + 1: column np = moved bead
  double2* X = (double2*)m.ewt;        // [nx][w]
  double2* Y = X + nx * w;             // [ny][w]
  double2* Z = Y + ny * w;             // [nz][w]
  __syncthreads();
  for (int p = threadIdx.x; p < w; p += blockDim.x) {
    if (p < np)
      ewald_bead_tables(s, X, Y, Z, w, p, m.s1x[t * np + p], m.s1y[t * np + p], m.s1z[t * np + p]);
    else
      ewald_bead_tables(s, X, Y, Z, w, p, m.mx[t], m.my[t], m.mz[t]);
  }
  __syncthreads();
  double so[2] = {0.0, 0.0}, sn_[2] = {0.0, 0.0};  // (of up to two shares)
  const bool shares = m.nshare > (int)(blockDim.x >> 5);
  for (int k = threadIdx.x; k < s.totk; k += blockDim.x) {
    const bool second = shares && ((k / blockDim.x) & 1);
    const int kx = __ldg(s.kvec + 3 * k), ky = __ldg(s.kvec + 3 * k + 1) + ky0,
              kz = __ldg(s.kvec + 3 * k + 2) + kz0;
    double cor = 0, coi = 0, cnr = 0, cni = 0;
    for (int j = 0; j < np; ++j) {
      const int jj = (j == ipart) ? np : j;
      const double qj = m.qpart[j];
      double2 a = X[kx * w + j];
      double tr = qj * a.x, ti = qj * a.y;
      double2 b = Y[ky * w + j];
      double ur = tr * b.x - ti * b.y, ui = tr * b.y + ti * b.x;
      b = Z[kz * w + j];
      const double vr = ur * b.x - ui * b.y, vi = ur * b.y + ui * b.x;
      cor += vr;
      coi += vi;
      if (jj == j) {
        cnr += vr;
        cni += vi;
      } else {
        a = X[kx * w + jj];
        tr = qj * a.x;
        ti = qj * a.y;
        b = Y[ky * w + jj];
        ur = tr * b.x - ti * b.y;
        ui = tr * b.y + ti * b.x;
        b = Z[kz * w + jj];
        cnr += ur * b.x - ui * b.y;
        cni += ur * b.y + ui * b.x;
      }
    }
    const double vk = __ldg(s.vk + k);
    const double o = (second ? so[1] : so[0]) + 2 * vk * (cor * cor + coi * coi);
    const double n = (second ? sn_[1] : sn_[0]) + 2 * vk * (cnr * cnr + cni * cni);
    so[0] = second ? so[0] : o;
    so[1] = second ? o : so[1];
    sn_[0] = second ? sn_[0] : n;
    sn_[1] = second ? n : sn_[1];
  }
  const double old_sum = share_sum(m.nshare, m.red, [&](int h) { return h ? so[1] : so[0]; });
  const double new_sum = share_sum(m.nshare, m.red, [&](int h) { return h ? sn_[1] : sn_[0]; });
  eold = old_sum * s.one_over_2v + s.self_energy;
  enew = new_sum * s.one_over_2v + s.self_energy;
}

// (new - old) * tau / epsilon of one slice, the level-0 Ewald term.
static __device__ double ewald_slice_diff(const DevSys& s, const Smem& m, int ipart, int t) {
  double eold, enew;
  ewald_slice_sums(s, m, ipart, t, eold, enew);
  return -(eold * s.tau / s.epsilon) + enew * s.tau / s.epsilon;
}

// evalLongRange of section slice t as staged in shared memory.
static __device__ double ewald_slice_energy(const DevSys& s, const Smem& m, int t) {
  double eold, enew;
  ewald_slice_sums(s, m, -1, t, eold, enew);
  return eold;
}

}  // namespace pimc

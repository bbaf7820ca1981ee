// Rigid displacement of whole particle paths: DisplaceMoveSampler::run/tryMove
// (src/advancer/DisplaceMoveSampler.cc:63-224) and, for fixed-node systems,
// DoubleDisplaceMoveSampler (src/advancer/DoubleDisplaceMoveSampler.cc:40-128),
// with a UniformMover (src/advancer/UniformMover.cc:25-42) and the actions'
// displacement differences: SHOAction (src/action/SHOAction.cc:107-143),
// PairAction (src/action/PairAction.cc:362-500), CoulombAction's Ewald term
// (src/action/CoulombAction.cc:123-146) and FixedNodeAction
// (src/fixednode/FixedNodeAction.cc:133-248).  SpringAction and PrimSHOAction
// contribute nothing (pi-qmc's base-class default).
//
// A replica's attempts follow one another, but the slices of an attempt are
// independent, so a cluster of 1, 2, 4 or 8 CTAs takes a replica and shares its
// slices: as many as keep the GPU busy with the replicas there are.  Every CTA
// draws and decides the same from the partial sums, exchanged through distributed
// shared memory: eight shares of every sum whatever the cluster, so that a replica's
// decisions do not depend on how many there are.  FP64 bound; what an attempt evaluates is
//  - the separations of the moved particles from the others, once per slice, each
//    lane's neighbour supplying the previous slice;
//  - with cached structure factors, the moved particles' terms alone (O(totk) per
//    slice against two full sums of O(N totk)), and an accepted move updates them;
//  - the Slater matrices of the moved paths, of whose elements only the moved
//    particles' rows and columns are new when the cached matrix is whole; an
//    accepted move updates the cached entries instead of dropping them.
// Four attempts of 19 electron gases (N = 54, M = 512, Ewald, 27 x 27 nodes): 504 ms
// with one CTA per replica and full sums, 9.4 ms so.
#pragma once
#include <cooperative_groups.h>

#include "entry_kernels.cuh"

namespace pimc {

constexpr int kMaxMoving = 4;
constexpr int kMaxDisplaceCluster = 8;

// Offsets (doubles) of a CTA's shared memory.
struct DisplaceLayout {
  int red, q, ictl;
  int sec;             // one staged slice, old and new, and
  int ewt, ewt_cols;   // its e^{ik.r} tables (replicas without cached structure factors)
  int ek, ek_stride, ek_batch;  // per warp: tables of ek_batch slices' moved beads (-ek:
                                // their place in the CTA's global area)
  int stage, stage_stride;  // slice pairs per warp, [lane group][2][3][n]
  int nodescr, nodescr_stride, nodecold_stride, split, in_smem, gcta;
  int total;
};

struct DisplaceParams {
  const DevSys* sys;
  DevState* state;
  double* paths;
  double* nodecache;
  long long* ekcache;
  double* scratch;         // per cluster: node dets and distances of the new and old pairs
  long long scratch_stride;  // doubles per cluster
  double* nodescr_g;       // per-CTA Slater scratch that is not in shared memory
  pimc_displace_record* rec;  // [nrep][nattempt] or null
  const int* order;
  int* next;
  int nattempt;
  int nrep;
  uint64_t seed;
  double box[3];
  int nmoving;
  int species;  // -1: any particle
  DisplaceLayout lay;
};

// Bead b of particle p at slice t (wrapping the slice index).
__device__ __forceinline__ const double* bead_at(const double* path, int np, int M, int p, int t) {
  t = t < 0 ? t + M : (t >= M ? t - M : t);
  return path + ((size_t)t * np + p) * 3;
}

// What the CTAs of a cluster exchange per attempt: its sums in kMaxDisplaceCluster shares,
// of which a CTA computes as many as its part of the cluster.
struct DisplaceShare {
  double ds[kMaxDisplaceCluster], node[kMaxDisplaceCluster];
  int bad, pad;
};

// One attempt's moved particles.
struct Moved {
  int n;
  int p[kMaxMoving];
  double d[kMaxMoving][3];
};

__device__ __forceinline__ int moved_index(const Moved& mv, int p) {
  for (int k = 0; k < mv.n; ++k)
    if (mv.p[k] == p) return k;
  return -1;
}

// The moved particles of a species, as a mask of its members.
__device__ __forceinline__ unsigned moved_mask(const DevSys& s, const Moved& mv, int sp) {
  unsigned r = 0;
  for (int k = 0; k < mv.n; ++k) {
    const int i = mv.p[k] - s.spec_first[sp];
    if (i >= 0 && i < s.spec_count[sp]) r |= 1u << i;
  }
  return r;
}

// Bead p of slice t, displaced (and returned to the box) when p is a moved particle.
__device__ __forceinline__ void displaced_bead(const DevSys& s, const Moved& mv,
                                               const double* path, int p, int t, double& x,
                                               double& y, double& z) {
  const double* b = path + ((size_t)t * s.npart + p) * 3;
  x = b[0];
  y = b[1];
  z = b[2];
  const int k = moved_index(mv, p);
  if (k >= 0) {
    x += mv.d[k][0];
    y += mv.d[k][1];
    z += mv.d[k][2];
    pbc(s, x, y, z);
  }
}

// The sums of an attempt, in nv shares: this warp's value of share v.  CTA rank of the
// cluster's C has shares rank, rank + C, ... (the first of the work goes to all CTAs).
struct DisplaceParts {
  static constexpr int nv = kMaxDisplaceCluster;
  double of[3][nv * (kBlock / 32)];  // action differences, Ewald terms, nodal actions
  static __device__ __forceinline__ double warp_tree(double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    return x;
  }
  __device__ __forceinline__ void put(int kind, int v, double x) {
    x = warp_tree(x);
    if ((threadIdx.x & 31) == 0) of[kind][v * (blockDim.x >> 5) + (threadIdx.x >> 5)] = x;
  }
};

// SHOAction and PairAction over slices [0, i2] (and [half, half + i2]) of the whole
// path, this thread's part of a share (warp gw of all shares' ngw).
__device__ __forceinline__ double displace_actions_share(const DevSys& s, const Moved& mv,
                                                         const double* path, int gw, int ngw) {
  const int np = s.npart, M = s.nslice, half = M / 2, lane = threadIdx.x & 31;
  const bool dbl = s.fixed_node != 0;
  const int nrange = dbl ? 2 : 1, len = dbl ? half : M;
  const int nmov = mv.n;
  double part = 0.0;
  // SHOAction: moving slots up to the first particle outside the species
  for (int sp = 0; sp < s.nspecies; ++sp) {
    const double om = s.sho_omega[sp];
    if (!(om > 0)) continue;
    int mstop = 0;
    while (mstop < nmov && mv.p[mstop] >= s.spec_first[sp] &&
           mv.p[mstop] < s.spec_first[sp] + s.spec_count[sp])
      ++mstop;
    const double mw = s.mass[sp] * om, ch = s.sho_cosh0[sp], div1 = 0.5 * s.sho_csch[sp];
    for (int it = gw * 32 + lane; it < mstop * nrange * len; it += ngw * 32) {
      const int k = it / (nrange * len), rest = it % (nrange * len);
      const int t = (rest / len) * half + rest % len;
      const int ip = mv.p[k];
      const double* b1 = bead_at(path, np, M, ip, t);
      const double* b0 = bead_at(path, np, M, ip, t - 1);
      double r1[3] = {b1[0], b1[1], b1[2]}, r0[3] = {b0[0], b0[1], b0[2]};
      double v = -mw * ((dot3(r1[0], r1[1], r1[2], r1[0], r1[1], r1[2]) +
                         dot3(r0[0], r0[1], r0[2], r0[0], r0[1], r0[2])) * ch -
                        2.0 * dot3(r0[0], r0[1], r0[2], r1[0], r1[1], r1[2])) * div1;
      for (int d = 0; d < 3; ++d) {
        r1[d] += mv.d[k][d];
        r0[d] += mv.d[k][d];
      }
      v += mw * ((dot3(r1[0], r1[1], r1[2], r1[0], r1[1], r1[2]) +
                  dot3(r0[0], r0[1], r0[2], r0[0], r0[1], r0[2])) * ch -
                 2.0 * dot3(r0[0], r0[1], r0[2], r1[0], r1[1], r1[2])) * div1;
      part += v;
    }
  }
  if (!s.coulomb) return part;
  // PairAction: a warp takes 31 links of one (moved particle, partner); lane l holds
  // the separations at slice t0 - 1 + l and lane l - 1 those before it
  const int chunks = (len + 30) / 31, per = nrange * chunks;
  for (int ti = 0; ti < s.ntab; ++ti) {
    const DevTable& tb = s.tab[ti];
    for (int w = gw; w < nmov * np * per; w += ngw) {  // warp-uniform
      const int im = w / (np * per), rest = w % (np * per), j = rest / per, c = rest % per;
      const int rg = c / chunks, tl0 = (c % chunks) * 31;
      const int i = mv.p[im];
      const bool in1 = i >= tb.ifirst1 && i < tb.ifirst1 + tb.npart1;
      const bool in2 = i >= tb.ifirst2 && i < tb.ifirst2 + tb.npart2;
      if (!in1 && !in2) continue;
      const int jb = in1 ? tb.ifirst2 : tb.ifirst1, jn = in1 ? tb.npart2 : tb.npart1;
      if (j < jb || j >= jb + jn) continue;
      const int jm = moved_index(mv, j);
      if (jm >= 0 && i <= j) continue;
      const int tl = tl0 + lane - 1;
      const bool live = tl < len;
      const int t = rg * half + (live ? tl : tl0);
      const double* bi = bead_at(path, np, M, i, t);
      const double* bj = bead_at(path, np, M, j, t);
      double ox = bi[0] - bj[0], oy = bi[1] - bj[1], oz = bi[2] - bj[2];
      double nx = bi[0] + mv.d[im][0] - bj[0], ny = bi[1] + mv.d[im][1] - bj[1],
             nz = bi[2] + mv.d[im][2] - bj[2];
      pbc(s, ox, oy, oz);
      if (tl < 0) {  // the range's previous slice: the image of the old one, moved
        nx = ox + mv.d[im][0];
        ny = oy + mv.d[im][1];
        nz = oz + mv.d[im][2];
      }
      if (jm >= 0) {
        nx -= mv.d[jm][0];
        ny -= mv.d[jm][1];
        nz -= mv.d[jm][2];
      }
      pbc(s, nx, ny, nz);
      const Sep n1{nx, ny, nz, square_root(dot3(nx, ny, nz, nx, ny, nz))};
      const Sep o1{ox, oy, oz, square_root(dot3(ox, oy, oz, ox, oy, oz))};
      const auto up = [](double v) { return __shfl_up_sync(0xffffffffu, v, 1); };
      const Sep n0{up(n1.x), up(n1.y), up(n1.z), up(n1.r)};
      const Sep o0{up(o1.x), up(o1.y), up(o1.z), up(o1.r)};
      if (lane > 0 && live)
        part += pair_term(tb, n1, n0, tb.norder > 0, 0) - pair_term(tb, o1, o0, tb.norder > 0, 0);
    }
  }
  return part;
}
static __device__ __noinline__ void displace_actions(const DevSys& s, const Moved& mv,
                                                     const double* path, int rank, int C,
                                                     DisplaceParts& parts) {
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
#pragma unroll 1
  for (int v = rank; v < parts.nv; v += C)
    parts.put(0, v, displace_actions_share(s, mv, path, v * nwarps + warp, parts.nv * nwarps));
}

// CoulombAction's long-range term from the cached structure factors: per slice, the
// moved particles' terms leave rho_k and come back displaced, on the cache's
// fixed-point grid.  Warps take batches of slices; the bead tables of a batch, then
// its k-vectors.  With commit the changed factors are stored instead (the same
// integers), and nothing is summed.  Returns this lane's share of
// sum_k 2 v_k (|rho'_k|^2 - |rho_k|^2).
static __device__ __noinline__ double displace_ewald(const DevSys& s, const Moved& mv,
                                                     const double* path, const double* qpart,
                                                     long long* ek, double* tables, int batch,
                                                     int gw, int ngw, bool commit) {
  const int M = s.nslice, totk = s.totk, lane = threadIdx.x & 31, nmov = mv.n;
  const int nx = s.ikmax[0] + 1, ky0 = s.ikmax[1], ny = 2 * ky0 + 1, kz0 = s.ikmax[2];
  const int w = 2 * nmov * batch;  // columns: (slice, particle, old / new)
  double2* X = (double2*)tables;
  double2* Y = X + nx * w;
  double2* Z = Y + ny * w;
  const double is = 1.0 / s.ek_scale;
  double acc = 0.0;
  for (int t0 = gw * batch; t0 < M; t0 += ngw * batch) {
    const int nt = min(batch, M - t0);
    __syncwarp();
    for (int it = lane; it < 6 * nmov * nt; it += 32) {  // (an axis per lane)
      const int c = it / 3, a = it - 3 * c;
      const int t = t0 + c / (2 * nmov), k = (c % (2 * nmov)) >> 1;
      const double* b = path + ((size_t)t * s.npart + mv.p[k]) * 3;
      double x = b[0], y = b[1], z = b[2];
      if (c & 1) displaced_bead(s, mv, path, mv.p[k], t, x, y, z);
      ewald_axis_table(s, (a == 0 ? X : (a == 1 ? Y : Z)) + c, w, a, a == 0 ? x : (a == 1 ? y : z));
    }
    __syncwarp();
    for (int it = lane; it < nt * totk; it += 32) {
      const int tt = it / totk, k = it - tt * totk;
      const int kx = __ldg(s.kvec + 3 * k), ky = __ldg(s.kvec + 3 * k + 1) + ky0,
                kz = __ldg(s.kvec + 3 * k + 2) + kz0;
      longlong2* at = (longlong2*)(ek + ((size_t)(t0 + tt) * totk + k) * 2);
      const longlong2 o = *at;
      longlong2 n = o;
      for (int im = 0; im < nmov; ++im) {
        const int col = (tt * nmov + im) * 2;
        long long are, aim, bre, bim;
        const double qs = __dmul_rn(qpart[mv.p[im]], s.ek_scale);
        ewald_term_fixed(s, X, Y, Z, w, col, kx, ky, kz, qs, are, aim);
        ewald_term_fixed(s, X, Y, Z, w, col + 1, kx, ky, kz, qs, bre, bim);
        n.x += bre - are;
        n.y += bim - aim;
      }
      if (commit) {
        *at = n;
      } else {
        // |rho'|^2 - |rho|^2 = (rho' - rho) . (rho' + rho)
        acc = __fma_rn(__ldg(s.vk + k),
                       __fma_rn(__ll2double_rn(n.x - o.x), __ll2double_rn(n.x + o.x),
                                __dmul_rn(__ll2double_rn(n.y - o.y), __ll2double_rn(n.y + o.y))),
                       acc);
      }
    }
  }
  return acc * (2 * is * is);
}

// The same without cached structure factors: evalLongRange of both configurations
// of every slice of this CTA's share.  All threads; every thread returns the sum of
// -(old) + (new), times tau / epsilon.
static __device__ __noinline__ double displace_ewald_full(const DevSys& s, const Smem& m,
                                                          const Moved& mv, const double* path,
                                                          int t0, int t1) {
  const int np = s.npart;
  double lr = 0.0;
  for (int t = t0; t < t1; ++t) {
    __syncthreads();
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
      const double* b = path + ((size_t)t * np + i) * 3;
      m.s1x[i] = b[0];
      m.s1y[i] = b[1];
      m.s1z[i] = b[2];
      double x, y, z;
      displaced_bead(s, mv, path, i, t, x, y, z);
      m.s1x[np + i] = x;
      m.s1y[np + i] = y;
      m.s1z[np + i] = z;
    }
    __syncthreads();
    const double eold = ewald_slice_energy(s, m, 0);
    const double enew = ewald_slice_energy(s, m, 1);
    lr += -(eold * s.tau / s.epsilon) + enew * s.tau / s.epsilon;
  }
  return lr;
}

// Slater determinants and distances of species sp's slice pairs (t, t + M/2), t in
// [t0, t1), warps over lane groups.  moved = false: the old pairs; valid cache
// entries are copied, the others evaluated and (with a cache) made whole.
// moved = true: the displaced ones, from the cached element matrices where there is
// a cache (whole after the first kind of pass), the moved particles' rows and columns
// computed.  Distances go to dist[t][2][ns_max], determinants to det[t] (displaced);
// returns whether this thread saw a singular matrix.
static __device__ __noinline__ bool displace_nodes(const DevSys& s, const Smem& m,
                                                   const Moved& mv, const double* path, int sp,
                                                   bool moved, int t0, int t1, double* cache,
                                                   double scale, int epoch, double* stage,
                                                   int stage_stride, double* det_out,
                                                   double* dist) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int n = s.spec_count[sp], f = s.spec_first[sp], half = s.nslice / 2, nsm = s.ns_max;
  const bool sho = s.node_kind[sp] == PIMC_NODES_SHO;
  const int W = node_group_width(n), G = 32 / W, g = lane / W, gl = lane & (W - 1);
  double* gscr = group_scr(m, warp * G + g, G, n, !sho);
  double* gcold = group_cold(m, warp * G + g, G, n, !sho);
  // (a warp's part is its own whatever the species: the next one's pass follows at once)
  double* st = stage + (size_t)warp * stage_stride + (size_t)g * 6 * n;  // [2][3][n]
  const unsigned pm = moved_mask(s, mv, sp);
  bool bad = false;
  for (int base = t0 + warp * G; base < t1; base += nwarps * G) {
    const int task = base + g;
    const bool act = task < t1;
    const int t = act ? task : base;
    double* e = cache ? cache_entry(s, cache, sp, t) : nullptr;
    const bool hit = !moved && e && e[0] == (double)epoch;
    double* d1 = dist + (size_t)t * 2 * nsm;
    double* d2 = d1 + nsm;
    const bool store = act && !hit;
    if (__any_sync(0xffffffffu, store)) {
      // stage this species' beads of slices t and t + M/2
      for (int p = gl; p < n; p += W)
        for (int side = 0; side < 2; ++side) {
          const int ts = t + side * half;
          double x, y, z;
          if (moved) {
            displaced_bead(s, mv, path, f + p, ts, x, y, z);
          } else {
            const double* b = path + ((size_t)ts * s.npart + f + p) * 3;
            x = b[0];
            y = b[1];
            z = b[2];
          }
          st[(side * 3 + 0) * n + p] = x;
          st[(side * 3 + 1) * n + p] = y;
          st[(side * 3 + 2) * n + p] = z;
        }
      __syncwarp();
      // node_eval_group reads particle f + p: views offset so that it lands on
      // staged entry p (the shuffles span the warp, so every group evaluates; a
      // group whose pair is cached stores nothing)
      SliceView v1{st - f, st + n - f, st + 2 * n - f, n, 0, -1, 0, 0, 0};
      SliceView v2{st + 3 * n - f, st + 4 * n - f, st + 5 * n - f, n, 0, -1, 0, 0, 0};
      double det = 0;
      int err = 0;
      double* ec = e ? e + 2 + 2 * n : nullptr;
      const unsigned rows = moved ? pm : (e ? cache_rowmask(e, cache_mask_slot(s, sp)) : 0u);
      node_eval_dispatch(W, s, sp, v1, v2, scale, gscr, 1, ec, moved ? pm : 0u, store, det, err,
                         d1, d2, nullptr, rows, gcold);
      if (store && gl == 0) {
        if (moved) det_out[t] = det;
        bad |= err != 0;
      }
      if (!moved && e && store) {
        // the entry is whole again
        __syncwarp(__activemask());
        for (int p = gl; p < n; p += W) {
          e[2 + p] = d1[p];
          e[2 + n + p] = d2[p];
        }
        if (gl == 0) {
          const double NaN = __longlong_as_double(0x7ff8000000000000LL);
          e[1] = det;
          // (an inverse block is not made here: such an entry is evaluated again
          // when a section visits it)
          e[0] = (err || sm_species(s, sp)) ? NaN : (double)epoch;
          e[cache_mask_slot(s, sp)] = 0.0;
          if (sm_species(s, sp)) e[cache_x_slot(s, sp)] = NaN;
        }
      }
    }
    __syncwarp();
    if (act && hit)
      for (int p = gl; p < n; p += W) {
        d1[p] = e[2 + p];
        d2[p] = e[2 + n + p];
      }
    __syncwarp();
  }
  return bad;
}

// An accepted move's cache entries of species sp, pairs t and t + M/2 for t in
// [t0, t1): the moved particles' columns (and, for t < M/2, whose determinants and
// distances are known, their rows) recomputed from the displaced path; an entry
// t + M/2 keeps its moved rows marked stale and is evaluated at its next visit.
static __device__ __noinline__ void displace_commit_nodes(const DevSys& s, const Moved& mv,
                                                          const double* path, int sp, int t0,
                                                          int t1, double* cache, int epoch,
                                                          const double* det, const double* dist) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int n = s.spec_count[sp], f = s.spec_first[sp], nn = n * n, half = s.nslice / 2;
  const int nsm = s.ns_max, np = s.npart, ms = cache_mask_slot(s, sp);
  const bool sho = s.node_kind[sp] == PIMC_NODES_SHO;
  const unsigned pm = moved_mask(s, mv, sp);
  const int np2 = __popc(pm), per = np2 * 2 * n;  // columns, then rows
  const double NaN = __longlong_as_double(0x7ff8000000000000LL);
  for (int it = threadIdx.x; it < 2 * (t1 - t0) * per; it += blockDim.x) {
    const int q = it / per, rest = it - q * per, t = t0 + (q >> 1) + (q & 1) * half;
    unsigned rm = pm;
    for (int k = rest / (2 * n); k > 0; --k) rm &= rm - 1u;
    const int p = __ffs(rm) - 1, x = rest % (2 * n);
    const bool row = x >= n;
    const int i = row ? p : x, j = row ? x - n : p;
    if (row && (t >= half || ((pm >> j) & 1u))) continue;
    double* e = cache_entry(s, cache, sp, t);
    if (t >= half && (__double_as_longlong(e[ms]) >> 63)) continue;  // not usable anyway
    const int ts = t >= half ? t - half : t + half;
    // views of the path itself: xyz interleaved, particle stride 3
    const double* b1 = path + ((size_t)t * np + f + j) * 3;
    const double* b2 = path + ((size_t)ts * np + f + i) * 3;
    SliceView v1{b1 - (f + j), b1 + 1 - (f + j), b1 + 2 - (f + j), 0, 0, -1, 0, 0, 0};
    SliceView v2{b2 - (f + i), b2 + 1 - (f + i), b2 + 2 - (f + i), 0, 0, -1, 0, 0, 0};
    const NodeElement v = sho ? node_element<true>(s, sp, v1, v2, i, j)
                              : node_element<false>(s, sp, v1, v2, i, j);
    double* ec = e + 2 + 2 * n + j * n + i;
    ec[0] = v.v;
    if (!sho) {
      ec[nn] = v.gx;
      ec[2 * nn] = v.gy;
      ec[3 * nn] = v.gz;
    }
  }
  __syncthreads();  // (the unusable entries' words are read above)
  for (int t = t0 + warp; t < t1; t += nwarps) {
    double* e = cache_entry(s, cache, sp, t);
    for (int p = lane; p < n; p += 32) {
      e[2 + p] = dist[(size_t)t * 2 * nsm + p];
      e[2 + n + p] = dist[((size_t)t * 2 + 1) * nsm + p];
    }
    if (lane == 0) {
      e[1] = det[t];
      e[0] = sm_species(s, sp) ? NaN : (double)epoch;
      e[ms] = 0.0;
      double* o = cache_entry(s, cache, sp, t + half);
      o[0] = NaN;
      o[ms] = __longlong_as_double(__double_as_longlong(o[ms]) | (long long)pm);
      if (sm_species(s, sp)) e[cache_x_slot(s, sp)] = o[cache_x_slot(s, sp)] = NaN;
    }
  }
}

__global__ void __launch_bounds__(kBlock) displace_kernel(DisplaceParams P) {
  namespace cg = cooperative_groups;
  extern __shared__ double smem[];
  __shared__ DevSys S;
  __shared__ Moved mv_;
  __shared__ int epoch[kMaxSpecies];
  __shared__ double scale[kMaxSpecies];
  __shared__ uint32_t status, ui_acc;
  __shared__ long long nacc;
  __shared__ int rnext[2], bad_, accept_;
  __shared__ DisplaceShare share[2];
  __shared__ DisplaceParts parts;
  __shared__ int flip[kMaxSpecies], ovalid[kMaxSpecies];
  __shared__ Smem M_;  // carved pointers, shared so that callees read them from shared memory
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  const int cluster = blockIdx.x / C;
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int gw = rank * nwarps + warp, ngw = C * nwarps;
  constexpr int nv = DisplaceParts::nv;
  const int nvw = nv * nwarps;
  cl.sync();  // every CTA has started: its shared memory may be written to
  for (int turn = 0;; ++turn) {
    if (threadIdx.x == 0 && rank == 0) {
      const int k = atomicAdd(P.next, 1);
      const int r = (k < P.nrep) ? P.order[k] : -1;
      for (int c = 0; c < C; ++c) *cl.map_shared_rank(&rnext[turn & 1], c) = r;
    }
    cl.sync();
    const int r = rnext[turn & 1];
    if (r < 0) break;
    {
      const int* src = (const int*)(P.sys + r);
      int* dst = (int*)&S;
      for (int i = threadIdx.x; i < (int)(sizeof(DevSys) / sizeof(int)); i += blockDim.x)
        dst[i] = src[i];
    }
    if (threadIdx.x == 0) {
      const DisplaceLayout& L = P.lay;
      Smem m{};
      m.red = smem + L.red;
      m.qpart = smem + L.q;
      m.ictl = (int*)(smem + L.ictl);
      m.nshare = nwarps;
      m.s1x = smem + L.sec;
      m.s1y = m.s1x + 2 * P.sys[r].npart;
      m.s1z = m.s1y + 2 * P.sys[r].npart;
      m.mx = m.s1x;  // (not read: evalLongRange of staged slices moves no bead)
      m.my = m.s1y;
      m.mz = m.s1z;
      m.ewt = smem + L.ewt;
      m.ewt_cols = L.ewt_cols;
      double* gbase = P.nodescr_g ? P.nodescr_g + (size_t)blockIdx.x * L.gcta : nullptr;
      m.ewx = L.ek > 0 ? smem + L.ek : gbase - L.ek;
      m.nodescr = L.in_smem ? smem + L.nodescr : gbase;
      m.nodescr_stride = L.nodescr_stride;
      m.nodecold = L.split ? gbase : nullptr;
      m.nodecold_stride = L.nodecold_stride;
      m.node_cold_follows = !L.split;
      M_ = m;
      status = P.state[r].status;
      nacc = 0;
      for (int k = 0; k < kMaxSpecies; ++k) {
        epoch[k] = P.state[r].epoch[k];
        scale[k] = P.state[r].node_scale[k];
        flip[k] = ovalid[k] = 0;
      }
    }
    __syncthreads();
    const DevSys& s = S;
    const Smem& m = M_;
    const Moved& mv = mv_;
    double* path = P.paths + s.path_offset;
    double* cache = (P.nodecache && s.nc_offset >= 0) ? P.nodecache + s.nc_offset : nullptr;
    long long* ek = (P.ekcache && s.ek_offset >= 0) ? P.ekcache + s.ek_offset : nullptr;
    const int np = s.npart, M = s.nslice, nmov = P.nmoving, nsm = s.ns_max;
    const int half = M / 2;
    const bool dbl = s.fixed_node != 0;
    // this CTA's slices: pairs (t, t + M/2), t in [h0, h1), for the node work and the
    // commits; [m0, m1) of all
    const int h0 = (int)((long long)half * rank / C), h1 = (int)((long long)half * (rank + 1) / C);
    const int m0 = (int)((long long)M * rank / C), m1 = (int)((long long)M * (rank + 1) / C);
    // per species: new determinants, then two distance sets, old and new by turns
    const long long spw = (long long)half * (1 + 4 * nsm);
    double* scr = P.scratch + (size_t)cluster * P.scratch_stride;
    const uint32_t att0 = P.state[r].attempt;
    for (int i = threadIdx.x; i < np; i += blockDim.x) m.qpart[i] = s.charge[species_of(s, i)];
    for (int a = 0; a < P.nattempt; ++a) {
      const uint32_t att = att0 + (uint32_t)a;
      // ---- particles and displacement (pi-qmc's random-number order)
      if (threadIdx.x == 0) {
        uint32_t ui = 0;
        mv_.n = nmov;
        for (int im = 0; im < nmov;) {
          int i;
          const double u = stream_uniform(P.seed, s.stream_id, att, ui++);
          if (P.species < 0) {
            i = (int)(np * u);
            if (i == np) continue;
          } else {
            const int nsp = s.spec_count[P.species], f = s.spec_first[P.species];
            i = (int)(nsp * u + f);
            if (i == nsp + f) i = nsp + f - 1;
          }
          bool dup = false;
          for (int jm = 0; jm < im; ++jm) dup |= mv_.p[jm] == i;
          if (!dup) mv_.p[im++] = i;
        }
        for (int k = 0; k < nmov; ++k)
          for (int d = 0; d < 3; ++d) mv_.d[k][d] = stream_uniform(P.seed, s.stream_id, att, ui++);
        for (int k = 0; k < nmov; ++k)
          for (int d = 0; d < 3; ++d) {
            mv_.d[k][d] -= 0.5;
            mv_.d[k][d] *= P.box[d];
          }
        ui_acc = ui;  // index of the Metropolis uniform
        bad_ = 0;
      }
      __syncthreads();
      // ---- Action differences, this CTA's shares
      displace_actions(s, mv, path, rank, C, parts);
      if (s.coulomb && s.ewald)
        for (int v = rank; v < nv; v += C) {
          if (ek) {
            parts.put(1, v, displace_ewald(s, mv, path, m.qpart, ek,
                                     m.ewx + (size_t)warp * P.lay.ek_stride, P.lay.ek_batch,
                                     v * nwarps + warp, nvw, false));
          } else {
            const int e0 = (int)((long long)M * v / nv), e1 = (int)((long long)M * (v + 1) / nv);
            const double lr = displace_ewald_full(s, m, mv, path, e0, e1);
            parts.put(1, v, threadIdx.x == 0 ? lr : 0.0);
          }
        }
      __syncthreads();  // (the Slater scratch lies over the warps' Ewald tables)
      // ---- FixedNodeAction per node species holding a moving particle
      if (dbl) {
        bool bad = false;
        for (int sp = 0; sp < s.nspecies; ++sp) {
          if (!s.node_kind[sp] || !moved_mask(s, mv, sp)) continue;
          double* ndet = scr + sp * spw;
          double* odist = ndet + half + (size_t)flip[sp] * half * 2 * nsm;
          double* ndist = ndet + half + (size_t)(flip[sp] ^ 1) * half * 2 * nsm;
          if (!ovalid[sp])
            bad |= displace_nodes(s, m, mv, path, sp, false, h0, h1, cache, scale[sp], epoch[sp],
                                  smem + P.lay.stage, P.lay.stage_stride, ndet, odist);
          __syncthreads();  // (the old pass made the entries whole)
          bad |= displace_nodes(s, m, mv, path, sp, true, h0, h1, cache, scale[sp], epoch[sp],
                                smem + P.lay.stage, P.lay.stage_stride, ndet, ndist);
        }
        if (bad) bad_ = 1;
        cl.sync();  // the other CTAs' determinants and distances
        bad = false;
        for (int v = rank; v < nv; v += C) {
          double np_part = 0.0;
          const int first = 32 * (warp * nv + v) + (threadIdx.x & 31);
          for (int sp = 0; sp < s.nspecies; ++sp) {
            if (!s.node_kind[sp] || !moved_mask(s, mv, sp)) continue;
            const int n = s.spec_count[sp];
            const double* ndet = scr + sp * spw;
            const double* odist = ndet + half + (size_t)flip[sp] * half * 2 * nsm;
            const double* ndist = ndet + half + (size_t)(flip[sp] ^ 1) * half * 2 * nsm;
            // a sign change against the first slice rejects
            for (int t = first; t < half; t += 32 * nvw)
              bad |= ndet[t] * ndet[0] < 0.0;
            // nodal action: -sum log(new) + sum log(old) over consecutive pairs
            for (int it = first; it < (half - 1) * n; it += 32 * nvw) {
              const int t = 1 + it / n, p = it % n;
              const double* a1 = ndist + (size_t)t * 2 * nsm;
              const double* a0 = ndist + (size_t)(t - 1) * 2 * nsm;
              const double* b1 = odist + (size_t)t * 2 * nsm;
              const double* b0 = odist + (size_t)(t - 1) * 2 * nsm;
              np_part -= log((1 - exp(-a1[p] * a0[p])) * (1 - exp(-a1[nsm + p] * a0[nsm + p])));
              np_part += log((1 - exp(-b1[p] * b0[p])) * (1 - exp(-b1[nsm + p] * b0[nsm + p])));
            }
          }
          parts.put(2, v, np_part);
        }
        if (bad) bad_ = 1;
      }
      __syncthreads();
      // ---- the shares, summed alike by every CTA
      DisplaceShare* mine = &share[a & 1];
      for (int v = rank + warp * C; v < nv; v += nwarps * C) {
        const int l = threadIdx.x & 31, at = v * nwarps + l;
        double x = parts.warp_tree(l < nwarps ? parts.of[0][at] : 0.0);
        if (s.coulomb && s.ewald) {
          const double lr = parts.warp_tree(l < nwarps ? parts.of[1][at] : 0.0);
          x += ek ? lr * s.one_over_2v * s.tau / s.epsilon : lr;
        }
        const double node = dbl ? parts.warp_tree(l < nwarps ? parts.of[2][at] : 0.0) : 0.0;
        if (l == 0) {
          mine->ds[v] = x;
          mine->node[v] = node;
        }
      }
      if (threadIdx.x == 0) mine->bad = bad_;
      cl.sync();
      double dst = 0.0, nodet = 0.0;
      bool bad = false;
      if (threadIdx.x < 32) {  // (a share per lane)
        if (threadIdx.x < nv) {
          const DisplaceShare* o = cl.map_shared_rank(mine, threadIdx.x % C);
          dst = o->ds[threadIdx.x];
          nodet = o->node[threadIdx.x];
          bad = o->bad;
        }
        dst = parts.warp_tree(dst);
        nodet = parts.warp_tree(nodet);
        bad = __any_sync(0xffffffffu, bad);
      }
      if (threadIdx.x == 0) {
        if (bad) nodet = 2e100;
        // ---- Metropolis test
        const double total = dst + nodet;
        const double u = stream_uniform(P.seed, s.stream_id, att, ui_acc);
        const bool acc = !(u > exp(-total + 0.0));
        accept_ = acc;
        if (!isfinite(dst)) status |= PIMC_STATUS_NONFINITE;
        if (acc) ++nacc;
        if (P.rec && rank == 0) {
          pimc_displace_record* rc = P.rec + (size_t)r * P.nattempt + a;
          for (int k = 0; k < kMaxMoving; ++k) {
            rc->ipart[k] = k < nmov ? mv_.p[k] : -1;
            for (int d = 0; d < 3; ++d) rc->disp[k][d] = k < nmov ? mv_.d[k][d] : 0.0;
          }
          rc->ds = dst;
          rc->ds_node = dbl ? nodet : 0.0;
          rc->accepted = acc ? 1 : 0;
        }
        if (dbl)
          for (int sp = 0; sp < s.nspecies; ++sp)
            if (s.node_kind[sp] && moved_mask(s, mv_, sp)) {
              // the old pairs' distances stand for the next attempt (a singular old
              // pair is found again)
              ovalid[sp] = !bad;
              if (acc) flip[sp] ^= 1;
            }
      }
      __syncthreads();
      if (accept_) {
        // ---- the accepted paths, their structure factors and Slater entries
        if (ek)
          displace_ewald(s, mv, path, m.qpart, ek,
                         m.ewx + (size_t)warp * P.lay.ek_stride, P.lay.ek_batch, gw,
                         ngw, true);
        cl.sync();  // every CTA is done with the old path
        for (int it = threadIdx.x; it < nmov * (m1 - m0); it += blockDim.x) {
          const int k = it / (m1 - m0), t = m0 + it % (m1 - m0);
          double* b = path + ((size_t)t * np + mv.p[k]) * 3;
          double x = b[0] + mv.d[k][0], y = b[1] + mv.d[k][1], z = b[2] + mv.d[k][2];
          pbc(s, x, y, z);
          b[0] = x;
          b[1] = y;
          b[2] = z;
        }
        cl.sync();
        if (dbl && cache)
          for (int sp = 0; sp < s.nspecies; ++sp) {
            if (!s.node_kind[sp] || !moved_mask(s, mv, sp)) continue;
            const double* ndet = scr + sp * spw;  // (the new distances are the old set now)
            displace_commit_nodes(s, mv, path, sp, h0, h1, cache, epoch[sp], ndet,
                                  ndet + half + (size_t)flip[sp] * half * 2 * nsm);
          }
      }
      __syncthreads();
    }
    if (threadIdx.x == 0 && rank == 0) {
      P.state[r].attempt = att0 + (uint32_t)P.nattempt;
      P.state[r].status = status;
      P.state[r].accepted += nacc;
      P.state[r].attempted += P.nattempt;
    }
  }
  cl.sync();  // no CTA leaves while another may still write to its shared memory
}

}  // namespace pimc

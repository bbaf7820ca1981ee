// Device-side data structures and physics for the bisection hot path.
// Each function cites the pi-qmc routine whose arithmetic it follows.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fixed_point.cuh"
#include "pimc_rng.h"

namespace pimc {

constexpr int kMaxSpecies = 4;
constexpr int kMaxTables = 10;
constexpr int kMaxNs = 32;  // particles per node-model species
constexpr int kMaxLevels = 8;  // levels 0..nlevel+1
constexpr int kBlock = 256;     // threads of the estimator and entry-point kernels
constexpr int kMaxBlock = 512;  // largest section-kernel block (64..512 threads)
constexpr int kWarps = kMaxBlock / 32;  // reduction slots

struct DevTable {
  const double* ugrid;  // (ngpts,2,ndata,2): coefficient, its difference to the next point's
  const float* ugrid32; // (ngpts,2,ndata) in FP32 (mixed precision)
  const double* logtab; // table of the logarithm (grid_log)
  int ngpts, norder, ndata, s1, s2;
  int ifirst1, npart1, ifirst2, npart2;
  double rgridinv, logrratioinv;
};

struct DevSys {
  int npart, nspecies, nslice, nlevel, nsec;
  int spec_first[kMaxSpecies], spec_count[kMaxSpecies];
  double mass[kMaxSpecies], lambda[kMaxSpecies], charge[kMaxSpecies];
  double sho_omega[kMaxSpecies], prim_a[kMaxSpecies], prim_b[kMaxSpecies];
  int node_kind[kMaxSpecies];
  double node_c[kMaxSpecies], node_cosh[kMaxSpecies];  // SHONodes constants
  double node_dk[kMaxSpecies];  // sqrt(2 m / tau): nodal distance = node_dk / |grad ln det|
  // FreeParticleNodes: PeriodicGaussian(alpha = m T, L) per species and axis.
  double pg_nome[kMaxSpecies][3], pg_pref[kMaxSpecies][3], pg_k[kMaxSpecies][3];
  int pg_nmax[kMaxSpecies][3];
  double pg_alpha[kMaxSpecies], pg_al[kMaxSpecies][3];  // alpha, alpha L
  double pg_c[kMaxSpecies][3];  // exp(-2 alpha L^2), or 0 where that image is left out
  int pg_images[kMaxSpecies];   // evaluated from the nearest images (pg_images_eval)
  double tau;
  // Per-level constants, evaluated on the host with the reference's expressions
  // (src/action/SpringAction.cc:72, src/advancer/mover/FreeMover.cc:78-79,
  // src/action/SHOAction.cc:31-36,77-82), so no thread repeats them.
  double spr_inv2s2[kMaxLevels][kMaxSpecies];
  double mov_sigma[kMaxLevels][kMaxSpecies], mov_inv2s2[kMaxLevels][kMaxSpecies];
  double sho_cosh[kMaxLevels][kMaxSpecies], sho_div1[kMaxLevels][kMaxSpecies];
  double sho_div2[kMaxLevels];
  double sho_coth[kMaxSpecies], sho_csch[kMaxSpecies], sho_cosh0[kMaxSpecies];
  // The mixed form's SHO link action without cancellation:
  // a |r1 - r0|^2 + b r0.r1, a = (m / 2 tau') (x coth x - 1), b = m w tanh(x / 2), x = w tau'
  float sho_a[kMaxLevels][kMaxSpecies], sho_b[kMaxLevels][kMaxSpecies];
  // Delayed rejection (MultiLevelSampler's delayedRejection): on, and the
  // second proposal's width and 1 / (2 width^2) at level nlevel - 1
  int dr;
  double dr_sigma[kMaxSpecies], dr_inv2s2[kMaxSpecies];
  double cell[3], cellb[3], rcut2;
  // FP32 pre-tests of the minimum image (pbc): rcut2 (1 - 1e-5) and rcut2 (1 + 1e-5),
  // and the reciprocal box sides
  float rcut2_lo, rcut2_hi, cellb_f[3];
  int spring, coulomb, ewald, mover, fixed_node;
  int mixed;  // PIMC_PREC_MIXED: pair-action terms in FP32, accumulated in FP64
  // lane-group widths of the species' Slater evaluations, a byte each: a full launch's,
  // and the widest of one that leaves SMs room (node_launch_width)
  unsigned node_widths, node_widest;
  double epsilon;
  int ntab;
  DevTable tab[kMaxTables];
  int totk;
  const int* kvec;
  const double* vk;
  double one_over_2v, self_energy, deltak[3];
  int ikmax[3];
  int ns_max;           // largest node-species count
  // The thermodynamic estimator's sums, by the system alone: chunks of slices, cut into
  // runs of thermo_run; part k of a chunk is the k-th thermo_sub links of every run.
  // (chunks times parts: kThermoChunks at most)
  int thermo_chunks, thermo_run, thermo_sub, thermo_parts;
  uint32_t stream_id;     // random stream of this replica (its replica or request id)
  long long nc_offset;    // doubles into the Slater-result cache pool (-1: no cache)
  int nc_stride;          // doubles per cache entry
  // Structure factors rho_k = sum_j q_j e^{ik.r_j} of every path slice, kept as
  // integers on a fixed-point grid so that incremental updates equal a fresh sum
  // bit for bit: [nslice][totk][re, im].
  long long ek_offset;    // int64 words into the structure-factor cache (-1: none)
  double ek_scale;        // grid spacing 1/ek_scale (a power of two)
  long long path_offset;  // doubles into the path pool
};

// Mutable per-replica state kept on the device between launches.
struct DevState {
  uint32_t attempt;
  uint32_t status;
  long long accepted;
  long long attempted;
  double node_scale[kMaxSpecies];
  int epoch[kMaxSpecies];  // bumped whenever a node model's scale changes
};

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ double dot3(double ax, double ay, double az, double bx, double by,
                                       double bz) {
  // (a0 b0 + a1 b1) + a2 b2 without contraction, as blitz::dot evaluates it.
  return __dadd_rn(__dadd_rn(__dmul_rn(ax, bx), __dmul_rn(ay, by)), __dmul_rn(az, bz));
}

// GB300's FP64 pipe takes 19 clocks of the SM for every warp instruction, and
// conversions and floor run on it too (16 clocks each); integer and FP32
// instructions take about a quarter of a clock.  So what decides (whether a
// vector is imaged, by which multiple of the box) runs on the integer and FP32
// pipes wherever the answer is certain there, and FP64 does only the arithmetic
// of the result.

// |v| cut to an FP32 from the high word: in [|v| (1 - 2^-20), |v|]; infinities,
// NaN and values past FP32's range give infinity or NaN.
__device__ __forceinline__ float abs_f32_trunc(double v) {
  const int h = (__double2hiint(v) & 0x7fffffff) - (896 << 20);
  return __int_as_float(min(max(h, 0), 0x0fffffff) << 3);
}

// (float)v, rounded to nearest even, on the integer pipe; zero, subnormal and
// out-of-range results take the conversion instruction.
__device__ __forceinline__ float f32_rn(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned m = hi & 0x7fffffffu;
  if (m - (897u << 20) >= (253u << 20)) return (float)v;
  unsigned b = __funnelshift_l(lo, m - (896u << 20), 3);  // the kept bits
  b += (lo << 3) + (b & 1u) > 0x80000000u;                // the 29 cut ones, ties to even
  return __uint_as_float(b | (hi & 0x80000000u));
}

// exp(x) by table (P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989): x = (64 e + j) ln2 / 64
// + r, |r| <= ln2 / 128, exp x = 2^e 2^(j/64) (1 + p(r)) with the series to r^5 (r^6 / 720
// < 2^-54).  Ten FP64 instructions where exp() takes sixteen; within 1 ulp too.
static __device__ const double kExp2[64] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951};
static __device__ __noinline__ double exp_call(double x) { return exp(x); }
__device__ __forceinline__ double exp_table(double x) {
  const unsigned m = (unsigned)__double2hiint(x) & 0x7fffffffu;
  if (m >= 0x4085e000u) return exp_call(x);  // |x| >= 700, NaN
  const double t = __fma_rn(x, 92.33248261689366, 6755399441055744.0);  // (3 2^51: rounds)
  const double k = __dsub_rn(t, 6755399441055744.0);
  const int n = __double2loint(t);
  // ln2 / 64 in two parts, the first of 36 bits
  double r = __fma_rn(-k, 0.010830424696223417, x);
  r = __fma_rn(-k, 2.572804622327669e-14, r);
  double p = __fma_rn(r, 1.0 / 120, 1.0 / 24);
  p = __fma_rn(r, p, 1.0 / 6);
  p = __fma_rn(r, p, 0.5);
  p = __fma_rn(__dmul_rn(r, r), p, r);
  const double c = __ldg(kExp2 + (n & 63));
  p = __fma_rn(c, p, c);
  return __hiloint2double(__double2hiint(p) + (int)((unsigned)(n >> 6) << 20), __double2loint(p));
}

// SuperCell::pbc (src/util/SuperCell.cc:25-34): minimum image, only applied
// when |v|^2 exceeds a quarter of the shortest side squared.
static __device__ __noinline__ double3 pbc_exact(const DevSys& s, double x, double y, double z) {
  if (dot3(x, y, z, x, y, z) > s.rcut2) {
    const double ix = floor(__dadd_rn(__dmul_rn(s.cellb[0], x), 1000.5)) - 1000;
    const double iy = floor(__dadd_rn(__dmul_rn(s.cellb[1], y), 1000.5)) - 1000;
    const double iz = floor(__dadd_rn(__dmul_rn(s.cellb[2], z), 1000.5)) - 1000;
    x = __dsub_rn(x, __dmul_rn(s.cell[0], ix));
    y = __dsub_rn(y, __dmul_rn(s.cell[1], iy));
    z = __dsub_rn(z, __dmul_rn(s.cell[2], iz));
  }
  return make_double3(x, y, z);
}

// The box side to subtract from component v of |v| ~ f (abs_f32_trunc) for its
// minimum image: 0 or +-L; ok is cleared where the rounding of v / L is not
// certain (within 4e-5 of a half-integer: the FP32 quotient errs by under 3e-6)
// or where it is beyond one box.
__device__ __forceinline__ double image_shift(double cell, float cellb, double v, float f,
                                              bool& ok) {
  const float u = f * cellb;
  ok &= fabsf(u - 0.5f) > 4e-5f && u < 1.4999f;  // (false for NaN)
  return u > 0.5f ? copysign(cell, v) : 0.0;
}

// pbc_exact with its test and its image numbers taken on the FP32 pipe where
// they are certain there: the same bits.  What is left of FP64 is nothing for a
// vector inside the cutoff (was 6 instructions) and three subtractions for an
// imaged one (was 24).  A step of 152 electron gases (N = 54, M = 512, 64 attempts)
// 115 -> 97 ms, of 9728 two-electron dots (32 attempts) 59.2 -> 53.2 ms.
__device__ __forceinline__ double3 pbc_far(const DevSys& s, double x, double y, double z,
                                           float fx, float fy, float fz, float r2) {
  bool ok = r2 > s.rcut2_hi;
  const double cx = image_shift(s.cell[0], s.cellb_f[0], x, fx, ok);
  const double cy = image_shift(s.cell[1], s.cellb_f[1], y, fy, ok);
  const double cz = image_shift(s.cell[2], s.cellb_f[2], z, fz, ok);
  return ok ? make_double3(__dsub_rn(x, cx), __dsub_rn(y, cy), __dsub_rn(z, cz))
            : pbc_exact(s, x, y, z);
}

// (a call: one copy for the movers' many images)
static __device__ __noinline__ double3 pbc_far_call(const DevSys& s, double x, double y, double z,
                                                    float fx, float fy, float fz, float r2) {
  return pbc_far(s, x, y, z, fx, fy, fz, r2);
}

// (returns whether the vector may have changed)
__device__ __forceinline__ bool pbc(const DevSys& s, double& x, double& y, double& z) {
  const float fx = abs_f32_trunc(x), fy = abs_f32_trunc(y), fz = abs_f32_trunc(z);
  const float r2 = fx * fx + fy * fy + fz * fz;
  if (r2 < s.rcut2_lo) return false;
  const double3 v = pbc_far_call(s, x, y, z, fx, fy, fz, r2);
  x = v.x;
  y = v.y;
  z = v.z;
  return true;
}

// |v|^2 of the FP32 terms, every rounding written out: the same bits in every
// kernel, however the compiler would contract the sum.
__device__ __forceinline__ float norm2_f(float x, float y, float z) {
  return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}
// The moves' order of the same (x and y fused the other way round), and of a.b.
__device__ __forceinline__ float dot_f(float ax, float ay, float az, float bx, float by, float bz) {
  return __fmaf_rn(az, bz, __fmaf_rn(ax, bx, __fmul_rn(ay, by)));
}
__device__ __forceinline__ float norm2_move_f(float x, float y, float z) {
  return dot_f(x, y, z, x, y, z);
}

// The mixed form's minimum image of an FP64 difference, rounded to FP32 for
// its FP32 terms (pbc's image, then the rounding, both without FP64
// conversions).
__device__ __forceinline__ void pbc_f(const DevSys& s, double x, double y, double z, float& fx,
                                      float& fy, float& fz) {
  fx = f32_rn(x);
  fy = f32_rn(y);
  fz = f32_rn(z);
  const float r2 = fx * fx + fy * fy + fz * fz;
  if (!(r2 < s.rcut2_lo)) {
    const double3 v = pbc_far(s, x, y, z, fabsf(fx), fabsf(fy), fabsf(fz), r2);
    fx = f32_rn(v.x);
    fy = f32_rn(v.y);
    fz = f32_rn(v.z);
  }
}

// PeriodicGaussian::evaluate (src/util/PeriodicGaussian.cc:20-40): the theta
// series value pref (1 + 2 sum_n q^(n^2) cos(n k x)) and its gradient
// -2 pref k sum_n n q^(n^2) sin(n k x), n < nmax.  pi-qmc builds the terms by a
// complex recurrence (q^(2n-1) e^(ikx) per step); here cos(n k x) and
// sin(n k x) follow the Chebyshev recurrence t_(n+1) = 2 cos(kx) t_n - t_(n-1)
// and the weights q^(n^2) the product q^(n^2) q^(2n+1): seven FP64 operations
// a term instead of fourteen, the same sums to ~1e-13 relative where the
// series nearly cancels (far smaller elsewhere).  Rounded operations
// throughout: every call site computes the same bits.
__device__ __forceinline__ double pg_eval(double nome, double pref, double k, int nmax, double x,
                                          double* grad) {
  double sw, cw;
  sincos(__dmul_rn(k, x), &sw, &cw);
  const double c2 = __dmul_rn(2.0, cw), q2 = __dmul_rn(nome, nome);
  double cp = 1.0, cc = cw, sp = 0.0, sc = sw;  // cos, sin of (n - 1) k x and n k x
  double w = nome, step = nome;                  // q^(n^2), q^(2n - 1)
  double s0 = 0.0, s1 = 0.0;
  for (int n = 1; n < nmax; ++n) {
    s0 = __fma_rn(w, cc, s0);
    s1 = __fma_rn(__dmul_rn(double(n), w), sc, s1);
    step = __dmul_rn(step, q2);
    w = __dmul_rn(w, step);
    const double cn = __fma_rn(c2, cc, -cp), sn = __fma_rn(c2, sc, -sp);
    cp = cc;
    cc = cn;
    sp = sc;
    sc = sn;
  }
  *grad = __dmul_rn(__dmul_rn(__dmul_rn(pref, 2.0), -k), s1);
  return __dmul_rn(pref, __fma_rn(2.0, s0, 1.0));
}

// One axis of pg_images_eval: r and rf are the images next to |x| and beyond it,
// relative to the Gaussian itself; returns 1 + r + rf and the bracket of the
// derivative, (L - |x|) r - |x| - (L + |x|) rf.
__device__ __forceinline__ double pg_axis(double al, double cell, double c, double ax, double& h) {
  const double r = exp_table(__dmul_rn(-al, __fma_rn(-2.0, ax, cell)));
  double p = __dadd_rn(1.0, r);
  h = __fma_rn(__dsub_rn(cell, ax), r, -ax);
  if (c > 0.0) {
    const double rf = __dmul_rn(c, reciprocal(r));  // r rf = exp(-2 alpha L^2)
    p = __dadd_rn(p, rf);
    h = __fma_rn(-__dadd_rn(cell, ax), rf, h);
  }
  return p;
}
__device__ __forceinline__ double with_sign_of(double v, double x) {
  return __longlong_as_double(__double_as_longlong(v) ^
                              (__double_as_longlong(x) & (long long)0x8000000000000000ULL));
}

// The product of the three axes' periodic Gaussians and its gradient from the
// nearest images of each axis, |x_d| <= L_d / 2:
// sum_m exp(-alpha (x - m L)^2) = exp(-alpha x^2) (1 + r + rf),
// r = exp(-alpha L (L - 2|x|)), rf = exp(-alpha L (L + 2|x|)),
// the Poisson resummation of the theta series of pg_eval.  The images left out
// are below exp(-2 alpha L^2) of the value, so it serves boxes with
// alpha L^2 >= 20 (8e-18); from 40 on rf is below 4e-18 too and left out
// (pg_c = 0).  Smaller boxes need more images and fewer terms of the series,
// and keep the series.  Four exponentials and 50 operations for an element
// against three series with sincos (380 FP64 instructions at alpha L^2 = 34,
// the 54-electron gas); every term is positive, so nothing cancels in the tails.
// 1024 evaluations of 27 x 27 matrices (host arrays) 1.93 -> 1.14 ms, a step of
// 152 electron gases 97 -> 88 ms.
// Rounded operations throughout: every call site computes the same bits.
__device__ __forceinline__ double pg_images_eval(const DevSys& s, int sp, double x, double y,
                                                 double z, double& gx, double& gy, double& gz) {
  const double al = s.pg_alpha[sp];
  const double e = exp_table(__dmul_rn(-al, dot3(x, y, z, x, y, z)));
  double hx, hy, hz;
  const double px = pg_axis(s.pg_al[sp][0], s.cell[0], s.pg_c[sp][0], fabs(x), hx);
  const double py = pg_axis(s.pg_al[sp][1], s.cell[1], s.pg_c[sp][1], fabs(y), hy);
  const double pz = pg_axis(s.pg_al[sp][2], s.cell[2], s.pg_c[sp][2], fabs(z), hz);
  const double pyz = __dmul_rn(py, pz);
  const double f = __dmul_rn(__dmul_rn(2.0, al), e);
  gx = with_sign_of(__dmul_rn(__dmul_rn(f, hx), pyz), x);
  gy = with_sign_of(__dmul_rn(__dmul_rn(f, hy), __dmul_rn(px, pz)), y);
  gz = with_sign_of(__dmul_rn(__dmul_rn(f, hz), __dmul_rn(px, py)), z);
  return __dmul_rn(e, __dmul_rn(px, pyz));
}

// log(q) for 1 <= q < 2^20, by table (P. T. P. Tang, "Table-driven implementation of
// the logarithm function in IEEE floating-point arithmetic", ACM TOMS 16, 1990): 128
// intervals an octave, c_j near the reciprocal of the interval's middle with few
// bits, r = m c_j - 1 with |r| < 2^-7.99, and log q = (e ln 2 - log c_j) + log1p(r), the
// first part tabulated per octave, the second by its series to r^6 (r^7 / 7 < 2^-58).
// Eight FP64 instructions where log() takes thirty.  The table: kLogReciprocals
// values c_j, then kLogEntries of e ln 2 - log c_j.
constexpr int kLogReciprocals = 128, kLogOctaves = 20;
constexpr int kLogEntries = kLogReciprocals * kLogOctaves;
__device__ __forceinline__ double grid_log(const double* tab, double q, unsigned k) {
  const int hi = __double2hiint(q);
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(q));
  const double r = __fma_rn(m, __ldg(tab + (k & (kLogReciprocals - 1))), -1.0);
  double p = __fma_rn(r, -1.0 / 6, 1.0 / 5);
  p = __fma_rn(r, p, -1.0 / 4);
  p = __fma_rn(r, p, 1.0 / 3);
  p = __fma_rn(r, p, -1.0 / 2);
  p = __fma_rn(__dmul_rn(r, r), p, r);
  return __dadd_rn(__ldg(tab + kLogReciprocals + k), p);
}

static __device__ __noinline__ double log_call(double q) { return log(q); }  // (rare)

// Pair-action table lookup on the logarithmic grid
// (PairAction::u00 / uk0 / uk0CalcDerivatives, src/action/PairAction.cc:601-655).
// Distances below the grid take its first point, those beyond it its last; a NaN or
// infinite distance ends in a clamped index too.  For finite q >= 1 the branches are
// pi-qmc's (i = int(x) > ngpts - 2 exactly when x >= ngpts - 1).
__device__ __forceinline__ void tab_locate(const DevTable& t, double q, int& i, double& x) {
  q *= t.rgridinv;
  const unsigned k = (unsigned)(__double2hiint(q) - 0x3ff00000) >> 13;
  if (k < (unsigned)kLogEntries) {
    x = grid_log(t.logtab, q, k) * t.logrratioinv;
  } else {  // below 1 (or negative: NaN paths), past 2^20, infinite or NaN
    x = q >= 1 ? log_call(q) * t.logrratioinv : 0.0;
    if (!(x < 2e9)) x = 2e9;
  }
  // the integer part by masks (x < 2^21; a conversion there and back takes 32 clocks)
  const int hi = __double2hiint(x), e = (hi >> 20) - 1023;
  double whole = 0.0;
  i = 0;
  if (hi >= 0x41400000) {
    i = (int)x;
    whole = i;
  } else if (e >= 0) {  // (a negative x has a negative e)
    i = ((hi & 0xfffff) | 0x100000) >> (20 - e);
    whole = __hiloint2double(hi & ~(0xfffff >> e), 0);
  }
  if (i > t.ngpts - 2) {
    i = t.ngpts - 2;
    x = 1;
  } else {
    x -= whole;
  }
}

// Coefficient k of row (i, which) at x between the grid points.
__device__ __forceinline__ double tab_at(const double* g, int k, double x) {
  const double2 v = __ldg((const double2*)g + k);
  return fma(x, v.y, v.x);
}

__device__ __forceinline__ double tab_u00(const DevTable& t, double r) {
  int i;
  double x;
  tab_locate(t, r, i, x);
  return tab_at(t.ugrid + (size_t)i * 4 * t.ndata, 0, x);
}

__device__ __forceinline__ double tab_uk0(const DevTable& t, double q, double s2) {
  int i;
  double x;
  tab_locate(t, q, i, x);
  const double* g = t.ugrid + (size_t)i * 4 * t.ndata;
  double a = 0;
  for (int k = t.norder; k >= 0; k--) a = a * s2 + tab_at(g, k, x);
  return a;
}

// The tau derivative of the series.
__device__ __forceinline__ double tab_uk0_tau(const DevTable& t, double q, double s2) {
  int i;
  double x;
  tab_locate(t, q, i, x);
  const double* g = t.ugrid + (size_t)(i * 2 + 1) * 2 * t.ndata;
  double a = 0;
  for (int k = t.norder; k >= 0; k--) a = a * s2 + tab_at(g, k, x);
  return a;
}

// FP32 variants for the mixed-precision form (same grid, FP32 coefficients).
__device__ __forceinline__ float tab_uk0_f(const DevTable& t, float q, float s2, int norder_eff) {
  q *= (float)t.rgridinv;
  float x = __fmul_rn(__logf(q), (float)t.logrratioinv);
  int i;  // range tests before the conversion, as tab_locate
  if (!(q >= 1.f)) {
    i = 0;
    x = 0.f;
  } else if (!(x < (float)(t.ngpts - 1))) {
    i = t.ngpts - 2;
    x = 1.f;
  } else {
    i = (int)x;
    x = __fsub_rn(x, (float)i);
  }
  const float* g0 = t.ugrid32 + (size_t)i * 2 * t.ndata;
  const float* g1 = g0 + 2 * t.ndata;
  float a = 0.f;
  for (int k = norder_eff; k >= 0; k--) a = fmaf(a, s2, fmaf(x, __ldg(g1 + k) - __ldg(g0 + k), __ldg(g0 + k)));
  return a;
}

// FP32 tau derivative of the off-diagonal series (uk0CalcDerivatives' utau).
__device__ __forceinline__ float tab_uk0d_tau_f(const DevTable& t, float q, float s2) {
  q *= (float)t.rgridinv;
  float x = __fmul_rn(__logf(q), (float)t.logrratioinv);
  int i;  // range tests before the conversion, as tab_locate
  if (!(q >= 1.f)) {
    i = 0;
    x = 0.f;
  } else if (!(x < (float)(t.ngpts - 1))) {
    i = t.ngpts - 2;
    x = 1.f;
  } else {
    i = (int)x;
    x = __fsub_rn(x, (float)i);
  }
  const float* g0 = t.ugrid32 + (size_t)i * 2 * t.ndata + t.ndata;
  const float* g1 = g0 + 2 * t.ndata;
  float a = 0.f;
  for (int k = t.norder; k >= 0; k--) a = fmaf(a, s2, fmaf(x, __ldg(g1 + k) - __ldg(g0 + k), __ldg(g0 + k)));
  return a;
}

// A compensated FP32 sum (Knuth's TwoSum per term, the rounding errors
// collected in a second float): the mixed form's sums over links and pairs.
struct FSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float t) {
    const float u = __fadd_rn(s, t);
    const float bb = __fsub_rn(u, s);
    c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(u, bb)), __fsub_rn(t, bb)));
    s = u;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// The sum of 32 nshare values, v(h) that of share warp + h nwarps (nwarps: the block's) on
// this lane: the same tree whichever block the shares are dealt to.  All threads.
template <class V>
__device__ __forceinline__ double share_sum(int nshare, double* red, V v) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
#pragma unroll 1
  for (int h = 0; w + h * nw < nshare; ++h) {
    double x = v(h);
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (l == 0) red[w + h * nw] = x;
  }
  __syncthreads();
  if (w == 0) {
    double x = (l < nshare) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (l == 0) red[kWarps] = x;
  }
  __syncthreads();
  return red[kWarps];
}

// Deterministic block sum of one double per thread (fixed tree order).
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (nw == 1) return __shfl_sync(0xffffffffu, v, 0);
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < nw) ? red[l] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (l == 0) red[kWarps] = v;
  }
  __syncthreads();
  return red[kWarps];
}

}  // namespace pimc

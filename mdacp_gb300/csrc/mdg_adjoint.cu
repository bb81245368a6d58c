// Adjoint of an NVE trajectory: gradients of a trajectory-averaged observable
// with respect to the LJ parameters (epsilon, sigma) and the initial state.
//
// No reference counterpart (a pattern on top of the drop-in).  The potential
// is the reference's smoothly truncated LJ (variables.cc:16-28) written with
// explicit parameters, V(r) = eps * phi(r / sigma),
//   phi(x) = 4 (x^-12 - x^-6 + C2 x^2 + C0) for x <= xc,
// the cut-off scaling with sigma (xc = cutoff in sigma units).  The step is
// the reference's drift-kick-drift (mdmanager.cc:151-157):
//   qh = q + p dt/2;  p' = p + F(qh) dt;  q' = qh + p' dt/2.
// Objectives J = (1/Ns) sum_{n=1..Ns} j(q_n, p_n) with j = U/N (mean
// potential energy per particle, MDManager::PotentialEnergy) or
// j = P = (2 KE - G) / (3 V), G = sum_pairs f(r) r^2 (MDManager::Pressure).
//
// Discrete adjoint (exact gradient of the discrete trajectory): walking the
// steps backwards, with a_q, a_p the adjoints of (q_n, p_n):
//   a_p += dt/2 a_q;  a_qh = a_q - dt H(qh) a_p;  g_theta += dt a_p . dF/dtheta(qh);
//   a_q = a_qh;  a_p += dt/2 a_qh;  then the objective terms of the earlier state.
// H v is the Hessian-vector product over the same pair list.  States are
// checkpointed every K steps in the forward pass; the backward pass recomputes
// each segment from its checkpoint (storing its K half-step positions and
// states) and then reverses it.  Each checkpoint segment starts by wrapping
// the positions into the box (a shift by whole box lengths: forces, objectives
// and adjoints are unchanged) and has its own pair list (every pair within
// cutoff*sigma + margin at the segment's first state, minimum image), built
// from the same state in both passes; the forward pass verifies that no
// particle moves more than margin/2 within a segment.  A list entry keeps the
// pair's image at the segment's first state, which stays the minimum image of
// every pair within the cut-off for the whole segment (box > 2 (rc + margin)),
// so the pair kernels form the separation with one subtraction per axis
// (from q_i, q_i - L or q_i + L) instead of a rounding.  The pair kernels give
// each particle several lanes and take the pair terms in fixed point on the
// integer units (P::fixed), else in Horner form in double without divisions
// (GB300's FP64 rate is 1/64 of FP32).
//
// A segment is held whole: only the step itself and the Hessian-vector product
// go state by state (400 and 200 launches per gradient of 200 steps); the
// objective, its gradient and the force's sigma derivative take all states of
// a segment in one launch.  A gradient of 4,000 atoms over 200 steps: 29.0 ms
// with every term in double and state by state, 14.3 with the terms in fixed
// point, 10.0 now (k_step 12.0 us x 400, k_reverse 25 x 200, k_build 50 x 20,
// k_objective 94 x 10 with the gradient and 64 x 10 without, k_force_sigma 68 x 10).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "mdg_internal.cuh"

namespace mdg {
namespace adj {

constexpr int kT = 128;
// Lanes sharing one particle's row in the pair kernels of the double form (FP64
// runs at 1/64 of the FP32 rate, so a few thousand particles need several lanes
// each to occupy every SM's FP64 pipes).
constexpr int kLanes = 8;
// The same in fixed point, for the kernels of one step (8 / 16 / 32 lanes: 7.7 /
// 5.8 / 5.3 ms per gradient of 864 atoms over 200 steps, 10.4 / 10.0 / 12.1 of
// 4,000, 33.2 / 34.6 / 44.2 of 16,384: more lanes shorten a row's chain where
// the rows don't fill the GPU; one value for all, the middle one's best, within
// 9 % of each size's own).
constexpr int kStepLanes = 16;
// Lanes per particle of the fixed-point kernels that take all states of a
// segment in one launch (1 / 2 / 4 lanes: 11.4 / 11.1 / 11.3 ms per gradient of
// 4,000 atoms at 8 lanes a step): rows enough to fill the GPU, and the FP64
// work that follows a row is done for more particles of a warp at once.
constexpr int kBatchLanes = 2;
// Lanes sharing one particle in the list build (a warp: the build's float
// test is light, so it needs many warps per SM to hide its load latency).
constexpr int kBuildLanes = 32;
constexpr int kMaskWords = 8;  // a lane's candidates kept as bits: up to 8,192 particles

struct P {
  double L[3];
  double inv_L[3];
  double eps, sig, dt, dt2;
  double xc2;      // (cutoff in sigma units)^2
  double c0, c2;   // correction constants of phi
  double sl2;      // list radius^2 (absolute)
  double sl2f;     // the float test's radius^2 (widened by 1e-3)
  double half_margin2;
  double volume;
  // eps / sigma^k products used per pair (no division in the pair terms)
  double inv_s2, e_s, e_s2, e_s3, e_s4;
  // coefficients of the pair terms in Horner form (pair_terms)
  double kf6, kf0, kfc, kp6, kp0, ke6, ke0, kec2, kec0, kd6, kd0, kdc, ks6, ks0, ksc;
  double kg6, kg0, kgc, kr6, kr0, krc, kq6, kq0, kqc;
  int n, cap, objective;
  // Fixed-point pair arithmetic (mdg_fixed.cuh) in reduced units x = r / sigma:
  // y = x^-2 is sigma^2 / r^2
  int fixed, unit_sigma;
  uint64_t fx_rc2, fx_near, fx_s2;  // (cutoff sigma)^2 and kFixNear sigma^2 in the unit of R; sigma^2, 2^-62
  int64_t fx_c8;
  int fx_L[3];
  float fx_l[3];
  float fx_fit_n, fx_fit_0;  // derivative_sums_fit
};

// A list entry: partner index << kImageBits | per axis two bits r + 1, the
// pair's image being q_j - r L (r in {-1, 0, 1}).
constexpr int kImageBits = 6;
constexpr int kMaxAdjointParticles = 1 << (32 - kImageBits);

// A checkpoint segment's states 0 .. K and the half steps 1 .. K that lead to
// states 1 .. K are held whole, each array [K + 1][n].  The forces at the half
// steps, their sigma derivatives, the objective's gradients at the states and
// the fixed-point positions are held for a window of W <= K steps at a time
// (kWindowBytes), [W + 1][n]; with them for all steps the longest segment that
// fits the memory would be 2.7 times shorter.  The kernels take a window's D:
// the whole arrays from its first state on, so that they count from 1 in both.
struct D {
  double4_32a *q, *p;        // the initial state
  double4_32a *aq, *ap, *aqh, *tmp, *tmp2;
  double4_32a *ckq, *ckp;    // checkpoints
  float4 *qf;                // float copy of the segment's first state (the list test)
  double4_32a *segq, *segp, *segqh;   // of the segment
  double4_32a *segf, *segs, *segg;    // of the window
  FixPos *segxq, *segxqh;    // segq and segqh in fixed point (P.fixed), of the window
  uint32_t *nbr;             // the current segment's list, row-major [n][cap]
  int *cnt;
  double *part;              // block partials, [W + 1][gridp][3]
  double *acc;               // running sums: J, g_eps, g_sig
  int *flag;
  unsigned int *done;        // blocks of the current reduction that wrote their partials
};

// Particle i's position and its images q_i - L, q_i + L per axis.
struct Home {
  double x, y, z, xm, ym, zm, xp, yp, zp;
};

__device__ __forceinline__ Home make_home(const P &c, const double4_32a &q) {
  return Home{q.x, q.y, q.z, q.x - c.L[0], q.y - c.L[1], q.z - c.L[2], q.x + c.L[0], q.y + c.L[1], q.z + c.L[2]};
}

// The partner of entry e and the separation d = q_j - r L - q_i in the
// entry's image, formed as q_j - (q_i + r L).
__device__ __forceinline__ int pair_sep(uint32_t e, const double4_32a *q, const Home &h, double &dx, double &dy,
                                        double &dz) {
  const int j = (int)(e >> kImageBits);
  const double4_32a qj = q[j];
  const uint32_t ix = e & 3u, iy = (e >> 2) & 3u, iz = (e >> 4) & 3u;
  dx = qj.x - (ix == 1u ? h.x : (ix == 0u ? h.xm : h.xp));
  dy = qj.y - (iy == 1u ? h.y : (iy == 0u ? h.ym : h.yp));
  dz = qj.z - (iz == 1u ? h.z : (iz == 0u ? h.zm : h.zp));
  return j;
}

// 1/x from the hardware estimate refined by one cubic Householder step
// (relative error of the estimate cubed, below double rounding).
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// Per pair at distance r (d = q_j - q_i): the reduced quantities.
struct PairTerms {
  double f;      // V'(r)/r: force on i is f d
  double fpr;    // f'(r)/r
  double phi;    // V(r)
  double fs;     // d f / d sigma
  double dphis;  // d V / d sigma
  double g;      // f r^2
  double gpr;    // g'(r)/r
  double gs;     // d g / d sigma
};

// With x^2 = r^2 / sigma^2, psi(x) = phi'(x)/x = -48 x^-14 + 24 x^-8 + 8 C2,
// chi(x) = x^2 psi(x):
//   f     = eps/s^2 psi              = x^-8 (kf6 x^-6 + kf0) + kfc
//   fpr   = eps/s^4 psi'(x)/x        = x^-10 (kp6 x^-6 + kp0)
//   phi   = eps phi(x)               = x^-6 (ke6 x^-6 + ke0) + (kec2 x^2 + kec0)
//   dphis = -eps/s x phi'(x)         = x^-6 (kd6 x^-6 + kd0) + kdc x^2
//   fs    = -eps/s^3 (2 psi + x psi'(x))  = x^-8 (ks6 x^-6 + ks0) + ksc
//   g     = eps chi(x)               = x^-6 (kg6 x^-6 + kg0) + kgc x^2
//   gpr   = eps/s^2 chi'(x)/x        = x^-8 (kr6 x^-6 + kr0) + krc
//   gs    = -eps/s x chi'(x)         = x^-6 (kq6 x^-6 + kq0) + kqc x^2
// (coefficients set in mdg_adjoint_create; the kernels keep the terms they use).
__device__ __forceinline__ bool pair_terms(const P &c, double r2, PairTerms &t) {
  const double x2 = r2 * c.inv_s2;
  // x2 >= +0: compared as bit patterns, on the integer pipe (same order)
  if (__double_as_longlong(x2) > __double_as_longlong(c.xc2)) return false;
  const double ix2 = recip(x2), ix4 = ix2 * ix2, ix6 = ix4 * ix2, ix8 = ix4 * ix4, ix10 = ix8 * ix2;
  t.f = fma(ix8, fma(c.kf6, ix6, c.kf0), c.kfc);
  t.fpr = ix10 * fma(c.kp6, ix6, c.kp0);
  t.phi = fma(ix6, fma(c.ke6, ix6, c.ke0), fma(c.kec2, x2, c.kec0));
  t.dphis = fma(ix6, fma(c.kd6, ix6, c.kd0), c.kdc * x2);
  t.fs = fma(ix8, fma(c.ks6, ix6, c.ks0), c.ksc);
  t.g = fma(ix6, fma(c.kg6, ix6, c.kg0), c.kgc * x2);
  t.gpr = fma(ix8, fma(c.kr6, ix6, c.kr0), c.krc);
  t.gs = fma(ix6, fma(c.kq6, ix6, c.kq0), c.kqc * x2);
  return true;
}

// Row i's entries k = lane, lane + kLanes, ...: body(t, dx, dy, dz, j) for
// each pair within the cut-off, in the row's order.
template <class Body>
__device__ __forceinline__ void for_pairs(const P &c, const D &d, int i, int lane, const double4_32a *q,
                                          const Home &h, Body body) {
  const int cnt = d.cnt[i];
  const uint32_t *row = d.nbr + (size_t)i * c.cap;
  for (int k = lane; k < cnt; k += kLanes) {
    double dx, dy, dz;
    const int j = pair_sep(row[k], q, h, dx, dy, dz);
    PairTerms t;
    if (pair_terms(c, dx * dx + dy * dy + dz * dz, t)) body(t, dx, dy, dz, j);
  }
}

// Sum over the LANES lanes that share a particle (all lanes hold the total).
template <int LANES>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// The pair kernels' sums in fixed point.  An FP64 pair of the step, of the
// objective's gradient and of the Hessian-vector product took 21, 22 and 39
// instructions of the FP64 pipe, which was busy 66-79 % of the time; here the
// pair terms, force sums and objective sums are integers, and 13 of them are
// left, all in the Hessian-vector product (its vectors have no fixed range).

// Powers of y = (r / sigma)^-2: y 2^-62, y^3 2^-61, y^4 2^-62, y^7 2^-59.
struct FixTerms {
  uint64_t y, y3, y4, y7;
};

__device__ __forceinline__ uint64_t fix_y(const P &c, uint64_t R) {
  const uint64_t y = fix_recip(R);
  return c.unit_sigma ? y : fix_mulhi(y, c.fx_s2) << 2;
}

__device__ __forceinline__ FixTerms fix_terms(const P &c, uint64_t R) {
  FixTerms t;
  uint64_t y2;
  t.y = fix_y(c, R);
  fix_powers(t.y, y2, t.y3);
  t.y4 = fix_sqrhi(y2);
  t.y7 = fix_mulhi(t.y4, t.y3);
  return t;
}

// psi = 24 y^4 - 48 y^7 + 8 C2, 2^-55 (fix_force).
__device__ __forceinline__ int64_t fix_psi(const P &c, const FixTerms &t) {
  const int64_t v = (int64_t)((t.y4 >> 4) - t.y7);
  return v + (v << 1) + c.fx_c8;
}

// An eighth of 144 y^4 - 576 y^7 - 16 C2 = -(2 psi + x psi'), 2^-55: the sigma
// derivative of the force, and minus the pressure objective's slope.
__device__ __forceinline__ int64_t fix_dsigma(const P &c, const FixTerms &t) {
  const int64_t q = (int64_t)((t.y4 >> 4) - (t.y7 << 1)) >> 2;
  return (q << 3) + q - (c.fx_c8 >> 2);
}

// psi'(x) / x = 672 y^8 - 192 y^5, over 48, 2^-55.
__device__ __forceinline__ int64_t fix_psi_slope(const FixTerms &t) {
  const int64_t a = (int64_t)(14 * (t.y7 >> 2) - (t.y4 >> 3));  // 14 y^7 - 4 y^4, 2^-57
  const int32_t ah = fix_shi(a), al = fix_slo(a), yh = fix_shi((int64_t)t.y), yl = fix_slo((int64_t)t.y);
  const int64_t m = fix_mads(ah, yl, fix_mads(al, yh, 0));
  return fix_mads((int32_t)fix_hi((uint64_t)m), 1, fix_mads(ah, yh, 0));
}

// v 2^-shift as a double, rounded, without the FP64 pipe's conversion.
__device__ __forceinline__ double fix_double(int64_t v, int shift) {
  const uint64_t a = v < 0 ? 0ull - (uint64_t)v : (uint64_t)v;
  if (a == 0) return 0.0;
  const int z = __clzll((long long)a);
  const uint64_t m = ((a << z) >> 10) + 1 >> 1;  // 53 bits, rounded (2^53 carries into the exponent)
  const uint64_t e = (uint64_t)(1023 + 63 - z - shift) << 52;
  return __longlong_as_double((long long)((e + (m - 0x10000000000000ull)) | ((uint64_t)v & 0x8000000000000000ull)));
}

// Row i's entries k = lane, lane + LANES, ... on the fixed-point positions x,
// the next one's position in flight: body(take, sep, R, j), take where the pair
// lies within the cut-off and beyond kFixNear; close(e) for a pair nearer than
// that, which takes the double terms.  (Two pairs at a time took 84 registers
// for 72 and 10.46 ms for 9.97 per gradient of 4,000 atoms, 39.0 for 34.6 of 16,384.)
template <int LANES, class Body, class Close>
__device__ __forceinline__ void for_pairs_fixed(const P &c, const D &d, int i, int lane, const FixPos *x, Body &&body,
                                                Close &&close) {
  const int cnt = d.cnt[i];
  const uint32_t *row = d.nbr + (size_t)i * c.cap;
  const FixPos own = ld_fix<false>(x + i);
  const uint32_t none = ((uint32_t)i << kImageBits) | 0x15u;
  auto entry = [&](int k) { return k < cnt ? row[k] : none; };
  uint32_t e = entry(lane);
  FixPos q = ld_fix<false>(x + (e >> kImageBits));
  uint32_t en = entry(lane + LANES);
  for (int k = lane; k < cnt; k += LANES) {
    const FixPos qn = ld_fix<false>(x + (en >> kImageBits));
    const uint32_t ef = entry(k + 2 * LANES);
    int dx = q.x - own.x, dy = q.y - own.y, dz = q.z - own.z;
    float lx = q.lx - own.lx, ly = q.ly - own.ly, lz = q.lz - own.lz;
    const uint32_t ix = e & 3u, iy = (e >> 2) & 3u, iz = (e >> 4) & 3u;  // d = q_j - r L - q_i, r + 1 stored
    if (ix != 1u) { dx += ix ? -c.fx_L[0] : c.fx_L[0]; lx += ix ? -c.fx_l[0] : c.fx_l[0]; }
    if (iy != 1u) { dy += iy ? -c.fx_L[1] : c.fx_L[1]; ly += iy ? -c.fx_l[1] : c.fx_l[1]; }
    if (iz != 1u) { dz += iz ? -c.fx_L[2] : c.fx_L[2]; lz += iz ? -c.fx_l[2] : c.fx_l[2]; }
    const FixSep sep = fix_sep(dx, dy, dz, lx, ly, lz);
    const uint64_t R = fix_r2(sep);
    const bool in = R <= c.fx_rc2, near = in && R < c.fx_near;
    body(in && !near, sep, R, (int)(e >> kImageBits));
    if (near) close(e);
    e = en;
    en = ef;
    q = qn;
  }
}

// A double pair of the row of i (close pairs and rows whose integer sums do
// not fit): body(t, dx, dy, dz, j) as for_pairs'.
template <class Body>
__device__ __forceinline__ void one_pair(const P &c, uint32_t e, const double4_32a *q, const Home &h, Body &&body) {
  double dx, dy, dz;
  const int j = pair_sep(e, q, h, dx, dy, dz);
  PairTerms t;
  if (pair_terms(c, dx * dx + dy * dy + dz * dz, t)) body(t, dx, dy, dz, j);
}

template <int LANES>
__device__ __forceinline__ void lane_sums(FixForce &f) {
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    f.x += __shfl_xor_sync(0xffffffffu, f.x, o);
    f.y += __shfl_xor_sync(0xffffffffu, f.y, o);
    f.z += __shfl_xor_sync(0xffffffffu, f.z, o);
    f.mx += __shfl_xor_sync(0xffffffffu, f.mx, o);
    f.my += __shfl_xor_sync(0xffffffffu, f.my, o);
    f.mz += __shfl_xor_sync(0xffffffffu, f.mz, o);
    f.cx += __shfl_xor_sync(0xffffffffu, f.cx, o);
    f.cy += __shfl_xor_sync(0xffffffffu, f.cy, o);
    f.cz += __shfl_xor_sync(0xffffffffu, f.cz, o);
    f.s += __shfl_xor_sync(0xffffffffu, f.s, o);
  }
}

// Whether the sum of psi d over n entries stays inside 2^11: as fix_sum_fits,
// which bounds the sum of |psi| x by 7 n - 1.13 sum(psi), here at most 960, and
// the separation is x sigma with sigma up to 1.8.
__device__ __forceinline__ bool sums_fit(const FixForce &f, int n) { return f.s >= (float)(7 * n - 850) * 8388608.0f; }

// The same for the sum of q d, q = fix_dsigma (the force's sigma derivative, the
// pressure's slope), f.s the sum of psi: q does not vanish where psi does, so its
// sum has a bound of its own (derivative_fit).
__device__ __forceinline__ bool derivative_sums_fit(const P &c, const FixForce &f, int n) {
  return f.s >= fmaf(c.fx_fit_n, (float)n, c.fx_fit_0);
}

// |q| x <= a - b psi for every pair that takes the fixed-point terms, so the sum
// of q d is at most sigma (a n - b sum(psi)), and below 1,900 of 2^11 where
// sum(psi) >= (a n - 1900 / sigma) / b.  a is found over the pairs' range of x for
// b = 1.82, the ratio of |q| to -psi of the closest of them: a = 11 at a cut-off
// of 2.5.
void derivative_fit(P &c) {
  const double b = 1.82, x0 = std::sqrt(kFixNear), x1 = std::sqrt(c.xc2);
  double a = 0.0;
  for (int k = 0; k <= 4096; k++) {
    const double x = x0 + (x1 - x0) * k / 4096.0, y = 1.0 / (x * x), y4 = y * y * y * y, y7 = y4 * y * y * y;
    const double psi = 24.0 * y4 - 48.0 * y7 + 8.0 * c.c2, q = 18.0 * y4 - 72.0 * y7 - 2.0 * c.c2;
    a = std::fmax(a, std::fabs(q) * x + b * psi);
  }
  a += 0.5;  // between the samples
  c.fx_fit_n = (float)(a / b * 8388608.0);
  c.fx_fit_0 = (float)(-1900.0 / (c.sig * b) * 8388608.0);
}

// scale times the vector sum; unit 2^-52.
__device__ __forceinline__ double3 fix_vector(const FixForce &f, double scale) {
  const double u = scale * (1.0 / (double)(1ull << kFixSumBits));
  return make_double3(fix_sum(f.x, f.mx, f.cx) * u, fix_sum(f.y, f.my, f.cy) * u, fix_sum(f.z, f.mz, f.cz) * u);
}

// Sums of z = y^3, z^2 (2^-54) and r^2 (2^-51) over a row and its pair count,
// as the single box's observers (mdg_fixed.cu).
struct FixSums {
  uint64_t z, zz, r;
  int m;
};
constexpr int kFixSumsRow = 361;  // longest row whose sums fit

__device__ __forceinline__ void fix_sums_add(FixSums &s, bool take, uint64_t y3, uint64_t R) {
  const uint64_t zz = fix_sqrhi(y3);
  s.z += take ? y3 >> 7 : 0;
  s.zz += take ? zz >> 4 : 0;
  s.r += take ? R >> 7 : 0;
  s.m += take ? 1 : 0;
}

template <int LANES>
__device__ __forceinline__ void lane_sums(FixSums &s) {
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
    s.zz += __shfl_xor_sync(0xffffffffu, s.zz, o);
    s.r += __shfl_xor_sync(0xffffffffu, s.r, o);
    s.m += __shfl_xor_sync(0xffffffffu, s.m, o);
  }
}

// The row's sums of x^-6, x^-12, x^2 as doubles, and its pair count.
__device__ __forceinline__ double3 fix_sums_double(const P &c, const FixSums &s) {
  const double u = 1.0 / (double)(1ull << 54), half = 0.5 * s.m;
  return make_double3(((double)s.z + half) * u, ((double)s.zz + half) * u,
                      ((double)s.r + half) * (1.0 / (double)(1ull << 51)) * c.inv_s2);
}

// Block sums of three values at once (thread 0 holds them).
__device__ __forceinline__ void block_sum3(double &a, double &b, double &e, double *sh) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    e += __shfl_down_sync(0xffffffffu, e, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sh[3 * (threadIdx.x >> 5)] = a;
    sh[3 * (threadIdx.x >> 5) + 1] = b;
    sh[3 * (threadIdx.x >> 5) + 2] = e;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a = b = e = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      a += sh[3 * w];
      b += sh[3 * w + 1];
      e += sh[3 * w + 2];
    }
  }
  __syncthreads();
}

// Writes this block's three partials; the last block of the grid to do so
// adds w times their sums (blocks in a fixed order, so the result does not
// depend on which block finished last) to acc[0..2] and rearms the counter.
// No block waits for another.
__device__ void partials_accumulate(const D &d, double A, double B, double E, double w) {
  __shared__ int last;
  __shared__ double sh2[96];
  if (threadIdx.x == 0) {
    const size_t at = 3 * ((size_t)blockIdx.y * gridDim.x + blockIdx.x);
    d.part[at + 0] = A;
    d.part[at + 1] = B;
    d.part[at + 2] = E;
    __threadfence();
    last = atomicAdd(d.done, 1u) == gridDim.x * gridDim.y - 1 ? 1 : 0;
  }
  __syncthreads();
  if (!last) return;
  double a = 0, b = 0, e = 0;
  for (size_t k = threadIdx.x; k < (size_t)gridDim.x * gridDim.y; k += blockDim.x) {
    a += __ldcg(d.part + 3 * k);
    b += __ldcg(d.part + 3 * k + 1);
    e += __ldcg(d.part + 3 * k + 2);
  }
  block_sum3(a, b, e, sh2);
  if (threadIdx.x == 0) {
    d.acc[0] += w * a;
    d.acc[1] += w * b;
    d.acc[2] += w * e;
    *d.done = 0;
  }
}

// Pair list at positions q (wrapped into the box): every partner within the
// list radius, minimum image.  kBuildLanes lanes share a particle: lane l
// tests partners j = l, l + kBuildLanes, ... (a particle's lanes read
// neighbouring positions together), keeps the hits as bits where they fit
// kMaskWords words (4,000 particles: 49.9 us, 60 with the test made again) and
// writes them at its offset in the row (a prefix sum over the lanes), so the row order is fixed:
// lane 0's partners, then lane 1's, ...  The test runs in float against a radius widened by 1e-3
// (float positions of a box of tens of sigma are within 1e-5), so every pair
// within the exact radius is listed; a few more do no harm (the pair terms cut
// at rc).  The float positions come from d.qf (k_begin writes them), so a
// candidate costs one 16-byte load and no conversions.  The recorded image is
// the double-precision minimum image, r = rint((q_j - q_i) / L) per axis, in
// {-1, 0, 1} for wrapped positions.
__global__ void __launch_bounds__(kT) k_build(P c, D d, const double4_32a *q) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = tid / kBuildLanes, lane = tid % kBuildLanes;
  const bool active = i < c.n;
  float qx = 0.f, qy = 0.f, qz = 0.f;
  if (active) {
    const float4 v = d.qf[i];
    qx = v.x;
    qy = v.y;
    qz = v.z;
  }
  const float lx = (float)c.L[0], ly = (float)c.L[1], lz = (float)c.L[2];
  const float sl2f = (float)c.sl2f;
  // wrapped positions differ by at most L per axis, so the minimum-image
  // separation is min(|d|, L - |d|): no rounding instruction per candidate
  auto within = [&](int j) {
    const float4 v = d.qf[j];
    float ax = fabsf(v.x - qx), ay = fabsf(v.y - qy), az = fabsf(v.z - qz);
    ax = fminf(ax, lx - ax);
    ay = fminf(ay, ly - ay);
    az = fminf(az, lz - az);
    return ax * ax + ay * ay + az * az <= sl2f && j != i;
  };
  // one pass where the lane's candidates fit its mask words, else tested again
  __shared__ uint32_t masks[kT][kMaskWords];
  uint32_t *mask = masks[threadIdx.x];
  const bool keep = c.n <= kBuildLanes * 32 * kMaskWords;
  int m = 0;
  if (active) {
    if (keep) {
      int word = 0;
      for (int j0 = lane; j0 < c.n; j0 += 32 * kBuildLanes, word++) {
        uint32_t bits = 0u;
#pragma unroll 8
        for (int u = 0; u < 32; u++) {
          const int j = j0 + u * kBuildLanes;
          if (within(min(j, c.n - 1)) && j < c.n) bits |= 1u << u;
        }
        mask[word] = bits;
        m += __popc(bits);
      }
    } else {
      for (int j = lane; j < c.n; j += kBuildLanes) m += within(j) ? 1 : 0;
    }
  }
  // offsets of the lanes' partners in the row
  int incl = m;
#pragma unroll
  for (int o = 1; o < kBuildLanes; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o, kBuildLanes);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, kBuildLanes - 1, kBuildLanes);
  if (active) {
    int w = incl - m;
    uint32_t *row = d.nbr + (size_t)i * c.cap;
    const double4_32a qi = q[i];
    auto append = [&](int j) {
      if (w < c.cap) {
        const double4_32a v = q[j];
        const int rx = (int)rint((v.x - qi.x) * c.inv_L[0]), ry = (int)rint((v.y - qi.y) * c.inv_L[1]),
                  rz = (int)rint((v.z - qi.z) * c.inv_L[2]);
        row[w] = ((uint32_t)j << kImageBits) | (uint32_t)(rx + 1) | ((uint32_t)(ry + 1) << 2) |
                 ((uint32_t)(rz + 1) << 4);
      }
      w++;
    };
    if (keep) {
      int word = 0;
      for (int j0 = lane; j0 < c.n; j0 += 32 * kBuildLanes, word++)
        for (uint32_t bits = mask[word]; bits; bits &= bits - 1u) append(j0 + (__ffs(bits) - 1) * kBuildLanes);
    } else {
      for (int j = lane; j < c.n; j += kBuildLanes)
        if (within(j)) append(j);
    }
    if (lane == 0) {
      d.cnt[i] = total < c.cap ? total : c.cap;
      if (total > c.cap) atomicMax(d.flag, total);
    }
  }
}

// Particle i's pair sums of the objective at positions q (every lane holds
// them after the lane sums; all threads of the block call it).
struct ObjSums {
  double u, us, G, Gs, gx, gy, gz;
};

template <int OBJ, bool GRAD>
__device__ __forceinline__ ObjSums objective_sums(const P &c, const D &d, int i, int lane, const double4_32a *q) {
  ObjSums r{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (i < c.n) {
    const Home h = make_home(c, q[i]);
    for_pairs(c, d, i, lane, q, h, [&](const PairTerms &t, double dx, double dy, double dz, int) {
      if (OBJ == 0) {
        r.u += 0.5 * t.phi;
        if (GRAD) {
          r.us += 0.5 * t.dphis;
          r.gx -= t.f * dx;  // dU/dq_i = -F_i
          r.gy -= t.f * dy;
          r.gz -= t.f * dz;
        }
      } else {
        r.G += 0.5 * t.g;
        if (GRAD) {
          r.Gs += 0.5 * t.gs;
          r.gx += t.gpr * dx;  // dG/dq_i = -sum g'(r) d/r;  dP/dq_i = -(1/3V) dG/dq_i
          r.gy += t.gpr * dy;
          r.gz += t.gpr * dz;
        }
      }
    });
  }
  if (GRAD) {
    r.gx = lane_sum<kLanes>(r.gx);
    r.gy = lane_sum<kLanes>(r.gy);
    r.gz = lane_sum<kLanes>(r.gz);
  }
  if (OBJ == 0) {
    r.u = lane_sum<kLanes>(r.u);
    if (GRAD) r.us = lane_sum<kLanes>(r.us);
  } else {
    r.G = lane_sum<kLanes>(r.G);
    if (GRAD) r.Gs = lane_sum<kLanes>(r.Gs);
  }
  return r;
}

// The same in fixed point by kBatchLanes lanes, to lane 0 (every thread of the
// warp calls it).
template <int OBJ, bool GRAD>
__device__ __forceinline__ ObjSums objective_sums_fixed(const P &c, const D &d, int i, int lane, const double4_32a *q,
                                                        const FixPos *x) {
  ObjSums r{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  FixSums s{0, 0, 0, 0};
  FixForce f{0, 0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f};  // psi d (potential energy) or the slope of chi / 8 (pressure)
  auto in_double = [&](const PairTerms &t, double dx, double dy, double dz, int) {
    if (OBJ == 0) {
      r.u += 0.5 * t.phi;
      if (GRAD) {
        r.us += 0.5 * t.dphis;
        r.gx -= t.f * dx;
        r.gy -= t.f * dy;
        r.gz -= t.f * dz;
      }
    } else {
      r.G += 0.5 * t.g;
      if (GRAD) {
        r.Gs += 0.5 * t.gs;
        r.gx += t.gpr * dx;
        r.gy += t.gpr * dy;
        r.gz += t.gpr * dz;
      }
    }
  };
  bool near = false;
  float psi = 0.f;
  int cnt = 0;
  if (i < c.n) {
    cnt = d.cnt[i];
    for_pairs_fixed<kBatchLanes>(
        c, d, i, lane, x,
        [&](bool take, const FixSep &sep, uint64_t R, int) {
          if (GRAD) {
            const FixTerms t = fix_terms(c, R);
            fix_sums_add(s, take, t.y3, R);
            const int64_t v = OBJ == 0 ? fix_psi(c, t) : fix_dsigma(c, t);
            fix_add(f, take ? v : 0, sep);
            if (OBJ == 1) psi += (float)fix_shi(take ? fix_psi(c, t) : 0);
          } else {
            uint64_t y2, z;
            fix_powers(fix_y(c, R), y2, z);
            fix_sums_add(s, take, z, R);
          }
        },
        [&](uint32_t e) {
          near = true;
          one_pair(c, e, q, make_home(c, q[i]), in_double);
        });
  }
  __syncwarp();
  lane_sums<kBatchLanes>(s);
  if (GRAD) lane_sums<kBatchLanes>(f);
  if (GRAD && OBJ == 1) {
#pragma unroll
    for (int o = 1; o < kBatchLanes; o <<= 1) psi += __shfl_xor_sync(0xffffffffu, psi, o);
    f.s = psi;
  }
  if (__any_sync(0xffffffffu, near)) {
    if (GRAD) {
      r.gx = lane_sum<kBatchLanes>(r.gx);
      r.gy = lane_sum<kBatchLanes>(r.gy);
      r.gz = lane_sum<kBatchLanes>(r.gz);
    }
    if (OBJ == 0) {
      r.u = lane_sum<kBatchLanes>(r.u);
      if (GRAD) r.us = lane_sum<kBatchLanes>(r.us);
    } else {
      r.G = lane_sum<kBatchLanes>(r.G);
      if (GRAD) r.Gs = lane_sum<kBatchLanes>(r.Gs);
    }
  }
  if (lane != 0 || i >= c.n) return r;
  if (cnt > kFixSumsRow || (GRAD && !(OBJ == 0 ? sums_fit(f, cnt) : derivative_sums_fit(c, f, cnt)))) {  // the row again in double
    r = ObjSums{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const Home h = make_home(c, q[i]);
    for (int k = 0; k < cnt; k++) one_pair(c, d.nbr[(size_t)i * c.cap + k], q, h, in_double);
    return r;
  }
  const double3 t = fix_sums_double(c, s);  // x^-6, x^-12, x^2
  if (OBJ == 0) {
    r.u += 2.0 * c.eps * ((t.y - t.x) + (c.c2 * t.z + c.c0 * (double)s.m));
    if (GRAD) {
      const double3 g = fix_vector(f, c.e_s2);
      r.us += c.e_s * (12.0 * (2.0 * t.y - t.x) - 4.0 * c.c2 * t.z);
      r.gx -= g.x;
      r.gy -= g.y;
      r.gz -= g.z;
    }
  } else {
    r.G += c.eps * (12.0 * (t.x - 2.0 * t.y) + 4.0 * c.c2 * t.z);
    if (GRAD) {
      const double3 g = fix_vector(f, -8.0 * c.e_s2);
      r.Gs += c.e_s * (72.0 * (t.x - 4.0 * t.y) - 8.0 * c.c2 * t.z);
      r.gx += g.x;
      r.gy += g.y;
      r.gz += g.z;
    }
  }
  return r;
}

// The force on particle i in fixed point, to lane 0 (every thread of the warp
// calls it).
__device__ __forceinline__ double3 force_sums_fixed(const P &c, const D &d, int i, int lane, const double4_32a *q,
                                                    const FixPos *x) {
  FixForce f{0, 0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f};
  double3 n = make_double3(0.0, 0.0, 0.0);
  auto in_double = [&](const PairTerms &t, double dx, double dy, double dz, int) {
    n.x += t.f * dx;
    n.y += t.f * dy;
    n.z += t.f * dz;
  };
  bool near = false;
  int cnt = 0;
  if (i < c.n) {
    cnt = d.cnt[i];
    for_pairs_fixed<kStepLanes>(
        c, d, i, lane, x,
        [&](bool take, const FixSep &sep, uint64_t R, int) {
          const int64_t v = fix_psi(c, fix_terms(c, R));
          fix_add(f, take ? v : 0, sep);
        },
        [&](uint32_t e) {
          near = true;
          one_pair(c, e, q, make_home(c, q[i]), in_double);
        });
  }
  __syncwarp();
  lane_sums<kStepLanes>(f);
  if (__any_sync(0xffffffffu, near)) n = make_double3(lane_sum<kStepLanes>(n.x), lane_sum<kStepLanes>(n.y), lane_sum<kStepLanes>(n.z));
  if (lane != 0 || i >= c.n) return n;
  if (!sums_fit(f, cnt)) {
    n = make_double3(0.0, 0.0, 0.0);
    const Home h = make_home(c, q[i]);
    for (int k = 0; k < cnt; k++) one_pair(c, d.nbr[(size_t)i * c.cap + k], q, h, in_double);
    return n;
  }
  const double3 F = fix_vector(f, c.e_s2);
  return make_double3(F.x + n.x, F.y + n.y, F.z + n.z);
}

// One step from the half-step positions q (x in fixed point): the forces F
// there (the lanes of a particle), then, by one thread per particle, p_out =
// p_in + F dt, q_out = q + p_out dt/2, the next step's first half-drift qh_next
// = q_out + p_out dt/2, and F itself where f_out is given.  Also the segment's
// displacement check (a particle more than margin/2 from q0, where the
// segment's list was built).  12.0 us at 4,000 particles (18.9 with the terms in
// double), a chain of launch, five or six entries a lane, the sum over the
// lanes and the update: the update's FP64 by a lane in eight of every warp, not
// by the block's first threads, cost 2 us of it.
template <bool FIXED>
__global__ void __launch_bounds__(kT) k_step(P c, D d, const double4_32a *q, const double4_32a *p_in, double4_32a *q_out,
                                             double4_32a *p_out, double4_32a *qh_next, const double4_32a *q0,
                                             double4_32a *f_out, const FixPos *x, FixPos *x_out, FixPos *xh_next) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kL = FIXED ? kStepLanes : kLanes;
  int i = tid / kL;
  const int lane = tid % kL;
  double3 F = make_double3(0.0, 0.0, 0.0);
  if (FIXED) {
    F = force_sums_fixed(c, d, i, lane, q, x);
  } else {
    if (i < c.n) {
      const Home h = make_home(c, q[i]);
      for_pairs(c, d, i, lane, q, h, [&](const PairTerms &t, double dx, double dy, double dz, int) {
        F.x += t.f * dx;
        F.y += t.f * dy;
        F.z += t.f * dz;
      });
    }
    F = make_double3(lane_sum<kL>(F.x), lane_sum<kL>(F.y), lane_sum<kL>(F.z));
  }
  // the block's particles move on to its first threads, one each: the FP64
  // work below is then a warp's, not four
  __shared__ double3 sF[kT / kL];
  if (lane == 0) sF[threadIdx.x / kL] = F;
  __syncthreads();
  i = blockIdx.x * (kT / kL) + threadIdx.x;
  if (threadIdx.x >= kT / kL || i >= c.n) return;
  F = sF[threadIdx.x];
  const double4_32a qi = q[i], z = q0[i];
  const double ux = qi.x - z.x, uy = qi.y - z.y, uz = qi.z - z.z;
  if (ux * ux + uy * uy + uz * uz > c.half_margin2) atomicMax(d.flag + 1, 1);
  if (f_out) f_out[i] = make_double4_32a(F.x, F.y, F.z, 0.0);
  double4_32a b = p_in[i];
  b.x += F.x * c.dt;
  b.y += F.y * c.dt;
  b.z += F.z * c.dt;
  p_out[i] = b;
  double4_32a a = qi;
  a.x += b.x * c.dt2;
  a.y += b.y * c.dt2;
  a.z += b.z * c.dt2;
  q_out[i] = a;
  if (FIXED) x_out[i] = fix_position(a.x, a.y, a.z, 0);
  a.x += b.x * c.dt2;
  a.y += b.y * c.dt2;
  a.z += b.z * c.dt2;
  qh_next[i] = a;
  if (FIXED) xh_next[i] = fix_position(a.x, a.y, a.z, 0);
}

// A segment's first state from (q, p): with wrap, positions into the box, q - k L
// per axis with k = floor(q / L) (particles already inside keep their bits), and
// the checkpoint; then state 0 of the segment, the float copy for the list
// test and the first half-drift.  The backward pass calls it without wrap on the
// checkpoint (ckq = ckp = null).
__global__ void k_begin(P c, D d, const double4_32a *q, const double4_32a *p, double4_32a *ckq, double4_32a *ckp, int wrap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.n) return;
  double4_32a a = q[i];
  const double4_32a b = p[i];
  if (wrap) {
    const double kx = floor(a.x * c.inv_L[0]), ky = floor(a.y * c.inv_L[1]), kz = floor(a.z * c.inv_L[2]);
    if (kx != 0.0) a.x = fma(-kx, c.L[0], a.x);
    if (ky != 0.0) a.y = fma(-ky, c.L[1], a.y);
    if (kz != 0.0) a.z = fma(-kz, c.L[2], a.z);
  }
  if (ckq) {
    ckq[i] = a;
    ckp[i] = b;
  }
  d.segq[i] = a;
  d.segp[i] = b;
  d.qf[i] = make_float4((float)a.x, (float)a.y, (float)a.z, 0.f);
  a.x += b.x * c.dt2;
  a.y += b.y * c.dt2;
  a.z += b.z * c.dt2;
  const size_t at = (size_t)c.n + i;
  d.segqh[at] = a;
  if (c.fixed) d.segxqh[at] = fix_position(a.x, a.y, a.z, 0);
}

// A window's first half step in fixed point, where the steps before it did not
// leave it (k_begin and k_step write it within a window).
__global__ void k_window(P c, D d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c.n) return;
  const double4_32a a = d.segqh[(size_t)c.n + i];
  d.segxqh[(size_t)c.n + i] = fix_position(a.x, a.y, a.z, 0);
}

// The reverse of a step's second half-drift q_n = qh + dt/2 p_n for particle
// i, from the adjoints a, b of (q_n, p_n): a_p += dt/2 a_q.  tmp receives the
// adjoint of p after the kick (the neighbours' H v reads it), aqh that of qh.
__device__ __forceinline__ void reverse_drift(const P &c, const D &d, int i, const double4_32a &a, double4_32a b,
                                              double4_32a *tmp) {
  b.x += c.dt2 * a.x;
  b.y += c.dt2 * a.y;
  b.z += c.dt2 * a.z;
  tmp[i] = b;
  d.aqh[i] = a;
}

// The objective at states first .. first + gridDim.y - 1 of the segment,
// weighted: values (and, with GRAD, the epsilon and sigma derivatives) into the
// running sums, and with GRAD w dj/dq of state k into segg[k].  All states of a
// segment share its list, so one launch takes them together: one state of 4,000
// particles leaves the GPU mostly idle and cost 9 us forward and 10 backward, in
// a launch of 20 it costs 3.2 and 4.7 (bound by the integer units).
template <int OBJ, bool GRAD, bool FIXED>
__global__ void __launch_bounds__(kT) k_objective(P c, D d, double w, int first) {
  __shared__ double sh[96];
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kL = FIXED ? kBatchLanes : kLanes;
  const int i = tid / kL, lane = tid % kL;
  const size_t at = (size_t)c.n * (first + blockIdx.y);
  const double4_32a *q = d.segq + at;
  const ObjSums r = FIXED ? objective_sums_fixed<OBJ, GRAD>(c, d, i, lane, q, d.segxq + at) : objective_sums<OBJ, GRAD>(c, d, i, lane, q);
  double val = 0, ge = 0, gs = 0;
  if (i < c.n && lane == 0) {
    const double scale = OBJ == 0 ? 1.0 / (double)c.n : 1.0 / (3.0 * c.volume);
    if (OBJ == 0) {
      val = r.u * scale;
      ge = r.u / c.eps * scale;
      gs = r.us * scale;
    } else {
      const double4_32a pi = d.segp[at + i];
      const double ke = 0.5 * (pi.x * pi.x + pi.y * pi.y + pi.z * pi.z);
      val = (2.0 * ke - r.G) * scale;
      ge = -r.G / c.eps * scale;
      gs = -r.Gs * scale;
    }
    if (GRAD) d.segg[at + i] = make_double4_32a(w * r.gx * scale, w * r.gy * scale, w * r.gz * scale, 0.0);
  }
  block_sum3(val, ge, gs, sh);
  partials_accumulate(d, val, ge, gs, w);
}

// sum_j dF_ij/dsigma of the half steps first .. first + gridDim.y - 1 of the
// segment, into segs (fixed-point form; the double form takes it in k_reverse).
__global__ void __launch_bounds__(kT) k_force_sigma(P c, D d, int first) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kL = kBatchLanes;
  const int i = tid / kL, lane = tid % kL;
  const size_t at = (size_t)c.n * (first + blockIdx.y);
  const double4_32a *q = d.segqh + at;
  double3 S = make_double3(0.0, 0.0, 0.0);
  auto in_double = [&](const PairTerms &t, double dx, double dy, double dz, int) {
    S.x += t.fs * dx;
    S.y += t.fs * dy;
    S.z += t.fs * dz;
  };
  FixForce f{0, 0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f};
  float psi = 0.f;
  bool near = false;
  int cnt = 0;
  if (i < c.n) {
    cnt = d.cnt[i];
    for_pairs_fixed<kL>(
        c, d, i, lane, d.segxqh + at,
        [&](bool take, const FixSep &sep, uint64_t R, int) {
          const FixTerms t = fix_terms(c, R);
          fix_add(f, take ? fix_dsigma(c, t) : 0, sep);
          psi += (float)fix_shi(take ? fix_psi(c, t) : 0);
        },
        [&](uint32_t e) {
          near = true;
          one_pair(c, e, q, make_home(c, q[i]), in_double);
        });
  }
  __syncwarp();
  lane_sums<kL>(f);
#pragma unroll
  for (int o = 1; o < kL; o <<= 1) psi += __shfl_xor_sync(0xffffffffu, psi, o);
  f.s = psi;
  if (__any_sync(0xffffffffu, near)) S = make_double3(lane_sum<kL>(S.x), lane_sum<kL>(S.y), lane_sum<kL>(S.z));
  if (i >= c.n || lane != 0) return;
  if (derivative_sums_fit(c, f, cnt)) {
    const double3 v = fix_vector(f, 8.0 * c.e_s3);
    S = make_double3(S.x + v.x, S.y + v.y, S.z + v.z);
  } else {  // the row again in double
    S = make_double3(0.0, 0.0, 0.0);
    const Home h = make_home(c, q[i]);
    for (int k = 0; k < cnt; k++) one_pair(c, d.nbr[(size_t)i * c.cap + k], q, h, in_double);
  }
  d.segs[at + i] = make_double4_32a(S.x, S.y, S.z, 0.0);
}

// The objective's terms of state k added to its adjoints a, b (w dj/dq from
// segg; dj/dp of the pressure here), then the reverse of step k's second half-drift.
__device__ __forceinline__ void state_terms(const P &c, const D &d, int i, size_t at, double w, double4_32a a, double4_32a b,
                                            double4_32a *tmp) {
  const double4_32a g = d.segg[at + i];
  a.x += g.x;
  a.y += g.y;
  a.z += g.z;
  if (c.objective == 1) {
    const double4_32a pi = d.segp[at + i];
    const double k = 2.0 * w / (3.0 * c.volume);
    b.x += k * pi.x;
    b.y += k * pi.y;
    b.z += k * pi.z;
  }
  reverse_drift(c, d, i, a, b, tmp);
}

// The segment's last state (number len): from the adjoints aq, ap of the state
// that follows it.
__global__ void k_seed(P c, D d, int len, double w, double4_32a *tmp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c.n) state_terms(c, d, i, (size_t)c.n * len, w, d.aq[i], d.ap[i], tmp);
}

// The rest of the reverse of step k at its half-step positions (kick and first
// half-drift).  In: tmp (read by the neighbours too) and aqh from the reverse of
// its second half-drift; the force there and, in the fixed-point form, its sigma
// derivative (the double form takes it along here: pair terms once more in a
// launch of their own cost 16,384 particles 80 us a step of 873).  Parameter
// terms dt * ap . dF/dtheta into part[k] (slots 1, 2).  For k > 1 it goes on
// with the objective's terms of state k - 1 and the reverse of step k - 1's
// second half-drift, into tmp_out (not tmp: other particles' lanes still read
// it) and aqh; for k = 1 aq, ap receive the adjoints of the segment's first
// state.  25 us at 4,000 particles (the FP64 pipe has 13 instructions a pair,
// 8 us of it; 45 us with all terms in double and the objective in it).
template <bool FIXED>
__global__ void __launch_bounds__(kT) k_reverse(P c, D d, int k, const double4_32a *tmp, double w, double4_32a *tmp_out) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kL = FIXED ? kStepLanes : kLanes;
  int i = tid / kL;
  const int lane = tid % kL;
  const size_t at = (size_t)c.n * k;
  const double4_32a *qh = d.segqh + at;
  double hx = 0, hy = 0, hz = 0;
  double sx = 0, sy = 0, sz = 0;  // double form: the force's sigma derivative
  double4_32a vi = i < c.n ? tmp[i] : make_double4_32a(0.0, 0.0, 0.0, 0.0);
  auto in_double = [&](const PairTerms &t, double dx, double dy, double dz, int j) {
    const double4_32a vj = tmp[j];
    const double wx = vi.x - vj.x, wy = vi.y - vj.y, wz = vi.z - vj.z;
    const double dw = dx * wx + dy * wy + dz * wz;
    // (H v)_i = sum_j f (v_i - v_j) + (f'/r) d (d . (v_i - v_j))
    hx += t.f * wx + t.fpr * dx * dw;
    hy += t.f * wy + t.fpr * dy * dw;
    hz += t.f * wz + t.fpr * dz * dw;
    if (!FIXED) {
      sx += t.fs * dx;
      sy += t.fs * dy;
      sz += t.fs * dz;
    }
  };
  if (FIXED) {
    // reduced sums psi w and (psi' / x) / 48 (d . w) d
    double ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0;
    if (i < c.n)
      for_pairs_fixed<kL>(
          c, d, i, lane, d.segxqh + at,
          [&](bool take, const FixSep &sep, uint64_t R, int j) {
            const double4_32a vj = tmp[j];
            const FixTerms t = fix_terms(c, R);
            const int64_t psi = take ? fix_psi(c, t) : 0, slope = take ? fix_psi_slope(t) : 0;
            // the separation as doubles: high words and rests in units of 2^-59
            auto whole = [](int h, float l) {
              return fix_double(((int64_t)h << 30) + (int64_t)__float2int_rn(l * 2147483648.0f), 59);
            };
            const double dx = whole(sep.x, sep.lx), dy = whole(sep.y, sep.ly), dz = whole(sep.z, sep.lz);
            const double wx = vi.x - vj.x, wy = vi.y - vj.y, wz = vi.z - vj.z;
            const double p = fix_double(psi, 55), s = fix_double(slope, 55) * fma(dz, wz, fma(dy, wy, dx * wx));
            ax = fma(p, wx, ax);
            ay = fma(p, wy, ay);
            az = fma(p, wz, az);
            bx = fma(s, dx, bx);
            by = fma(s, dy, by);
            bz = fma(s, dz, bz);
          },
          [&](uint32_t e) { one_pair(c, e, qh, make_home(c, qh[i]), in_double); });
    __syncwarp();
    const double e4 = 48.0 * c.e_s4;
    hx = fma(c.e_s2, ax, fma(e4, bx, hx));
    hy = fma(c.e_s2, ay, fma(e4, by, hy));
    hz = fma(c.e_s2, az, fma(e4, bz, hz));
  } else if (i < c.n) {
    const Home h = make_home(c, qh[i]);
    for_pairs(c, d, i, lane, qh, h, in_double);
  }
  hx = lane_sum<kL>(hx);
  hy = lane_sum<kL>(hy);
  hz = lane_sum<kL>(hz);
  // one thread per particle from here on, as in k_step
  __shared__ double3 sH[kT / kL], sS[FIXED ? 1 : kT / kL];
  if (lane == 0) sH[threadIdx.x / kL] = make_double3(hx, hy, hz);
  if (!FIXED) {
    sx = lane_sum<kL>(sx);
    sy = lane_sum<kL>(sy);
    sz = lane_sum<kL>(sz);
    if (lane == 0) sS[threadIdx.x / kL] = make_double3(sx, sy, sz);
  }
  __syncthreads();
  i = blockIdx.x * (kT / kL) + threadIdx.x;
  double te = 0, ts = 0;
  if (threadIdx.x < kT / kL && i < c.n) {
    vi = tmp[i];
    hx = sH[threadIdx.x].x;
    hy = sH[threadIdx.x].y;
    hz = sH[threadIdx.x].z;
    // parameter terms: dt * a_p . dF_i/deps (= F_i/eps), dt * a_p . dF_i/dsigma
    const double4_32a F = d.segf[at + i];
    const double3 S = FIXED ? make_double3(d.segs[at + i].x, d.segs[at + i].y, d.segs[at + i].z) : sS[threadIdx.x];
    te = c.dt * (vi.x * F.x + vi.y * F.y + vi.z * F.z) / c.eps;
    ts = c.dt * (vi.x * S.x + vi.y * S.y + vi.z * S.z);
    // kick: a_qh = a_q - dt H a_p ; then drift qh = q + dt/2 p : a_p += dt/2 a_qh
    double4_32a a = d.aqh[i], pb = vi;
    a.x -= c.dt * hx;
    a.y -= c.dt * hy;
    a.z -= c.dt * hz;
    pb.x += c.dt2 * a.x;
    pb.y += c.dt2 * a.y;
    pb.z += c.dt2 * a.z;
    if (k > 1) {
      state_terms(c, d, i, (size_t)c.n * (k - 1), w, a, pb, tmp_out);
    } else {
      d.aq[i] = a;
      d.ap[i] = pb;
    }
  }
  static_assert(kT / kL <= 32, "one warp holds the block's particles");
  if (threadIdx.x >= 32) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    te += __shfl_down_sync(0xffffffffu, te, o);
    ts += __shfl_down_sync(0xffffffffu, ts, o);
  }
  if (threadIdx.x == 0) {
    double *part = d.part + 3 * ((size_t)k * gridDim.x + blockIdx.x);
    part[1] = te;
    part[2] = ts;
  }
}

// Adds the parameter terms of steps 1 .. len (k_reverse's partials) to the
// running sums, in a fixed order.
__global__ void __launch_bounds__(1024) k_reverse_sums(D d, int len, int blocks) {
  __shared__ double sh[96];
  double none = 0, te = 0, ts = 0;
  const double *part = d.part + 3 * (size_t)blocks;
  for (int k = threadIdx.x; k < len * blocks; k += blockDim.x) {
    te += part[3 * (size_t)k + 1];
    ts += part[3 * (size_t)k + 2];
  }
  block_sum3(none, te, ts, sh);
  if (threadIdx.x == 0) {
    d.acc[1] += te;
    d.acc[2] += ts;
  }
}

}  // namespace adj
}  // namespace mdg

using namespace mdg::adj;
using mdg::FixPos;

struct mdg_adjoint {
  mdg_adjoint_params prm;
  std::string err;
  P c;
  D d;
  cudaStream_t s = nullptr;
  int grid = 1;    // one thread per particle
  int gridp = 1;   // pair kernels of one step
  int grids = 1;   // the kernels over all states of a segment
  int gridb = 1;   // kBuildLanes threads per particle (list build)
  int nck = 0;
  int window = 1;  // steps whose forces, derivatives and fixed-point positions are held
  char *slab = nullptr;  // every device array
  bool forward_done = false;
  // the device work of a forward and of a backward pass, captured once and
  // replayed (every pointer is fixed at creation)
  cudaGraphExec_t gx_forward = nullptr, gx_backward = nullptr;
};

namespace {

int afail(mdg_adjoint *a, int code, const std::string &m) {
  if (a) a->err = m;
  return code;
}

#define MDG_ACK(call)                                                                                    \
  do {                                                                                                   \
    cudaError_t e_ = (call);                                                                             \
    if (e_ != cudaSuccess) return afail(a, MDG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// The device's arrays as the window from state lo of the segment on sees them.
D window(const mdg_adjoint *a, int lo) {
  D d = a->d;
  const size_t at = (size_t)a->c.n * lo;
  d.segq += at;
  d.segp += at;
  d.segqh += at;
  return d;
}

// Steps lo + 1 .. lo + m of a segment from its state lo and the half-drift that
// follows it: states and half steps (and the forces at the half steps).  again:
// the same steps once more, for what the window holds; they write the same
// states.  The segment's list is built ahead of its first window.
void run_steps(mdg_adjoint *a, int lo, int m, bool forces, bool again) {
  const size_t N = (size_t)a->c.n;
  D d = window(a, lo);
  if (lo == 0 && !again) k_build<<<a->gridb, kT, 0, a->s>>>(a->c, d, d.segq);
  else if (a->c.fixed) k_window<<<a->grid, kT, 0, a->s>>>(a->c, d);
  for (int k = 1; k <= m; k++) {
    const size_t at = N * k, before = N * (k - 1), after = N * (k + 1);
    double4_32a *f = forces ? d.segf + at : nullptr;
    // the half step that follows the segment's last state is written too, and not used
    if (a->c.fixed)
      k_step<true><<<a->gridp, kT, 0, a->s>>>(a->c, d, d.segqh + at, d.segp + before, d.segq + at, d.segp + at, d.segqh + after,
                                              a->d.segq, f, d.segxqh + at, d.segxq + at, d.segxqh + after);
    else
      k_step<false><<<a->gridp, kT, 0, a->s>>>(a->c, d, d.segqh + at, d.segp + before, d.segq + at, d.segp + at, d.segqh + after,
                                               a->d.segq, f, nullptr, nullptr, nullptr);
  }
}

// The longest window's arrays: 1 GB (4,000 particles 1,677 steps, 100,000 67).
constexpr size_t kWindowBytes = (size_t)1 << 30;

constexpr int kStates = 32768;  // states a launch (a grid's second dimension ends at 65,535)

template <bool GRAD>
void launch_objective(mdg_adjoint *a, const D &d, int len, double w) {
  for (int first = 1; first <= len; first += kStates) {
    const dim3 grid(a->grids, len - first + 1 < kStates ? len - first + 1 : kStates);
    if (a->c.objective == 0) {
      if (a->c.fixed) k_objective<0, GRAD, true><<<grid, kT, 0, a->s>>>(a->c, d, w, first);
      else k_objective<0, GRAD, false><<<grid, kT, 0, a->s>>>(a->c, d, w, first);
    } else {
      if (a->c.fixed) k_objective<1, GRAD, true><<<grid, kT, 0, a->s>>>(a->c, d, w, first);
      else k_objective<1, GRAD, false><<<grid, kT, 0, a->s>>>(a->c, d, w, first);
    }
  }
}

void launch_force_sigma(mdg_adjoint *a, const D &d, int len) {
  for (int first = 1; first <= len; first += kStates) {
    const dim3 grid(a->grids, len - first + 1 < kStates ? len - first + 1 : kStates);
    k_force_sigma<<<grid, kT, 0, a->s>>>(a->c, d, first);
  }
}

// The horizon from the state in d.q, d.p: per segment its checkpoint and list,
// its steps, and the objective at its states.
int enqueue_forward(mdg_adjoint *a) {
  const size_t N = (size_t)a->c.n;
  D &d = a->d;
  MDG_ACK(cudaMemsetAsync(d.flag, 0, 2 * sizeof(int), a->s));
  MDG_ACK(cudaMemsetAsync(d.acc, 0, 3 * sizeof(double), a->s));
  const int Ns = a->prm.steps, K = a->prm.checkpoint_every;
  const double4_32a *q = d.q, *p = d.p;
  for (int start = 0; start < Ns; start += K) {
    const int len = Ns - start < K ? Ns - start : K;
    const size_t ck = N * (size_t)(start / K);
    k_begin<<<a->grid, kT, 0, a->s>>>(a->c, d, q, p, d.ckq + ck, d.ckp + ck, 1);
    for (int lo = 0; lo < len; lo += a->window) {
      const int m = std::min(a->window, len - lo);
      run_steps(a, lo, m, false, false);
      launch_objective<false>(a, window(a, lo), m, 1.0 / Ns);
    }
    q = d.segq + N * len;
    p = d.segp + N * len;
  }
  return cudaGetLastError() == cudaSuccess ? MDG_OK : afail(a, MDG_ERR_CUDA, "adjoint forward launch failed");
}

// Reverse of the horizon, segment by segment from the last: recompute the
// segment from its checkpoint (with the same list), then window by window from
// its last the objective's gradient at all states and the forces' sigma
// derivatives at all half steps, and the reverse of the steps.  The windows
// before the last run their steps once more for it.
int enqueue_backward(mdg_adjoint *a) {
  const size_t N = (size_t)a->c.n, bytes = N * 32;
  D &d = a->d;
  const int Ns = a->prm.steps, K = a->prm.checkpoint_every;
  const double w = 1.0 / Ns;
  MDG_ACK(cudaMemsetAsync(d.aq, 0, bytes, a->s));
  MDG_ACK(cudaMemsetAsync(d.ap, 0, bytes, a->s));
  MDG_ACK(cudaMemsetAsync(d.acc, 0, 3 * sizeof(double), a->s));
  for (int seg_end = Ns; seg_end > 0;) {
    const int seg_start = ((seg_end - 1) / K) * K;
    const int len = seg_end - seg_start;
    const size_t ck = N * (size_t)(seg_start / K);
    k_begin<<<a->grid, kT, 0, a->s>>>(a->c, d, d.ckq + ck, d.ckp + ck, nullptr, nullptr, 0);
    const int last = (len - 1) / a->window * a->window;
    for (int lo = 0; lo < last; lo += a->window) run_steps(a, lo, a->window, false, false);
    for (int lo = last; lo >= 0; lo -= a->window) {
      const int m = std::min(a->window, len - lo);
      const D dw = window(a, lo);
      run_steps(a, lo, m, true, lo < last);
      launch_objective<true>(a, dw, m, w);
      if (a->c.fixed) launch_force_sigma(a, dw, m);
      double4_32a *tmp = d.tmp, *tmp_alt = d.tmp2;
      k_seed<<<a->grid, kT, 0, a->s>>>(a->c, dw, m, w, tmp);
      for (int k = m; k >= 1; k--) {
        if (a->c.fixed) k_reverse<true><<<a->gridp, kT, 0, a->s>>>(a->c, dw, k, tmp, w, tmp_alt);
        else k_reverse<false><<<a->gridp, kT, 0, a->s>>>(a->c, dw, k, tmp, w, tmp_alt);
        std::swap(tmp, tmp_alt);
      }
      k_reverse_sums<<<1, 1024, 0, a->s>>>(d, m, a->gridp);
    }
    seg_end = seg_start;
  }
  return cudaGetLastError() == cudaSuccess ? MDG_OK : afail(a, MDG_ERR_CUDA, "adjoint backward launch failed");
}

// Runs `enqueue` as a CUDA graph captured on first use.
int run_graph(mdg_adjoint *a, cudaGraphExec_t *gx, int (*enqueue)(mdg_adjoint *)) {
  if (!*gx) {
    MDG_ACK(cudaStreamBeginCapture(a->s, cudaStreamCaptureModeThreadLocal));
    const int rc = enqueue(a);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(a->s, &g);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    MDG_ACK(e);
    const cudaError_t ei = cudaGraphInstantiate(gx, g, 0);
    cudaGraphDestroy(g);
    MDG_ACK(ei);
  }
  MDG_ACK(cudaGraphLaunch(*gx, a->s));
  return MDG_OK;
}

}  // namespace

extern "C" {

void mdg_adjoint_params_default(mdg_adjoint_params *p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->cutoff = 2.5;
  p->margin = 2.0;
  p->dt = 0.002;
  p->epsilon = 1.0;
  p->sigma = 1.0;
  p->steps = 200;
  p->checkpoint_every = 20;
  p->objective = MDG_OBJ_POTENTIAL;
}

int mdg_adjoint_create(const mdg_adjoint_params *p, int32_t n, mdg_adjoint **out) {
  if (!p || !out || n <= 1 || p->steps <= 0 || p->checkpoint_every <= 0 || !(p->dt > 0) || !(p->epsilon > 0) ||
      !(p->sigma > 0) || (p->objective != MDG_OBJ_POTENTIAL && p->objective != MDG_OBJ_PRESSURE))
    return MDG_ERR_INVALID;
  *out = nullptr;
  if (n >= kMaxAdjointParticles) return MDG_ERR_INVALID;
  const double sl = p->cutoff * p->sigma + p->margin;
  for (int k = 0; k < 3; k++)
    if (!(p->box[k] > 2.0 * sl)) return MDG_ERR_INVALID;
  mdg_adjoint *a = new mdg_adjoint();
  a->prm = *p;
  memset(&a->d, 0, sizeof(a->d));
  P &c = a->c;
  for (int k = 0; k < 3; k++) {
    c.L[k] = p->box[k];
    c.inv_L[k] = 1.0 / p->box[k];
  }
  c.eps = p->epsilon;
  c.sig = p->sigma;
  c.inv_s2 = 1.0 / (p->sigma * p->sigma);
  c.e_s = p->epsilon / p->sigma;
  c.e_s2 = c.e_s / p->sigma;
  c.e_s3 = c.e_s2 / p->sigma;
  c.e_s4 = c.e_s3 / p->sigma;
  c.dt = p->dt;
  c.dt2 = 0.5 * p->dt;
  c.xc2 = p->cutoff * p->cutoff;
  const double s2 = 1.0 / c.xc2, s6 = s2 * s2 * s2, s8 = s6 * s2, s12 = s6 * s6, s14 = s12 * s2;
  c.c2 = 6.0 * s14 - 3.0 * s8;  // variables.cc:16-28 in sigma units
  c.c0 = -s12 + s6 - c.c2 / s2;
  const double ep = c.eps;
  c.kf6 = -48.0 * c.e_s2; c.kf0 = 24.0 * c.e_s2; c.kfc = 8.0 * c.c2 * c.e_s2;
  c.kp6 = 672.0 * c.e_s4; c.kp0 = -192.0 * c.e_s4;
  c.ke6 = 4.0 * ep; c.ke0 = -4.0 * ep; c.kec2 = 4.0 * ep * c.c2; c.kec0 = 4.0 * ep * c.c0;
  c.kd6 = 48.0 * c.e_s; c.kd0 = -24.0 * c.e_s; c.kdc = -8.0 * c.c2 * c.e_s;
  c.ks6 = -576.0 * c.e_s3; c.ks0 = 144.0 * c.e_s3; c.ksc = -16.0 * c.c2 * c.e_s3;
  c.kg6 = -48.0 * ep; c.kg0 = 24.0 * ep; c.kgc = 8.0 * ep * c.c2;
  c.kr6 = 576.0 * c.e_s2; c.kr0 = -144.0 * c.e_s2; c.krc = 16.0 * c.c2 * c.e_s2;
  c.kq6 = -576.0 * c.e_s; c.kq0 = 144.0 * c.e_s; c.kqc = -16.0 * c.c2 * c.e_s;
  c.sl2 = sl * sl;
  c.sl2f = (sl + 1e-3) * (sl + 1e-3);
  c.half_margin2 = 0.25 * p->margin * p->margin;
  // Fixed-point pair arithmetic where every listed pair, each particle within
  // margin / 2 of its place at the segment's start, stays below 4 sigma apart
  // on every axis, sigma^2 / r^2 fits its format beyond kFixNear and the cut-off
  // lies beyond it
  c.fixed = sl + p->margin < 3.9 && p->sigma >= 0.8 && p->sigma <= 1.8 && p->cutoff >= 1.0 ? 1 : 0;
  c.unit_sigma = p->sigma == 1.0 ? 1 : 0;
  if (c.fixed) {
    const double s2v = p->sigma * p->sigma, rcut = p->cutoff * p->sigma;
    c.fx_rc2 = (uint64_t)std::ldexp(rcut * rcut, mdg::kFixR2Bits);
    c.fx_near = (uint64_t)std::ldexp(mdg::kFixNear * s2v, mdg::kFixR2Bits);
    c.fx_s2 = (uint64_t)std::ldexp(s2v, 62);
    c.fx_c8 = mdg::fix_c8(8.0 * c.c2);
    derivative_fit(c);
    for (int k = 0; k < 3; k++) {
      const int64_t L = mdg::fix_from_double(p->box[k]);
      c.fx_L[k] = mdg::fix_shi(L);
      c.fx_l[k] = mdg::fix_rest(L);
    }
  }
  c.volume = p->box[0] * p->box[1] * p->box[2];
  c.n = n;
  c.objective = p->objective;
  const double rho = n / c.volume;
  c.cap = ((int)(rho * 4.18879020478639 * sl * sl * sl * 1.5 + 32) + 7) & ~7;
  a->grid = (n + kT - 1) / kT;
  a->gridp = (int)(((long long)n * (c.fixed ? kStepLanes : kLanes) + kT - 1) / kT);
  a->grids = c.fixed ? (int)(((long long)n * kBatchLanes + kT - 1) / kT) : a->gridp;
  a->gridb = (int)(((long long)n * kBuildLanes + kT - 1) / kT);
  a->nck = p->steps / p->checkpoint_every + 1;
  const size_t N = (size_t)n, K = (size_t)p->checkpoint_every;
  D &d = a->d;
  cudaError_t e = cudaSetDevice(p->device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&a->s, cudaStreamNonBlocking);
  const size_t X = c.fixed ? N : 0;
  const size_t step_bytes = N * (c.fixed ? 160 : 64);
  size_t W = std::max<size_t>(1, std::min(K, kWindowBytes / step_bytes));
  for (int pass = 0; pass < 2 && e == cudaSuccess; pass++) {
    mdg::Slab s;
    s.base = a->slab;
    for (auto v : {&d.q, &d.p, &d.aq, &d.ap, &d.aqh, &d.tmp, &d.tmp2}) s.take(v, N);
    s.take(&d.ckq, N * a->nck);
    s.take(&d.ckp, N * a->nck);
    for (auto v : {&d.segq, &d.segp}) s.take(v, N * (K + 1));
    s.take(&d.segqh, N * (K + 2));
    for (auto v : {&d.segf, &d.segg}) s.take(v, N * (W + 1));
    s.take(&d.segs, X * (W + 1));
    s.take(&d.segxq, X * (W + 1));
    s.take(&d.segxqh, X * (W + 2));
    s.take(&d.nbr, N * (size_t)c.cap);
    s.take(&d.cnt, N);
    s.take(&d.qf, N);
    s.take(&d.part, 3 * (size_t)std::max(a->gridp, a->grids) * (W + 1));
    s.take(&d.acc, 3);
    s.take(&d.flag, 2);
    s.take(&d.done, 1);
    if (pass == 0) {
      e = cudaMalloc((void **)&a->slab, s.used);
      if (e == cudaErrorMemoryAllocation && W > 1) {  // what is left beside the segment itself
        cudaGetLastError();
        e = cudaSuccess;
        a->slab = nullptr;
        W = (W + 1) / 2;
        pass = -1;
      }
    }
  }
  a->window = (int)W;
  if (e == cudaSuccess) e = cudaMemset(d.done, 0, sizeof(unsigned int));
  if (e != cudaSuccess) {
    fprintf(stderr, "mdg_adjoint_create: %s\n", cudaGetErrorString(e));
    mdg_adjoint_destroy(a);
    return MDG_ERR_CUDA;
  }
  *out = a;
  return MDG_OK;
}

int mdg_adjoint_destroy(mdg_adjoint *a) {
  if (!a) return MDG_OK;
  cudaSetDevice(a->prm.device);
  if (a->s) cudaStreamSynchronize(a->s);
  if (a->gx_forward) cudaGraphExecDestroy(a->gx_forward);
  if (a->gx_backward) cudaGraphExecDestroy(a->gx_backward);
  if (a->slab) cudaFree(a->slab);
  if (a->s) cudaStreamDestroy(a->s);
  delete a;
  return MDG_OK;
}

const char *mdg_adjoint_last_error(const mdg_adjoint *a) { return a ? a->err.c_str() : "null adjoint"; }

int mdg_adjoint_forward(mdg_adjoint *a, const double *q4, const double *p4, double *J) {
  if (!a || !q4 || !p4 || !J) return MDG_ERR_INVALID;
  MDG_ACK(cudaSetDevice(a->prm.device));
  const size_t N = (size_t)a->c.n, bytes = N * 32;
  D &d = a->d;
  MDG_ACK(cudaMemcpyAsync(d.q, q4, bytes, cudaMemcpyHostToDevice, a->s));
  MDG_ACK(cudaMemcpyAsync(d.p, p4, bytes, cudaMemcpyHostToDevice, a->s));
  const int rc = run_graph(a, &a->gx_forward, enqueue_forward);
  if (rc) return rc;
  int flag[2] = {0, 0};
  double acc[3];
  MDG_ACK(cudaMemcpyAsync(acc, d.acc, sizeof acc, cudaMemcpyDeviceToHost, a->s));
  MDG_ACK(cudaMemcpyAsync(flag, d.flag, sizeof flag, cudaMemcpyDeviceToHost, a->s));
  MDG_ACK(cudaStreamSynchronize(a->s));
  if (flag[0]) return afail(a, MDG_ERR_CAPACITY, "adjoint pair list capacity exceeded");
  if (flag[1])
    return afail(a, MDG_ERR_STATE, "a particle moved more than margin/2 within a checkpoint segment; raise margin");
  *J = acc[0];
  a->forward_done = true;
  return MDG_OK;
}

int mdg_adjoint_backward(mdg_adjoint *a, double *dq0, double *dp0, double *deps, double *dsigma) {
  if (!a) return MDG_ERR_INVALID;
  if (!a->forward_done) return afail(a, MDG_ERR_NOT_READY, "run mdg_adjoint_forward first");
  MDG_ACK(cudaSetDevice(a->prm.device));
  const size_t N = (size_t)a->c.n, bytes = N * 32;
  D &d = a->d;
  const int rc = run_graph(a, &a->gx_backward, enqueue_backward);
  if (rc) return rc;
  double acc[3];
  MDG_ACK(cudaMemcpyAsync(acc, d.acc, sizeof acc, cudaMemcpyDeviceToHost, a->s));
  if (dq0) MDG_ACK(cudaMemcpyAsync(dq0, d.aq, bytes, cudaMemcpyDeviceToHost, a->s));
  if (dp0) MDG_ACK(cudaMemcpyAsync(dp0, d.ap, bytes, cudaMemcpyDeviceToHost, a->s));
  MDG_ACK(cudaStreamSynchronize(a->s));
  // acc[1], acc[2]: objective parameter terms (weighted) plus the kick terms
  if (deps) *deps = acc[1];
  if (dsigma) *dsigma = acc[2];
  return MDG_OK;
}

}  // extern "C"

// Device functions shared by the step kernels: home cells and images, the
// FP64 pair loop, the Langevin noise, block sums.
#pragma once
#include "mdg_internal.cuh"

namespace mdg {

__device__ __forceinline__ double rcp_hh3(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

struct CellPos {
  int cx, cy, cz;
  bool edge;
};

__device__ __forceinline__ CellPos cell_pos(const Geom &g, int key) {
  CellPos r;
  cell_unkey(key, r.cx, r.cy, r.cz);
  r.edge = r.cx == 0 || r.cy == 0 || r.cz == 0 || r.cx == g.nc[0] - 1 || r.cy == g.nc[1] - 1 || r.cz == g.nc[2] - 1;
  return r;
}

// The same from the coordinates packed in the w word of qf / loc (equal
// between the two: both are written with the home cell of the last build).
__device__ __forceinline__ CellPos cell_pos_packed(const Geom &g, float w) {
  CellPos r;
  cell_unpack(w, r.cx, r.cy, r.cz);
  r.edge = r.cx == 0 || r.cy == 0 || r.cz == 0 || r.cx == g.nc[0] - 1 || r.cy == g.nc[1] - 1 || r.cz == g.nc[2] - 1;
  return r;
}

// Image of partner position qj seen from a particle in cell cp through stencil
// offset bits of entry e: +-L where the offset crosses the periodic boundary.
__device__ __forceinline__ void apply_image(const Geom &g, const CellPos &cp, uint32_t e, double4_32a &qj) {
  const int ox = entry_sx(e), oy = entry_sy(e), oz = entry_sz(e);
  if (ox == 0 && cp.cx == 0) qj.x -= g.L[0];
  else if (ox == 2 && cp.cx == g.nc[0] - 1) qj.x += g.L[0];
  if (oy == 0 && cp.cy == 0) qj.y -= g.L[1];
  else if (oy == 2 && cp.cy == g.nc[1] - 1) qj.y += g.L[1];
  if (oz == 0 && cp.cz == 0) qj.z -= g.L[2];
  else if (oz == 2 && cp.cz == g.nc[2] - 1) qj.z += g.L[2];
}

// Sum over the row of slot i of f(r) (q_j - q_i), f(r) = 24 r^-8 - 48 r^-14 + 8 C2,
// the force on i (fcalculator.cc:263-277 without the dt factor).
// `list`/`counts` is the inner (pruned) list in an ordinary step and the outer
// list for a stand-alone force evaluation.  With PRUNE the outer list is
// walked and every entry within the prune radius is copied to the inner row
// of slot i (d.pl); *kept receives the new row length.
template <bool PRUNE>
__device__ __forceinline__ double3 force_fp64(const Geom &g, const Dev &d, const double4_32a *__restrict__ pos, int i,
                                              const CellPos &cp, const uint32_t *__restrict__ list,
                                              const int *__restrict__ counts, int *kept) {
  const double4_32a qi = pos[i];
  int cnt = counts[i];
  if (!MDG_IN_RANGE(d.flags, kCheckStepRow, cnt, g.list_cap + 1)) cnt = 0;
  const uint32_t *row = list + i;
  const double thr = (double)g.prune_thr2;
  // r2 >= +0, so its bit pattern orders like the value (a NaN compares above
  // every finite bound): the cutoff tests run on the integer pipe instead of
  // the FP64 pipe (1/64 of the FP32 rate; 6 % of the FP64 step at 4M atoms)
  const long long rc2_bits = __double_as_longlong(g.rc2), thr_bits = __double_as_longlong(thr);
  int m = 0;
  double fx = 0.0, fy = 0.0, fz = 0.0;
  for (int k = 0; k < cnt; k++) {
    const uint32_t e = __ldg(row + (size_t)k * g.stride);
    if (!MDG_IN_RANGE(d.flags, kCheckStepSlot, entry_slot(e), g.n)) continue;
    double4_32a qj = ldg4(pos + entry_slot(e));
    if (cp.edge) apply_image(g, cp, e, qj);
    const double dx = qj.x - qi.x, dy = qj.y - qi.y, dz = qj.z - qi.z;
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (PRUNE && __double_as_longlong(r2) <= thr_bits) d.pl[(size_t)(m++) * g.stride + i] = e;
    if (__double_as_longlong(r2) <= rc2_bits) {
      const double inv = rcp_hh3(r2);
      const double i6 = inv * inv * inv;
      const double df = (i6 * inv) * fma(-48.0, i6, 24.0) + g.c2x8;
      fx = fma(df, dx, fx);
      fy = fma(df, dy, fy);
      fz = fma(df, dz, fz);
    }
  }
  if (PRUNE) *kept = m;
  return make_double3(fx, fy, fz);
}

// A pair's energy and virial term at r2, weighted 1/2, in the reference's
// expressions and rounding (observer.cc:17-79); zero beyond rc.
__device__ __forceinline__ void pair_observables(const Geom &g, double r2, double &e, double &v) {
  e = v = 0.0;
  if (r2 > g.rc2) return;
  const double r4 = __dmul_rn(r2, r2), r6 = __dmul_rn(r4, r2), r8 = __dmul_rn(r6, r2), r10 = __dmul_rn(r8, r2),
               r12 = __dmul_rn(r10, r2);
  e = 0.5 * (4.0 * (1.0 / r12 - 1.0 / r6 + __dmul_rn(g.c2, r2) + g.c0));
  v = 0.5 * ((__dsub_rn(__dmul_rn(24.0, r6), 48.0) / (__dmul_rn(__dmul_rn(r6, r6), r2)) + g.c2x8) * r2);
}

// Pair energy and virial sums of the outer row of slot i at q_end in double.
__device__ inline void observe_row_fp64(const Geom &g, const Dev &d, int i, const CellPos &cp, int cnt, double &pe,
                                        double &vir) {
  const double4_32a qi = d.q_end[i];
  for (int k = 0; k < cnt; k++) {
    const uint32_t e = d.nl[(size_t)k * g.stride + i];
    if (!MDG_IN_RANGE(d.flags, kCheckObserve, entry_slot(e), g.n)) continue;
    double4_32a qj = d.q_end[entry_slot(e)];
    if (cp.edge) apply_image(g, cp, e, qj);
    const double dx = __dsub_rn(qi.x, qj.x), dy = __dsub_rn(qi.y, qj.y), dz = __dsub_rn(qi.z, qj.z);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    double a, b;
    pair_observables(g, r2, a, b);
    pe += a;
    vir += b;
  }
}

__device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) and Box-Muller in float:
// the Langevin noise stream, keyed by seed, counted by (particle, step).
__device__ __forceinline__ void langevin_normals(uint64_t seed, uint32_t id, uint64_t step, double z[3]) {
  uint32_t c0 = id, c1 = (uint32_t)step, c2 = (uint32_t)(step >> 32), c3 = 0x4C4A4D44u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; r++) {
    if (r) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
    const uint32_t hi0 = mulhi32(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = mulhi32(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
  }
  const float s24 = 5.9604644775390625e-08f;
  const float u1 = (float)((c0 >> 8) + 1u) * s24, u2 = (float)(c1 >> 8) * s24;
  const float u3 = (float)((c2 >> 8) + 1u) * s24, u4 = (float)(c3 >> 8) * s24;
  const float twopi = 6.28318530717958647692f;
  const float ra = sqrtf(-2.0f * logf(u1)), rb = sqrtf(-2.0f * logf(u3));
  z[0] = (double)(ra * cosf(twopi * u2));
  z[1] = (double)(ra * sinf(twopi * u2));
  z[2] = (double)(rb * cosf(twopi * u4));
}

__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
  __syncthreads();
  return t;
}

}  // namespace mdg

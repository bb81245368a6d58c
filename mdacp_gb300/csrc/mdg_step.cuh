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

// A load of data that the kernel does not write (COH = false), or that it
// does (COH: the resident kernel, whose grid barriers make it visible).
template <bool COH>
__device__ __forceinline__ uint32_t ld_ro(const uint32_t *p) {
  if (!COH) return __ldg(p);
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
template <bool COH>
__device__ __forceinline__ int ld_ro(const int *p) {
  return COH ? (int)ld_ro<true>(reinterpret_cast<const uint32_t *>(p)) : *p;
}
template <bool COH>
__device__ __forceinline__ float4 ld_ro(const float4 *p) {
  if (!COH) return __ldg(p);
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
template <bool COH>
__device__ __forceinline__ double4_32a ld_ro(const double4_32a *p) {
  if (!COH) return ldg4(p);
  double4_32a v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p) : "memory");
  return v;
}

// Sum over the row of slot i of f(r) (q_j - q_i), f(r) = 24 r^-8 - 48 r^-14 + 8 C2,
// the force on i (fcalculator.cc:263-277 without the dt factor).
// `list`/`counts` is the inner (pruned) list in an ordinary step and the outer
// list for a stand-alone force evaluation.  With PRUNE the outer list is
// walked and every entry within the prune radius is copied to the inner row
// of slot i (d.pl); *kept receives the new row length.  COH: rows and positions
// that the calling kernel itself writes.
template <bool PRUNE, bool COH>
__device__ __forceinline__ double3 force_fp64(const Geom &g, const Dev &d, const double4_32a *__restrict__ pos, int i,
                                              const CellPos &cp, const uint32_t *__restrict__ list,
                                              const int *__restrict__ counts, int *kept) {
  const double4_32a qi = COH ? ld_ro<true>(pos + i) : pos[i];
  int cnt = ld_ro<COH>(counts + i);
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
    const uint32_t e = ld_ro<COH>(row + (size_t)k * g.stride);
    if (!MDG_IN_RANGE(d.flags, kCheckStepSlot, entry_slot(e), g.n)) continue;
    double4_32a qj = ld_ro<COH>(pos + entry_slot(e));
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

// Adds a pair's energy and virial term at r2, weighted 1/2, in the reference's
// expressions and rounding (observer.cc:17-79); nothing beyond rc (adding zeros
// there took the FP64 pipe 4 % of the observers' time).
__device__ __forceinline__ void pair_observables(const Geom &g, double r2, double &e, double &v) {
  if (r2 > g.rc2) return;
  const double r4 = __dmul_rn(r2, r2), r6 = __dmul_rn(r4, r2), r8 = __dmul_rn(r6, r2), r10 = __dmul_rn(r8, r2),
               r12 = __dmul_rn(r10, r2);
  e += 0.5 * (4.0 * (1.0 / r12 - 1.0 / r6 + __dmul_rn(g.c2, r2) + g.c0));
  v += 0.5 * ((__dsub_rn(__dmul_rn(24.0, r6), 48.0) / (__dmul_rn(__dmul_rn(r6, r6), r2)) + g.c2x8) * r2);
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
    pair_observables(g, r2, pe, vir);
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

// Neighbour-list entries whose index and position loads are issued together
// in the mixed-form force loop.
#ifndef MDG_STEP_UNROLL
#define MDG_STEP_UNROLL 4
#endif
constexpr int kUnroll = MDG_STEP_UNROLL;

// List rows requested into L2 this many entries ahead of the pair loop (0:
// none).  16 measured best at 4M atoms (step kernel 0.476 -> 0.440 ms; 8: 0.472,
// 12: 0.472, 20: 0.442, 24: 0.445, 32: 0.452, 64: 0.458).
#ifndef MDG_ENTRY_L2_AHEAD
#define MDG_ENTRY_L2_AHEAD 16
#endif
constexpr int kEntryAhead = MDG_ENTRY_L2_AHEAD;

// Walks the row of slot i on home-cell-local float positions and hands each
// entry's partner offset q_j - q_i and its r^2 to pair(e, dx, dy, dz, r2).
// The offset between the home cells of i and j is ox*w + s*(L - nc*w) per
// axis, s the periodic wrap of the stencil step, evaluated as the quadratic
// of axis_quad.  EDGE: the home cell touches the periodic boundary, so the
// offset is the quadratic; otherwise it is linear with the cell width as
// slope (b = 0, a = w: fmaf(fmaf(0, t, a), t, c) = fmaf(a, t, c) exactly), the
// width coming from the kernel parameters instead of two registers per axis.
// An entry whose slot a checked build rejects (code `site`) and the padding of
// the last batch get a partner at 1e30, whose r^2 overflows to +inf.
template <bool EDGE, int SITE, bool COH, int UNROLL, class Pair>
__device__ __forceinline__ void walk_row(const Geom &g, const Dev &d, const float4 *__restrict__ loc, int i,
                                         const float4 &li, const CellPos &cp, const uint32_t *__restrict__ list,
                                         int cnt, Pair &&pair) {
  AxisQuad qx, qy, qz;
  if (EDGE) {
    qx = axis_quad(g.w32[0], g.dl32[0], cp.cx == 0, cp.cx == g.nc[0] - 1, li.x, 1.0f);
    qy = axis_quad(g.w32[1], g.dl32[1], cp.cy == 0, cp.cy == g.nc[1] - 1, li.y, 0.25f);
    qz = axis_quad(g.w32[2], g.dl32[2], cp.cz == 0, cp.cz == g.nc[2] - 1, li.z, 0.0625f);
  } else {
    qx.a = g.w32[0];
    qy.a = 0.25f * g.w32[1];
    qz.a = 0.0625f * g.w32[2];
    qx.b = qy.b = qz.b = 0.0f;
    qx.c = -li.x;
    qy.c = -li.y;
    qz.c = -li.z;
  }
  const uint32_t *row = list + i;
  const size_t stride = (size_t)g.stride;
  auto gather = [&](uint32_t e) -> float4 {
    const int j = entry_slot(e);
    if (!MDG_IN_RANGE(d.flags, SITE, j, g.n)) return make_float4(1e30f, 1e30f, 1e30f, 0.f);
    return ld_ro<COH>(loc + j);
  };
  auto offset = [&](uint32_t e, const float4 &lj) {
    const float tx = step_float(e, 0x03u, 8388609.0f);   // t
    const float ty = step_float(e, 0x0Cu, 8388612.0f);   // 4 t
    const float tz = step_float(e, 0x30u, 8388624.0f);   // 16 t
    float dx, dy, dz;
    if (EDGE) {
      dx = lj.x + fmaf(fmaf(qx.b, tx, qx.a), tx, qx.c);
      dy = lj.y + fmaf(fmaf(qy.b, ty, qy.a), ty, qy.c);
      dz = lj.z + fmaf(fmaf(qz.b, tz, qz.a), tz, qz.c);
    } else {
      dx = lj.x + fmaf(qx.a, tx, qx.c);
      dy = lj.y + fmaf(qy.a, ty, qy.c);
      dz = lj.z + fmaf(qz.a, tz, qz.c);
    }
    pair(e, dx, dy, dz, dx * dx + dy * dy + dz * dz);
  };
  int k = 0;
  // the next batch's list entries are requested before this batch's partner
  // positions are used, so the entry load (from DRAM) overlaps the gathers;
  // the last full batch requests the row's remaining (< UNROLL) entries
  const int full = cnt - cnt % UNROLL;
  uint32_t en[UNROLL];
#pragma unroll
  for (int u = 0; u < UNROLL; u++) en[u] = u < cnt ? ld_ro<COH>(row + (size_t)u * stride) : 0u;
#pragma unroll 1
  for (; k < full; k += UNROLL) {
    uint32_t e[UNROLL];
    float4 l[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) e[u] = en[u];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) l[u] = gather(e[u]);
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const int kn = k + UNROLL + u;
      en[u] = kn < cnt ? ld_ro<COH>(row + (size_t)kn * stride) : 0u;
    }
    if (kEntryAhead > 0) {
      // rows kEntryAhead further on, into L2: lane l requests row
      // k + kEntryAhead + (l mod 4) of its own column, so one instruction
      // covers the warp's four next rows, one 128-byte line each
      const int kp = k + kEntryAhead + (int)(threadIdx.x & 3);
      if (kp < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (size_t)kp * stride));
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) offset(e[u], l[u]);
  }
  if (k < cnt) {
    // the remainder as one batch
    constexpr int kTail = UNROLL > 1 ? UNROLL - 1 : 1;
    float4 l[kTail];
#pragma unroll
    for (int u = 0; u < kTail; u++)
      l[u] = k + u < cnt ? gather(en[u]) : make_float4(1e30f, 1e30f, 1e30f, 0.f);
#pragma unroll
    for (int u = 0; u < kTail; u++) offset(en[u], l[u]);
  }
}

// Mixed form of force_fp64: the sum over the row of slot i of f(r) (q_j - q_i)
// in float.  KAHAN: the per-particle sums compensated (MDG_MIXED), else plain
// float (MDG_MIXED_PLAIN).  With PRUNE every entry within the prune radius is
// copied to the inner row of slot i, as in force_fp64.
template <bool PRUNE, bool KAHAN, bool EDGE, bool COH, int UNROLL>
__device__ __forceinline__ double3 pair_loop(const Geom &g, const Dev &d, const float4 *__restrict__ loc, int i,
                                             const float4 &li, const CellPos &cp, const uint32_t *__restrict__ list,
                                             const int *__restrict__ counts, int *kept) {
  int cnt = ld_ro<COH>(counts + i);
  if (!MDG_IN_RANGE(d.flags, kCheckStepRow, cnt, g.list_cap + 1)) cnt = 0;
  const size_t stride = (size_t)g.stride;
  float sx = 0.f, sy = 0.f, sz = 0.f;
  float cx = 0.f, cy = 0.f, cz = 0.f;  // Kahan corrections
  const float rc2 = g.rc2f, c2x8 = g.c2x8f, thr = g.prune_thr2;
  int m = 0;
  walk_row<EDGE, kCheckStepSlot, COH, UNROLL>(g, d, loc, i, li, cp, list, cnt, [&](uint32_t e, float dx, float dy, float dz, float r2) {
    if (PRUNE && r2 <= thr) d.pl[(size_t)(m++) * stride + i] = e;
    // evaluated for every entry and masked: no divergent branch per pair
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(r2));
    const float i6 = inv * inv * inv;
    float df = (i6 * inv) * fmaf(-48.0f, i6, 24.0f) + c2x8;
    df = r2 <= rc2 ? df : 0.0f;
    if (KAHAN) {
      // a zero term (a pair beyond rc) leaves s - c unchanged as a real
      // number (t - s is exact, and so is the new correction), but it moves
      // the correction into s and the later additions round differently:
      // lists that differ only by pairs beyond rc give forces that agree to
      // about one float rounding, not bit for bit
      kahan_fma(sx, cx, df, dx);
      kahan_fma(sy, cy, df, dy);
      kahan_fma(sz, cz, df, dz);
    } else {
      sx = fmaf(df, dx, sx);
      sy = fmaf(df, dy, sy);
      sz = fmaf(df, dz, sz);
    }
  });
  if (PRUNE) *kept = m;
  // the compensated sum rounded once to float (relative 6e-8 of the force),
  // then one conversion per component: GB300 runs double at 1/64 of float
  if (KAHAN) return make_double3((double)(sx - cx), (double)(sy - cy), (double)(sz - cz));
  return make_double3((double)sx, (double)sy, (double)sz);
}

// The pair loop for the calling warp: the linear offset when no active lane's
// home cell touches the periodic boundary (about four warps in five at 66
// cells a side), the quadratic otherwise; both give the same forces bit for
// bit.  Registers are allocated for the larger loop, but the interior one
// needs six fewer and runs without the other's spills.
template <bool PRUNE, bool KAHAN, bool COH = false, int UNROLL = kUnroll>
__device__ __forceinline__ double3 force_mixed(const Geom &g, const Dev &d, const float4 *__restrict__ loc, int i,
                                               const float4 &li, const CellPos &cp, const uint32_t *__restrict__ list,
                                               const int *__restrict__ counts, int *kept) {
  if (__all_sync(__activemask(), !cp.edge)) return pair_loop<PRUNE, KAHAN, false, COH, UNROLL>(g, d, loc, i, li, cp, list, counts, kept);
  return pair_loop<PRUNE, KAHAN, true, COH, UNROLL>(g, d, loc, i, li, cp, list, counts, kept);
}

// The rest of slot i's step after its force F: kick, thermostat, both
// half-drifts, the displacement tests and the stores.  lb: the mixed forms'
// local position at this force evaluation, the FP64 form's at the build; exp1,
// lang: the Nose-Hoover factor and the Langevin stream position; *rebuild and
// *reselect are set when the next step needs a new list or inner list.  Returns
// the kinetic energy (Nose-Hoover).
template <int THERMO, int COMPAT, int MIXED>
__device__ __forceinline__ double step_one(const Geom &g, const Dev &d, int par, int i, bool prune, int kept,
                                           const double3 &F, const float4 &lb, const double4_32a *qm, double4_32a *qn, double exp1,
                                           unsigned long long lang, int *rebuild, int *reselect) {
  // the w words are padding (zero in the FP64 form, packed reference
  // positions in the mixed form): never scaled, never in the kinetic energy
  double4_32a p = d.p[i];
  if (THERMO == MDG_NOSEHOOVER) {
    const double e1 = exp1;
    p.x *= e1; p.y *= e1; p.z *= e1;
    p.x += F.x * g.dt; p.y += F.y * g.dt; p.z += F.z * g.dt;
    p.x *= e1; p.y *= e1; p.z *= e1;
  } else {
    p.x += F.x * g.dt; p.y += F.y * g.dt; p.z += F.z * g.dt;
  }
  if (THERMO == MDG_LANGEVIN) {
    double z[3];
    langevin_normals(g.seed, (uint32_t)d.id[i], lang, z);
    p.x += (-g.gamma * p.x + g.hb_d * z[0]) * g.dt;
    p.y += (-g.gamma * p.y + g.hb_d * z[1]) * g.dt;
    p.z += (-g.gamma * p.z + g.hb_d * z[2]) * g.dt;
  }
  const double4_32a q0 = qm[i];
  double4_32a qe = q0, q1;
  if (MIXED) {  // one rounding per half-drift (fused)
    if (!(THERMO == MDG_LANGEVIN && COMPAT)) {
      qe.x = fma(p.x, g.dt2, q0.x);
      qe.y = fma(p.y, g.dt2, q0.y);
      qe.z = fma(p.z, g.dt2, q0.z);
    }
    q1 = qe;
    q1.x = fma(p.x, g.dt2, qe.x);
    q1.y = fma(p.y, g.dt2, qe.y);
    q1.z = fma(p.z, g.dt2, qe.z);
  } else {  // the reference's separate product and sum
    if (!(THERMO == MDG_LANGEVIN && COMPAT)) {
      qe.x = __dadd_rn(q0.x, __dmul_rn(p.x, g.dt2));
      qe.y = __dadd_rn(q0.y, __dmul_rn(p.y, g.dt2));
      qe.z = __dadd_rn(q0.z, __dmul_rn(p.z, g.dt2));
    }
    q1 = qe;
    q1.x = __dadd_rn(qe.x, __dmul_rn(p.x, g.dt2));
    q1.y = __dadd_rn(qe.y, __dmul_rn(p.y, g.dt2));
    q1.z = __dadd_rn(qe.z, __dmul_rn(p.z, g.dt2));
  }
  float4 ln;
  if (MIXED) {
    // positions relative to the home-cell centre: the new local position is
    // one conversion, and the displacement since the build is measured in
    // float against the build's local position, packed in q_mid.w
    ln = make_float4((float)q1.x, (float)q1.y, (float)q1.z, lb.w);
    float bx, by, bz;
    unpack_ref(g, q0.w, bx, by, bz);
    const float fx = ln.x - bx, fy = ln.y - by, fz = ln.z - bz;
    // the half-margin rule, or a non-finite position (the rebuild's wrap
    // reports it) under either policy
    if ((g.rebuild_policy == MDG_REBUILD_HALFMARGIN && fx * fx + fy * fy + fz * fz > g.half_margin2_ref) ||
        !(fx == fx && fy == fy && fz == fz))
      *rebuild = 1;
  } else {
    const double4_32a qb = d.q_build[i];
    const double ux = q1.x - qb.x, uy = q1.y - qb.y, uz = q1.z - qb.z;
    // displacement since the build: in double for the rebuild test, in
    // float for the new home-cell-local position (qf holds the local
    // position at the build) and the inner-list test
    ln = make_float4(lb.x + (float)ux, lb.y + (float)uy, lb.z + (float)uz, lb.w);
    if ((g.rebuild_policy == MDG_REBUILD_HALFMARGIN && ux * ux + uy * uy + uz * uz > g.half_margin2) ||
        !(q1.x == q1.x && q1.y == q1.y && q1.z == q1.z))
      *rebuild = 1;
  }
  d.loc[par ^ 1][i] = ln;
  // prune reference: the positions of this force evaluation when the
  // inner list was re-selected now, else those of the last selection
  // (mixed: packed in p.w)
  float4 lp;
  if (prune) {
    lp = MIXED ? lb : d.loc[par][i];
    if (MIXED) p.w = pack_ref(g, lp.x, lp.y, lp.z);
    else d.loc_p[i] = lp;
    d.pcount[i] = kept;
  } else if (MIXED) {
    unpack_ref(g, p.w, lp.x, lp.y, lp.z);
  } else {
    lp = d.loc_p[i];
  }
  const float vx = ln.x - lp.x, vy = ln.y - lp.y, vz = ln.z - lp.z;
  if (vx * vx + vy * vy + vz * vz > (MIXED ? g.half_prune2_ref : g.half_prune2)) *reselect = 1;
  d.p[i] = p;
  // the mixed form leaves q_end behind: q_mid - p dt/2 gives it back when a
  // rebuild or a reader needs it (32 bytes a particle fewer per step)
  if (!MIXED) d.q_end[i] = qe;
  qn[i] = q1;
  return THERMO == MDG_NOSEHOOVER ? 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z : 0.0;
}

}  // namespace mdg

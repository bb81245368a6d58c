// One MD step as one kernel, plus the observers and the state exchange.
//
// k_step replaces, for one step of MDManager::Calculate (mdmanager.cc:116-148):
//   ForceCalculator::CalculateForce (fcalculator.cc:35-50, 229-290): the LJ
//     pair force of the smoothly truncated potential, applied as p += F dt;
//   the thermostat of MDManager::CalculateLangevin / CalculateNoseHoover
//     (mdmanager.cc:160-192, fcalculator.cc:743-778);
//   the second half-drift ForceCalculator::UpdatePositionHalf (fcalculator.cc:21-32)
//     and the first half-drift of the following step;
//   the expiry test of PairList::IsPairListExpired (pairlist.cc:26-45), here the
//     displacement criterion: moved more than margin/2 since the build.
// It is a gather over the full neighbour list: one thread per particle, no
// atomics, no reaction scatter (the "Reactless" form, fcalculator.cc:504-542).
//
// FP64 form: the pair force is evaluated in double precision.  1/r^2 comes
// from the hardware reciprocal estimate (rcp.approx.ftz.f64) refined by one
// Householder step of order three, y <- y (1 + e + e^2), e = 1 - r^2 y, which
// cubes the relative error of the estimate.
// Mixed form (MDG_MIXED): particle positions relative to their home-cell
// centre in float; the pair force in float; the per-particle force sum in
// compensated float (Kahan: each term's lost low part carried in a second
// float, four float operations per component and pair), so the sum's error
// does not grow with the number of partners; converted to double once per
// particle; momentum and position updates in double with fused multiply-adds,
// the mid-step positions kept relative to the centre of the home cell (so the
// float position partners gather is one conversion and the displacement since
// the build is tested in float against the build's local position, which
// travels packed in q_mid's padding word, as the prune reference does in p's)
// and the step-boundary positions not written (the readers rebuild them from
// q_mid and p).  MDG_MIXED_PLAIN sums the pair forces in plain float instead (an
// error near u sqrt(40) |f_ij|, u = 2^-24, over about 40 terms).  GB300 runs
// double precision at 1/64 of the float rate, so the per-particle double work
// (momentum, two half-drifts) is kept to one operation per component each,
// and the per-pair work stays in float.
#include "mdg_internal.cuh"
#include "mdg_step.cuh"

namespace mdg {

namespace {

constexpr int kStepThreads = 128;  // observers, forces, state exchange
// Threads per block of the mixed-form step kernel: 128 for the ordinary
// variant, 384 for the re-selecting one, which walks the outer rows and
// writes the inner rows of consecutive slots (4M atoms, mean step kernel of
// a 20-step window 5 steps after a fresh list / of 400 steps with their
// rebuilds and re-selections, in ms: ordinary/re-selecting 128/128 0.4314 /
// 0.4473; 128/128 at 80 registers for the re-selecting variant 0.4278 /
// 0.4445; 384/384 0.4202 / 0.4322; 256/384 0.4150 / 0.4275; 128/512 0.4132 /
// 0.4261; 128/384 0.4119 / 0.4238).  The FP64 form (FP64-pipe bound) keeps
// 128 for both: 5.795 against 5.831 ms at 384.
#ifndef MDG_STEP_THREADS_MIXED
#define MDG_STEP_THREADS_MIXED 128
#endif
#ifndef MDG_PRUNE_THREADS_MIXED
#define MDG_PRUNE_THREADS_MIXED 384
#endif
// (Nose-Hoover: one size for both variants, whose block sums k_nh_update adds)
template <int THERMO, int MIXED, int PMODE>
__host__ __device__ constexpr int step_threads() {
  return !MIXED ? kStepThreads
                : (PMODE == 1 || THERMO == MDG_NOSEHOOVER ? MDG_STEP_THREADS_MIXED : MDG_PRUNE_THREADS_MIXED);
}
// Resident blocks per SM requested for the ordinary step variant (the
// register budget follows: 65536 / (blocks * 128) per thread).  The kernel
// waits on gathers, so occupancy pays: 12 blocks (40 registers, 48 warps per
// SM) ran 16 % faster than the unconstrained 61-register build at 4M atoms.
#ifndef MDG_STEP_MIN_BLOCKS
#define MDG_STEP_MIN_BLOCKS 12
#endif
// The same for the compensated mixed form.  Its three correction terms fit
// in 40 registers since the build reference is no longer held across the
// pair loop (it travels packed in q_mid.w); before, 12 blocks with a 48-byte
// spill still measured 6 % faster than 10 blocks at 48 registers without it
// (4M atoms, 400 steps: 0.472 against 0.501 ms per step kernel).
#ifndef MDG_STEP_MIN_BLOCKS_KAHAN
#define MDG_STEP_MIN_BLOCKS_KAHAN 12
#endif
#ifndef MDG_PRUNE_MIN_BLOCKS
#define MDG_PRUNE_MIN_BLOCKS 8
#endif
// PMODE: 0 = decide from flags->prune_now in the kernel (both paths compiled);
// 1 = ordinary step only, 2 = re-selecting step only (each a no-op when the
// flag says otherwise, so the graph path can run the lighter variant).
template <int THERMO, int COMPAT, int MIXED, int PMODE>
// The resident-block counts of the launch bounds are for 128-thread blocks.
__global__ void __launch_bounds__(step_threads<THERMO, MIXED, PMODE>(), (PMODE != 1          ? MDG_PRUNE_MIN_BLOCKS
                                                         : MIXED == MDG_MIXED ? MDG_STEP_MIN_BLOCKS_KAHAN
                                                                              : MDG_STEP_MIN_BLOCKS) *
                                                            128 / step_threads<THERMO, MIXED, PMODE>())
    k_step(Geom g, Dev d, int par) {
  const DevFlags *f = d.flags;
  if (f->halt != 0) return;
  if (PMODE == 1 && f->prune_now != 0) return;
  if (PMODE == 2 && f->prune_now == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < g.n;
  const double4_32a *qm = d.q_mid[par];
  double4_32a *qn = d.q_mid[par ^ 1];
  double ke = 0.0;
  // inner-list re-selection: the same for the whole grid this step
  const bool prune = PMODE == 2 ? true : (PMODE == 1 ? false : f->prune_now != 0);
  int kept = 0;
  if (active) {
    // mixed: this force evaluation's local position (partners gather the
    // same array); FP64: the build-time local position.  The w word of
    // either holds the home-cell coordinates
    const float4 lb = MIXED ? d.loc[par][i] : d.qf[i];
    const CellPos cp = cell_pos_packed(g, lb.w);
    double3 F;
    if (prune)
      F = MIXED ? force_mixed<true, MIXED == MDG_MIXED>(g, d, d.loc[par], i, lb, cp, d.nl, d.ncount, &kept)
                : force_fp64<true, false>(g, d, qm, i, cp, d.nl, d.ncount, &kept);
    else
      F = MIXED ? force_mixed<false, MIXED == MDG_MIXED>(g, d, d.loc[par], i, lb, cp, d.pl, d.pcount, nullptr)
                : force_fp64<false, false>(g, d, qm, i, cp, d.pl, d.pcount, nullptr);
    ke = step_one<THERMO, COMPAT, MIXED>(g, d, par, i, prune, kept, F, lb, qm, qn, THERMO == MDG_NOSEHOOVER ? f->exp1 : 1.0,
                                         THERMO == MDG_LANGEVIN ? f->lang - 1ull : 0ull, &d.flags->rebuild,
                                         &d.flags->prune_next);
  }
  if (MIXED && i == 0) d.flags->end_stale = 1;
  if (THERMO == MDG_NOSEHOOVER) {
    __shared__ double sh[step_threads<THERMO, MIXED, PMODE>() / 32];
    const double t = block_sum(ke, sh);
    if (threadIdx.x == 0) d.partials[blockIdx.x] = t;
  }
  if (prune) {  // inner-list size for the statistics (uniform branch)
    unsigned long long v = (unsigned long long)kept;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&d.flags->inner_pairs, v);
  }
}

// Nose-Hoover bookkeeping after a step (mdmanager.cc:169-174) and before the
// next (mdmanager.cc:161-164): T from the block sums in fixed order.
__global__ void k_nh_update(Geom g, Dev d, int nparts, int first) {
  DevFlags *f = d.flags;
  if (f->halt != 0) return;
  __shared__ double sh[32];
  double v = 0.0;
  for (int b = threadIdx.x; b < nparts; b += blockDim.x) v += d.partials[b];
  const double ke = block_sum(v, sh);
  if (threadIdx.x == 0) {
    const double T = ke / (double)g.n / 1.5;
    const double dt2 = g.dt * 0.5;
    const double t1 = (T - g.temperature) / (g.tau * g.tau);
    const double zeta = first ? f->zeta : f->zeta_a + t1 * dt2;
    f->zeta = zeta;
    f->t_cur = T;
    f->zeta_a = zeta + t1 * dt2;
    f->exp1 = exp(-dt2 * f->zeta_a);
  }
}

__global__ void __launch_bounds__(kStepThreads) k_kinetic(Geom g, Dev d) {
  __shared__ double sh[kStepThreads / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ke = 0.0;
  if (i < g.n) {
    const double4_32a p = d.p[i];
    ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
  }
  const double t = block_sum(ke, sh);
  if (threadIdx.x == 0) d.partials[blockIdx.x] = t;
}

// Observers at the step-boundary positions q_end: kinetic energy
// (observer.cc:5-15), pair energy (observer.cc:17-48) and virial
// (observer.cc:50-79), each pair evaluated with the reference's expression
// and rounding and weighted 1/2 (each pair is listed from both sides).  The FP64
// form outside the fixed-point range (k_observe_fixed is the others').
__global__ void __launch_bounds__(kStepThreads) k_observe(Geom g, Dev d) {
  __shared__ double sh[kStepThreads / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ke = 0.0, pe = 0.0, vir = 0.0;
  if (i < g.n) {
    const double4_32a p = d.p[i];
    ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
    observe_row_fp64(g, d, i, cell_pos(g, d.cell[i]), d.ncount[i], pe, vir);
  }
  const double a = block_sum(ke, sh);
  const double b = block_sum(pe, sh);
  const double c = block_sum(vir, sh);
  if (threadIdx.x == 0) {
    d.partials[3 * blockIdx.x + 0] = a;
    d.partials[3 * blockIdx.x + 1] = b;
    d.partials[3 * blockIdx.x + 2] = c;
  }
}

// Mixed-form observers: the same sums with each pair's energy and virial
// term evaluated in float (from the home-cell-local float positions of q_end,
// as the mixed force) and summed over the row in compensated float, walked
// like the step kernel's row; the rows are added in double.
template <bool EDGE>
__device__ __forceinline__ void observe_row(const Geom &g, const Dev &d, const float4 *__restrict__ loc, int i,
                                            const float4 &li, const CellPos &cp, int cnt, double &pe, double &vir) {
  const float rc2 = g.rc2f, c2 = (float)g.c2, c0 = (float)g.c0, c2x8 = g.c2x8f;
  // compensated sums: the error of each row sum stays near one float
  // rounding of the sum, whatever the row length (GB300 runs double, and
  // conversions to 64-bit types, at 1/64 of the float rate)
  float se = 0.f, ce = 0.f, sv = 0.f, cv = 0.f;
  walk_row<EDGE, kCheckObserve, false, kUnroll>(g, d, loc, i, li, cp, d.nl, cnt,
                                [&](uint32_t, float, float, float, float r2) {
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(r2));
    const float i6 = inv * inv * inv;
    float e_ij = 4.0f * (i6 * i6 - i6 + fmaf(c2, r2, c0));
    float v_ij = ((i6 * inv) * fmaf(-48.0f, i6, 24.0f) + c2x8) * r2;
    // masked, not branched; a padding partner's inf / NaN terms drop here
    e_ij = r2 <= rc2 ? e_ij : 0.0f;
    v_ij = r2 <= rc2 ? v_ij : 0.0f;
    kahan_fma(se, ce, e_ij, 1.0f);
    kahan_fma(sv, cv, v_ij, 1.0f);
  });
  pe = 0.5 * (double)(se - ce);
  vir = 0.5 * (double)(sv - cv);
}

__global__ void __launch_bounds__(kStepThreads) k_observe_mixed(Geom g, Dev d, const float4 *__restrict__ loc) {
  __shared__ double sh[kStepThreads / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ke = 0.0, pe = 0.0, vir = 0.0;
  if (i < g.n) {
    const double4_32a p = d.p[i];
    ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
    const float4 li = loc[i];
    const CellPos cp = cell_pos_packed(g, li.w);
    int cnt = d.ncount[i];
    if (!MDG_IN_RANGE(d.flags, kCheckObserve, cnt, g.list_cap + 1)) cnt = 0;
    // the linear offset for warps with no lane at the periodic boundary
    if (__all_sync(__activemask(), !cp.edge)) observe_row<false>(g, d, loc, i, li, cp, cnt, pe, vir);
    else observe_row<true>(g, d, loc, i, li, cp, cnt, pe, vir);
  }
  const double a = block_sum(ke, sh);
  const double b = block_sum(pe, sh);
  const double c = block_sum(vir, sh);
  if (threadIdx.x == 0) {
    d.partials[3 * blockIdx.x + 0] = a;
    d.partials[3 * blockIdx.x + 1] = b;
    d.partials[3 * blockIdx.x + 2] = c;
  }
}

__global__ void k_observe_final(Dev d, int nparts, double *out) {
  __shared__ double sh[32];
  double a = 0.0, b = 0.0, c = 0.0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
    a += d.partials[3 * k + 0];
    b += d.partials[3 * k + 1];
    c += d.partials[3 * k + 2];
  }
  const double ta = block_sum(a, sh), tb = block_sum(b, sh), tc = block_sum(c, sh);
  if (threadIdx.x == 0) {
    out[0] = ta;
    out[1] = tb;
    out[2] = tc / 3.0;
  }
}

// Forces at q_end in the handle's precision, written in caller order to io4.
template <int MIXED>
__global__ void __launch_bounds__(kStepThreads) k_forces(Geom g, Dev d, const float4 *loc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const CellPos cp = cell_pos(g, d.cell[i]);
  const double3 F = MIXED ? force_mixed<false, MIXED == MDG_MIXED>(g, d, loc, i, loc[i], cp, d.nl, d.ncount, nullptr)
                          : force_fp64<false, false>(g, d, d.q_end, i, cp, d.nl, d.ncount, nullptr);
  d.io4[d.id[i]] = make_double4_32a(F.x, F.y, F.z, 0.0);
}

// Float positions of q_end relative to the home-cell centres (k_forces<1> input).
// In the mixed form q_mid[par] is already home-cell-local: the step-boundary
// local position is q_mid - p dt/2, with no box coordinates in between.
__global__ void k_loc_from_end(Geom g, Dev d, float4 *loc, int par) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  int cx, cy, cz;
  cell_unkey(d.cell[i], cx, cy, cz);
  if (g.local_pos) {
    const double4_32a u = d.q_mid[par][i], p = d.p[i];
    loc[i] = make_float4((float)fma(-p.x, g.dt2, u.x), (float)fma(-p.y, g.dt2, u.y), (float)fma(-p.z, g.dt2, u.z),
                         cell_pack(cx, cy, cz));
    return;
  }
  const double4_32a q = d.q_end[i];
  loc[i] = make_float4((float)(q.x - cell_centre(g, 0, cx)), (float)(q.y - cell_centre(g, 1, cy)),
                       (float)(q.z - cell_centre(g, 2, cz)), cell_pack(cx, cy, cz));
}

// The caller's arrays in the caller's order; their fourth lane is padding
// and comes back zero (the mixed form keeps packed reference positions in it).
__global__ void k_unsort(Geom g, Dev d, double4_32a *qo, double4_32a *po) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const int id = d.id[i];
  if (qo) {
    double4_32a q = d.q_end[i];
    q.w = 0.0;
    qo[id] = q;
  }
  if (po) {
    double4_32a p = d.p[i];
    p.w = 0.0;
    po[id] = p;
  }
}

__global__ void k_sort_in(Geom g, Dev d, const double4_32a *qi, const double4_32a *pi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  double4_32a q = qi[i], p = pi[i];
  q.w = 0.0;
  p.w = 0.0;
  d.q_end[i] = q;
  d.p[i] = p;
  d.id[i] = i;
  d.inv[i] = i;
}

__global__ void k_pairs(Geom g, Dev d, const long long *row_off, int32_t *rec) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const CellPos cp = cell_pos(g, d.cell[i]);
  const int cnt = d.ncount[i];
  long long o = row_off[i];
  for (int k = 0; k < cnt; k++) {
    const uint32_t e = d.nl[(size_t)k * g.stride + i];
    const int j = (int)entry_slot(e);
    const int ox = entry_sx(e), oy = entry_sy(e), oz = entry_sz(e);
    const int sx = (ox == 0 && cp.cx == 0) ? -1 : ((ox == 2 && cp.cx == g.nc[0] - 1) ? 1 : 0);
    const int sy = (oy == 0 && cp.cy == 0) ? -1 : ((oy == 2 && cp.cy == g.nc[1] - 1) ? 1 : 0);
    const int sz = (oz == 0 && cp.cz == 0) ? -1 : ((oz == 2 && cp.cz == g.nc[2] - 1) ? 1 : 0);
    rec[3 * (o + k) + 0] = d.id[i];
    rec[3 * (o + k) + 1] = d.id[j];
    rec[3 * (o + k) + 2] = (sx + 1) + 3 * (sy + 1) + 9 * (sz + 1);
  }
}

inline int blocks_for(int n) { return n > 0 ? (n + kStepThreads - 1) / kStepThreads : 1; }

}  // namespace

template <int T, int C, int M>
void launch_step_variant(const Geom &g, const Dev &d, int par, int pmode, cudaStream_t s) {
  constexpr int t0 = step_threads<T, M, 0>(), t1 = step_threads<T, M, 1>(), t2 = step_threads<T, M, 2>();
  auto grid = [&](int threads) { return g.n > 0 ? (g.n + threads - 1) / threads : 1; };
  if (pmode == 0) k_step<T, C, M, 0><<<grid(t0), t0, 0, s>>>(g, d, par);
  if (pmode == 1 || pmode == 3) k_step<T, C, M, 1><<<grid(t1), t1, 0, s>>>(g, d, par);
  if (pmode == 2 || pmode == 3) k_step<T, C, M, 2><<<grid(t2), t2, 0, s>>>(g, d, par);
  // the Nose-Hoover block sums of this step: one per block of the variant that ran
  static_assert(T != MDG_NOSEHOOVER || (t0 == t1 && t1 == t2), "one partial-sum count for every variant");
  if (T == MDG_NOSEHOOVER) k_nh_update<<<1, 1024, 0, s>>>(g, d, grid(t1), 0);
}

template <int T, int C>
void launch_step_precision(const Geom &g, const Dev &d, int par, int precision, int pmode, cudaStream_t s) {
  if (precision == MDG_MIXED) launch_step_variant<T, C, MDG_MIXED>(g, d, par, pmode, s);
  else if (precision == MDG_MIXED_PLAIN) launch_step_variant<T, C, MDG_MIXED_PLAIN>(g, d, par, pmode, s);
  else launch_step_variant<T, C, MDG_FP64>(g, d, par, pmode, s);
}

// pmode: 0 one kernel deciding on the device; 1 / 2 only the ordinary / the
// re-selecting variant (graph conditional bodies); 3 both variants in turn.
// mixed: the handle's mdg_precision.
void launch_step(const Geom &g, const Dev &d, int par, int thermostat, int compat, int mixed, cudaStream_t s,
                 int pmode) {
  if (g.fixed) {
    const int grid = launch_step_fixed(g, d, par, thermostat, compat, pmode, s);
    if (thermostat == MDG_NOSEHOOVER) k_nh_update<<<1, 1024, 0, s>>>(g, d, grid, 0);
    return;
  }
  if (thermostat == MDG_LANGEVIN) {
    if (compat) launch_step_precision<MDG_LANGEVIN, 1>(g, d, par, mixed, pmode, s);
    else launch_step_precision<MDG_LANGEVIN, 0>(g, d, par, mixed, pmode, s);
  } else if (thermostat == MDG_NOSEHOOVER) {
    launch_step_precision<MDG_NOSEHOOVER, 0>(g, d, par, mixed, pmode, s);
  } else {
    launch_step_precision<MDG_NVE, 0>(g, d, par, mixed, pmode, s);
  }
}

void launch_nh_init(const Geom &g, const Dev &d, cudaStream_t s) {
  const int grid = blocks_for(g.n);
  k_kinetic<<<grid, kStepThreads, 0, s>>>(g, d);
  k_nh_update<<<1, 1024, 0, s>>>(g, d, grid, 1);
}

void launch_observe(const Geom &g, const Dev &d, double *out_dev, cudaStream_t s, int mixed, int par, int call) {
  int grid = blocks_for(g.n);
  if (g.fixed) {
    grid = launch_observe_fixed(g, d, par, call, s);
  } else if (mixed) {
    // the buffer the next step overwrites before reading it
    k_loc_from_end<<<grid, kStepThreads, 0, s>>>(g, d, d.loc[par ^ 1], par);
    k_observe_mixed<<<grid, kStepThreads, 0, s>>>(g, d, d.loc[par ^ 1]);
  } else {
    k_observe<<<grid, kStepThreads, 0, s>>>(g, d);
  }
  k_observe_final<<<1, 1024, 0, s>>>(d, grid, out_dev);
}

void launch_forces(const Geom &g, const Dev &d, int mixed, int par, int call, cudaStream_t s) {
  const int grid = blocks_for(g.n);
  if (g.fixed) {
    launch_forces_fixed(g, d, par, call, s);
  } else if (mixed) {
    // the buffer the next step overwrites before reading it
    k_loc_from_end<<<grid, kStepThreads, 0, s>>>(g, d, d.loc[par ^ 1], par);
    if (mixed == MDG_MIXED_PLAIN) k_forces<MDG_MIXED_PLAIN><<<grid, kStepThreads, 0, s>>>(g, d, d.loc[par ^ 1]);
    else k_forces<MDG_MIXED><<<grid, kStepThreads, 0, s>>>(g, d, d.loc[par ^ 1]);
  } else {
    k_forces<0><<<grid, kStepThreads, 0, s>>>(g, d, nullptr);
  }
}

void launch_unsort(const Geom &g, const Dev &d, int par, double4_32a *qo, double4_32a *po, cudaStream_t s) {
  if (g.local_pos) launch_end_from_mid(g, d, par, s);
  k_unsort<<<blocks_for(g.n), kStepThreads, 0, s>>>(g, d, qo, po);
}

void launch_sort_in(const Geom &g, const Dev &d, const double4_32a *qi, const double4_32a *pi, cudaStream_t s) {
  k_sort_in<<<blocks_for(g.n), kStepThreads, 0, s>>>(g, d, qi, pi);
}

void launch_pairs(const Geom &g, const Dev &d, const long long *row_off, int32_t *rec, cudaStream_t s) {
  k_pairs<<<blocks_for(g.n), kStepThreads, 0, s>>>(g, d, row_off, rec);
}

}  // namespace mdg

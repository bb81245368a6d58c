// The FP64 form's step, observers and forces with the pair arithmetic in
// 64-bit fixed point (mdg_fixed.cuh): the same step as k_step (mdg_step.cu),
// the same state and integration in double, rounding for rounding; only the
// pair separation, distance and force run on the integer units.
//
// Used when Geom::fixed is set: search length + margin below 4 sigma (the
// positions are kept modulo 8 sigma) and a cut-off of at least one sigma;
// anything else keeps the double pair loop of k_step.  So does a step whose
// positions are not safe modulo 8 (flags->fx_wide: a particle further from
// its place at the build than Geom::fx_guard allows for two of them), and a
// row whose force sums might leave their range (fix_sum_fits); a pair closer
// than r^2 = kFixNear takes the double expression by itself.
//
// Extra state: xq[2] the fixed-point positions of q_mid[2] (what partners
// gather, 32 bytes, the w word holds the home cell), xb the high words at the
// last build and xp at the last inner-list selection (displacement tests).
#include "mdg_fixed_step.cuh"

namespace mdg {

namespace {

// Threads per block: one thread per particle, or kWide threads whose LANES
// neighbours share a particle's row.
constexpr int kOne = 128, kWide = 256;
// Blocks per SM asked for with one thread per particle (80 registers; the
// integer multiply-adds keep their pipe about 80 % busy): 4M atoms, step kernel
// 1.073 ms with 6 blocks, 1.115 with 5.
constexpr int kOneBlocks = 6;
template <int LANES>
__host__ __device__ constexpr int fx_threads() { return LANES == 1 ? kOne : kWide; }
template <int LANES>
__host__ __device__ constexpr int fx_particles() { return fx_threads<LANES>() / LANES; }

// The step of k_step (mdg_step.cu) on the fixed-point positions; PMODE as there.
template <int THERMO, int COMPAT, int PMODE, int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>(), LANES == 1 ? kOneBlocks : 2) k_step_fixed(Geom g, Dev d, int par) {
  constexpr int kThreads = fx_threads<LANES>(), kParticles = fx_particles<LANES>();
  const DevFlags *f = d.flags;
  if (f->halt != 0) return;
  if (PMODE == 1 && f->prune_now != 0) return;
  if (PMODE == 2 && f->prune_now == 0) return;
  const bool prune = PMODE == 2 ? true : (PMODE == 1 ? false : f->prune_now != 0);
  const bool wide = f->fx_wide[par] != 0;
  const double4_32a *qm = d.q_mid[par];
  const FixPos *xq = d.xq[par];
  const int first = blockIdx.x * kParticles;
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  int i = first + threadIdx.x / LANES;
  bool active = i < g.n;
  int kept = 0;
  double3 F = make_double3(0.0, 0.0, 0.0);
  {
    const int ia = active ? i : g.n - 1;
    const FixPos own = xq[ia];
    if (prune) F = force_fixed<true, LANES, false>(g, d, xq, qm, own, ia, wide, d.nl, d.ncount, active, lane, kept);
    else F = force_fixed<false, LANES, false>(g, d, xq, qm, own, ia, wide, d.pl, d.pcount, active, lane, kept);
  }
  if (LANES > 1) {
    // the block's particles move on to its first threads, one each
    __shared__ double3 sF[kParticles];
    __shared__ int sk[kParticles];
    if (lane == 0) {
      sF[threadIdx.x / LANES] = F;
      sk[threadIdx.x / LANES] = kept;
    }
    __syncthreads();
    i = first + threadIdx.x;
    active = threadIdx.x < kParticles && i < g.n;
    kept = 0;
    if (active) {
      F = sF[threadIdx.x];
      kept = sk[threadIdx.x];
    }
  }
  double ke = 0.0;
  if (active) {
    ke = step_one_fixed<THERMO, COMPAT>(g, d, par, i, prune, kept, F, THERMO == MDG_NOSEHOOVER ? f->exp1 : 1.0,
                                        THERMO == MDG_LANGEVIN ? f->lang - 1ull : 0ull, &d.flags->rebuild, &d.flags->prune_next);
  }
  if (THERMO == MDG_NOSEHOOVER) {
    __shared__ double sh[kThreads / 32];
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

// Fixed-point positions of q_end into xq[dst] (the buffer the next step
// overwrites before reading it); a particle too far from its place at the
// build marks fx_wide_end with this call's number.
__global__ void k_fix_end(Geom g, Dev d, int dst, int call) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const int4 xb = d.xb[i];
  const double4_32a q = d.q_end[i];
  const FixPos x = fix_position(q.x, q.y, q.z, xb.w);
  const float u = 1.0f / (float)(1 << (kFixPosBits - 32));
  const float bx = (float)(x.x - xb.x) * u, by = (float)(x.y - xb.y) * u, bz = (float)(x.z - xb.z) * u;
  if (fast(g, d.p[i]) || fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz))) > g.fx_guard) d.flags->fx_wide_end = call;
  d.xq[dst][i] = x;
}

template <int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>()) k_forces_fixed(Geom g, Dev d, int src, int call) {
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  const int i = blockIdx.x * fx_particles<LANES>() + threadIdx.x / LANES;
  const bool active = i < g.n;
  const int ia = active ? i : g.n - 1;
  int kept = 0;
  const double3 F = force_fixed<false, LANES, false>(g, d, d.xq[src], d.q_end, d.xq[src][ia], ia, d.flags->fx_wide_end == call,
                                              d.nl, d.ncount, active, lane, kept);
  const double s = 1.0 / (double)(1ull << kFixSumBits);
  if (active && lane == 0) d.io4[d.id[i]] = make_double4_32a(F.x * s, F.y * s, F.z * s, 0.0);
}

// Longest row whose sums of z^2 (2.83 at most each, units of 2^-54) fit.
constexpr int kFixObserveRow = 361;

// Observers (observer.cc:5-79) at q_end: a row's pair energies are
// 4 (sum z^2 - sum z + C2 sum r^2 + C0 count) and its virial terms
// 24 sum z - 48 sum z^2 + 8 C2 sum r^2 with z = r^-6, summed as integers (the
// cut bits' mean, half a unit, added back); each pair is listed from both sides
// and weighted 1/2.
template <bool EDGE, int LANES>
__device__ __forceinline__ void observe_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                              const FixPos &own, int i, const CellPos &cp, int cnt, int lane,
                                              uint64_t &sz, uint64_t &szz, uint64_t &sr, int &m, double &ne, double &nv) {
  const uint64_t rc2 = g.fx_rc2;
  const uint32_t near = g.fx_near;
  walk_fixed<EDGE, LANES, false, kCheckObserve, false>(
      g, d, xq, own, i, cp, d.nl, cnt, lane, [&](bool, uint32_t, const FixSep &, uint64_t R) {
        const bool in = R <= rc2, close = in && fix_hi(R) < near, take = in && !close;
        uint64_t y2, z;
        fix_powers(fix_recip(R), y2, z);
        const uint64_t zz = fix_sqrhi(z);  // 2^-58
        sz += take ? z >> 7 : 0;
        szz += take ? zz >> 4 : 0;
        sr += take ? R >> 7 : 0;  // 2^-51
        m += take ? 1 : 0;
        return close;
      },
      [&](uint32_t e) {
        {
          double4_32a qj = d.q_end[entry_slot(e)];
          const double4_32a qi = d.q_end[i];
          apply_image(g, cp, e, qj);
          const double dx = __dsub_rn(qi.x, qj.x), dy = __dsub_rn(qi.y, qj.y), dz = __dsub_rn(qi.z, qj.z);
          const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
          pair_observables(g, r2, ne, nv);
        }
      });
}

template <int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>()) k_observe_fixed(Geom g, Dev d, int src, int call) {
  __shared__ double sh[fx_threads<LANES>() / 32];
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  const int i = blockIdx.x * fx_particles<LANES>() + threadIdx.x / LANES;
  const bool active = i < g.n;
  double ke = 0.0, pe = 0.0, vir = 0.0;
  const int ia = active ? i : g.n - 1;
  const FixPos own = d.xq[src][ia];
  const CellPos cp = cell_pos(g, (int)own.w);
  int cnt = active ? d.ncount[ia] : 0;
  if (!MDG_IN_RANGE(d.flags, kCheckObserve, cnt, g.list_cap + 1)) cnt = 0;
  if (active && lane == 0) {
    const double4_32a p = d.p[ia];
    ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
  }
  if (d.flags->fx_wide_end == call || cnt > kFixObserveRow) {
    if (active && lane == 0) observe_row_fp64(g, d, ia, cp, cnt, pe, vir);
  } else {
    uint64_t sz = 0, szz = 0, sr = 0;
    int m = 0;
    double ne = 0.0, nv = 0.0;
    if (__all_sync(__activemask(), !cp.edge)) observe_fixed<false, LANES>(g, d, d.xq[src], own, ia, cp, cnt, lane, sz, szz, sr, m, ne, nv);
    else observe_fixed<true, LANES>(g, d, d.xq[src], own, ia, cp, cnt, lane, sz, szz, sr, m, ne, nv);
    const double u = 1.0 / (double)(1ull << 54), half = 0.5 * m;
    const double z = ((double)sz + half) * u, zz = ((double)szz + half) * u;
    const double r = g.c2 * (((double)sr + half) * (1.0 / (double)(1ull << 51)));
    pe = ne + 2.0 * ((zz - z) + (r + g.c0 * (double)m));
    vir = nv + 12.0 * (z - 2.0 * zz) + 4.0 * r;
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

template <int LANES>
int fx_grid(int n) { return n > 0 ? (n + fx_particles<LANES>() - 1) / fx_particles<LANES>() : 1; }

template <int T, int C, int LANES>
int launch_lanes(const Geom &g, const Dev &d, int par, int pmode, cudaStream_t s) {
  constexpr int t = fx_threads<LANES>();
  const int grid = fx_grid<LANES>(g.n);
  if (pmode == 0) k_step_fixed<T, C, 0, LANES><<<grid, t, 0, s>>>(g, d, par);
  if (pmode == 1 || pmode == 3) k_step_fixed<T, C, 1, LANES><<<grid, t, 0, s>>>(g, d, par);
  if (pmode == 2 || pmode == 3) k_step_fixed<T, C, 2, LANES><<<grid, t, 0, s>>>(g, d, par);
  return grid;
}

template <int T, int C>
int launch_thermo(const Geom &g, const Dev &d, int par, int pmode, cudaStream_t s) {
  const int lanes = fx_lanes(g.n);
  return lanes == 32  ? launch_lanes<T, C, 32>(g, d, par, pmode, s)
         : lanes == 8 ? launch_lanes<T, C, 8>(g, d, par, pmode, s)
         : lanes == 2 ? launch_lanes<T, C, 2>(g, d, par, pmode, s)
                      : launch_lanes<T, C, 1>(g, d, par, pmode, s);
}

}  // namespace

int launch_step_fixed(const Geom &g, const Dev &d, int par, int thermostat, int compat, int pmode, cudaStream_t s) {
  if (thermostat == MDG_LANGEVIN)
    return compat ? launch_thermo<MDG_LANGEVIN, 1>(g, d, par, pmode, s) : launch_thermo<MDG_LANGEVIN, 0>(g, d, par, pmode, s);
  if (thermostat == MDG_NOSEHOOVER) return launch_thermo<MDG_NOSEHOOVER, 0>(g, d, par, pmode, s);
  return launch_thermo<MDG_NVE, 0>(g, d, par, pmode, s);
}

void launch_forces_fixed(const Geom &g, const Dev &d, int par, int call, cudaStream_t s) {
  const int dst = par ^ 1, lanes = fx_lanes(g.n);
  k_fix_end<<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  if (lanes == 32) k_forces_fixed<32><<<fx_grid<32>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 8) k_forces_fixed<8><<<fx_grid<8>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 2) k_forces_fixed<2><<<fx_grid<2>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else k_forces_fixed<1><<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
}

int launch_observe_fixed(const Geom &g, const Dev &d, int par, int call, cudaStream_t s) {
  const int dst = par ^ 1, lanes = fx_lanes(g.n);
  k_fix_end<<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  if (lanes == 32) k_observe_fixed<32><<<fx_grid<32>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 8) k_observe_fixed<8><<<fx_grid<8>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 2) k_observe_fixed<2><<<fx_grid<2>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else k_observe_fixed<1><<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  return lanes == 32 ? fx_grid<32>(g.n) : lanes == 8 ? fx_grid<8>(g.n) : lanes == 2 ? fx_grid<2>(g.n) : fx_grid<1>(g.n);
}

}  // namespace mdg

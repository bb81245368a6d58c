// The steps of a small box in one resident kernel.
//
// A step graph costs a small box more than its steps: the prelude kernel, the
// conditional node and the launch of its body take 11-13 us a step (864
// atoms FP64: 24 us per single-step call, of which 11 are the step kernel;
// 108,000 atoms mixed: 50 us for a 30 us kernel), and a rebuild is ten
// launches.  Here one cooperative launch runs all steps of an mdg_calculate
// call: one block per SM, each with its share of the slots, a grid barrier
// after every step, and the rebuild as phases between further barriers.  The
// particles' arithmetic is the step kernels' own (step_one, force_mixed,
// step_one_fixed, force_fixed; finalize_one, build_slot_row and build_cell_rows
// for the list).
//
// All blocks are resident at once (the cooperative launch fails otherwise),
// so every barrier is reached; its wait is bounded all the same, and a block
// that gives up halts the run (kHaltBarrier).  Data that the kernel itself
// writes are read with ordinary loads, which the barrier's fence makes
// current, never through the read-only path.
//
// Requests for the next step (a new list, a new inner list) go to a slot of
// their own per step, three in turn: set during step s - 1, read by every block
// after its barrier, cleared by block 0 during step s + 1, when every block is
// past the barrier that follows its read.
#include "mdg_fixed_step.cuh"
#include "mdg_rebuild.cuh"

namespace mdg {

struct ResidentCtl {
  unsigned arrived;   // blocks past their barriers, all barriers of a launch together
  unsigned left;      // blocks that are done with the launch
  int failed;         // a block gave up waiting
  int rebuild[3], reselect[3];
  unsigned long long inner[3];
};

namespace {

constexpr int kFixedForm = 3;  // template value beside MDG_MIXED and MDG_MIXED_PLAIN

// Threads of a block: 512 (128 registers), or for the mixed forms
// of boxes with more particles than 512 per SM 1024 (64), and beside other handles'
// launches 256 (narrow_block).  With 512 or fewer the mixed
// row walk has kFewUnroll gathers in flight (864 / 16,384 / 70,304 atoms, us
// per step: 4 10.2 / 13.7 / 18.5, 8 9.2 / 12.7 / 19.2, 16 11.1 / 15.3 / 22.1;
// 1024 threads 14.3 / 18.9 / 23.8).
constexpr int kFewUnroll = 8;

// The list build's shared memory: masks of 128 candidates a warp, 2.2 KB (the
// rest of the SM's memory is the steps' L1 cache).
constexpr int kResidentTile = 4;
// Whether a rebuild's rows take nine lanes each (small boxes) rather than a warp
// per cell (two or four where there are fewer cells than two a warp).  us per step at dt
// 0.005 (a rebuild every 14 to 20 steps): 864 atoms 10.20 with nine lanes, 10.62
// with the warps; 32,000 atoms FP64 34.7 with a thread per row, 32.7 with the
// warps; 108,000 mixed 38.7 and 38.4 (39.0 with one warp a cell).
bool lanes_per_row(int n, long long threads) { return (long long)n * kRowLanes <= 2 * threads; }

// About two seconds of polling; a barrier is reached within microseconds.
constexpr int kPollLimit = 1 << 22;

__device__ __forceinline__ unsigned load_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier number `k` (from 1) of this launch over all blocks.  Returns false
// (to every thread of the block) when the others did not arrive in time.
__device__ __forceinline__ bool grid_barrier(ResidentCtl *c, unsigned k) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&c->arrived, 1u);
    const unsigned want = k * gridDim.x;
    int n = 0;
    while (load_acquire(&c->arrived) < want && n < kPollLimit) n++;
    ok = n < kPollLimit && *(volatile int *)&c->failed == 0;
    if (n >= kPollLimit) *(volatile int *)&c->failed = 1;
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// Sum over the block, to thread 0: warps, then their sums by the first warp
// (a serial sum of 16 or 32 doubles by one thread takes a microsecond).
__device__ __forceinline__ double resident_sum(double v) {
  __shared__ double sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  __syncthreads();
  return v;
}

// State that every block carries alike from step to step.
struct Run {
  unsigned barriers;
  bool stale;  // mixed forms: q_end is behind the steps
  int par;
};

// The rebuild of launch_rebuild and launch_build_list as phases; false when it
// halted (or a barrier failed).  Slots are sorted by cell and, in a cell, by
// caller index, as there: here each particle counts the smaller indices in its
// cell instead of sorting the cell.
__device__ __noinline__ bool resident_rebuild(const Geom &g, const Dev &d, ResidentCtl *c, Run &r, int row_lanes) {
  DevFlags *f = d.flags;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  __shared__ int sh[32];
  __shared__ int carry;
  if (tid == 0) {
    f->pairs = 0;
    f->max_count = 0;
    f->fx_wide[0] = f->fx_wide[1] = 0;  // finalize_one sets them anew
  }
  const bool from_mid = g.local_pos && r.stale;
  for (int i = tid; i < g.n; i += nt) wrap_bin_one(g, d, i, from_mid, r.par);
  if (!grid_barrier(c, ++r.barriers) || *(volatile int *)&f->halt != 0) return false;
  // starts of the cells: this block's share of the counts, then the shares before it
  const int share = (g.nrank + gridDim.x - 1) / gridDim.x, c0 = min(share * (int)blockIdx.x, g.nrank),
            c1 = min(c0 + share, g.nrank);
  auto block_total = [&](int v) {  // sum over the block, to every thread
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
    return t;
  };
  int v = 0;
  for (int k = c0 + threadIdx.x; k < c1; k += blockDim.x) v += d.cell_count[k];
  v = block_total(v);
  if (threadIdx.x == 0) d.block_sums[blockIdx.x] = v;
  if (!grid_barrier(c, ++r.barriers)) return false;
  v = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) v += d.block_sums[k];
  v = block_total(v);
  if (threadIdx.x == 0) carry = v;
  __syncthreads();
  for (int base = c0; base < c1; base += blockDim.x) {
    const int k = base + threadIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int own = k < c1 ? d.cell_count[k] : 0;
    int x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    int off = carry;
    for (int w = 0; w < wid; w++) off += sh[w];
    if (k < c1) {
      d.cell_start[k] = off + x - own;
      d.cell_count[k] = 0;
      d.cell_fill[k] = 0;
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = off + x;
    __syncthreads();
  }
  if (tid == 0) d.cell_start[g.nrank] = g.n;
  if (!grid_barrier(c, ++r.barriers)) return false;
  auto rank_of = [&](int key) {
    int x, y, z;
    cell_unkey(key, x, y, z);
    return cell_rank(g, x, y, z);
  };
  for (int i = tid; i < g.n; i += nt) {
    const int cell = rank_of(d.cell[i]);
    const int dst = d.cell_start[cell] + atomicAdd(&d.cell_fill[cell], 1);
    if (!MDG_IN_RANGE(f, kCheckScatter, dst, g.n)) continue;
    d.order[dst] = i;
    d.t_id[dst] = d.id[i];
  }
  if (!grid_barrier(c, ++r.barriers)) return false;
  for (int k = tid; k < g.n; k += nt) {
    const int i = d.order[k], id = d.t_id[k], key = d.cell[i], cell = rank_of(key);
    const int a = d.cell_start[cell], b = d.cell_start[cell + 1];
    int at = a;
    for (int m = a; m < b; m++) at += d.t_id[m] < id ? 1 : 0;
    if (!MDG_IN_RANGE(f, kCheckScatter, at, g.n)) continue;
    double4_32a q = d.q_end[i];
    // index and home cell ride in the padding lane
    q.w = __longlong_as_double((long long)(((unsigned long long)(unsigned)key << 32) | (unsigned)id));
    d.t_q[at] = q;
    d.t_p[at] = d.p[i];
  }
  if (!grid_barrier(c, ++r.barriers)) return false;
  for (int k = tid; k < g.n; k += nt) {
    double4_32a q = d.t_q[k];
    const unsigned long long w = (unsigned long long)__double_as_longlong(q.w);
    q.w = 0.0;
    const int id = (int)(unsigned)w, key = (int)(unsigned)(w >> 32);
    if (!MDG_IN_RANGE(f, kCheckScatter, id, g.n)) continue;
    if (g.local_pos) finalize_one<true, false>(g, d, k, q, d.t_p[k], id, key, r.par);
    else finalize_one<false, true>(g, d, k, q, d.t_p[k], id, key, r.par);  // an FP64 box here is in fixed point
  }
  if (!grid_barrier(c, ++r.barriers)) return false;
  r.stale = false;
  // rows: nine lanes each while that fills fewer lanes than there are threads
  // twice over, else a warp per cell, or two or four of few cells
  const int wl = threadIdx.x & 31, warp = tid >> 5, warps = nt >> 5;
  int pairs = 0, longest = 0;
  if (row_lanes) {
    const int per = 32 / kRowLanes, k = wl / kRowLanes, lane = wl % kRowLanes;
    for (int i0 = warp * per; i0 < g.n; i0 += warps * per) {
      const int i = i0 + k;
      const bool active = k < per && i < g.n;
      const int cnt = build_slot_row(g, d, i, active, lane, wl - lane);
      if (active && lane == 0) keep_row_length(g, d, i, cnt, pairs, longest);
    }
  } else {
    extern __shared__ __align__(16) unsigned char s_dynamic[];
    CellRows<kResidentTile> *rows = reinterpret_cast<CellRows<kResidentTile> *>(s_dynamic);
    const int cells = g.nc[0] * g.nc[1] * g.nc[2], split = cells >= 2 * warps ? 1 : (cells >= warps ? 2 : 4);
    for (int item = warp; item < g.nrank * split; item += warps)
      build_cell_rows(g, d, rows[threadIdx.x >> 5], item / split, item % split, split, pairs, longest);
  }
  pairs = __reduce_add_sync(0xffffffffu, pairs);  // at most 2^20 particles of 2^10 entries
  longest = __reduce_max_sync(0xffffffffu, longest);
  if (wl == 0 && longest) {
    atomicAdd(&f->pairs, (unsigned long long)pairs);
    atomicMax(&f->max_count, longest);
  }
  return grid_barrier(c, ++r.barriers) && *(volatile int *)&f->halt == 0;
}

// The force and advance of the block's slots [lo, hi) in one step; the
// block's kinetic energy (Nose-Hoover) to thread 0.
template <int FORM, int THERMO, int COMPAT, int LANES, int THREADS, bool PRUNE>
__device__ __forceinline__ double resident_step(const Geom &g, const Dev &d, int par, int lo, int hi, double exp1,
                                                unsigned long long lang, int *rebuild, int *reselect, unsigned long long *inner) {
  constexpr int kThreads = THREADS;
  const uint32_t *list = PRUNE ? d.nl : d.pl;
  const int *counts = PRUNE ? d.ncount : d.pcount;
  double ke = 0.0;
  unsigned long long kept_sum = 0;
  if constexpr (FORM == kFixedForm) {
    constexpr int kParticles = kThreads / LANES;
    __shared__ double3 sF[LANES > 1 ? kParticles : 1];
    __shared__ int sk[LANES > 1 ? kParticles : 1];
    const bool wide = *(volatile int *)&d.flags->fx_wide[par] != 0;
    const int lane = threadIdx.x % LANES;
    for (int i0 = lo; i0 < hi; i0 += kParticles) {
      int i = i0 + threadIdx.x / LANES, kept = 0;
      bool active = i < hi;
      double3 F = make_double3(0.0, 0.0, 0.0);
      // warps without a particle skip the row walk
      if (__any_sync(0xffffffffu, active)) {
        const int ia = active ? i : hi - 1;
        F = force_fixed<PRUNE, LANES, true>(g, d, d.xq[par], d.q_mid[par], ld_fix<true>(d.xq[par] + ia), ia, wide, list, counts,
                                            active, lane, kept);
      }
      if (LANES > 1) {
        if (active && lane == 0) {
          sF[threadIdx.x / LANES] = F;
          sk[threadIdx.x / LANES] = kept;
        }
        __syncthreads();
        i = i0 + threadIdx.x;
        active = threadIdx.x < kParticles && i < hi;
        kept = 0;
        if (active) {
          F = sF[threadIdx.x];
          kept = sk[threadIdx.x];
        }
      }
      if (active) ke += step_one_fixed<THERMO, COMPAT>(g, d, par, i, PRUNE, kept, F, exp1, lang, rebuild, reselect);
      kept_sum += (unsigned long long)(active ? kept : 0);
      if (LANES > 1) __syncthreads();
    }
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += kThreads) {
      int kept = 0;
      const float4 lb = ld_ro<true>(d.loc[par] + i);
      const double3 F = force_mixed<PRUNE, FORM == MDG_MIXED, true, THREADS <= 512 ? kFewUnroll : kUnroll>(g, d, d.loc[par], i, lb, cell_pos_packed(g, lb.w), list,
                                                                    counts, &kept);
      ke += step_one<THERMO, COMPAT, FORM>(g, d, par, i, PRUNE, kept, F, lb, d.q_mid[par], d.q_mid[par ^ 1], exp1, lang, rebuild,
                                           reselect);
      kept_sum += (unsigned long long)kept;
    }
  }
  if (PRUNE) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) kept_sum += __shfl_down_sync(0xffffffffu, kept_sum, o);
    if ((threadIdx.x & 31) == 0 && kept_sum) atomicAdd(inner, kept_sum);
  }
  if (THERMO == MDG_NOSEHOOVER) ke = resident_sum(ke);
  return ke;
}

template <int FORM, int THERMO, int COMPAT, int LANES, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 2 : 1) k_resident(const __grid_constant__ Geom g,
                                                                      const __grid_constant__ Dev d, ResidentCtl *c, int par,
                                                                      int nsteps, int share, int row_lanes) {
  constexpr int kThreads = THREADS;
  DevFlags *f = d.flags;
  // the flags of the state before this launch: nobody writes them until its end
  // (a halt is set in the rebuild only, between barriers; by a failed check
  // anywhere, and read after the next rebuild's first barrier)
  if (*(volatile int *)&f->halt != 0) return;
  Run r{0u, f->end_stale != 0, par};
  bool rebuild = f->rebuild != 0, reselect = f->prune_next != 0;
  const unsigned long long lang0 = f->lang;
  double zeta = f->zeta, zeta_a = f->zeta_a, exp1 = f->exp1, T = f->t_cur;
  unsigned long long rebuilds = 0, prunes = 0;
  // a rebuild of the first step may set the halt before its first barrier (and a
  // checked build any step): not before every block has read it above
  bool halted = false, lost = (rebuild || kCheck) && !grid_barrier(c, ++r.barriers);
  const int lo = min((int)blockIdx.x * share, g.n), hi = min(lo + share, g.n);
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  int s = 0, selected = -1;  // slot of the last selection's row total
  for (; s < nsteps && !lost; s++) {
    if (s > 0) {
      rebuild = *(volatile int *)&c->rebuild[s % 3] != 0;
      reselect = *(volatile int *)&c->reselect[s % 3] != 0;
      if (first) {
        if (selected >= 0) f->inner_pairs = *(volatile unsigned long long *)&c->inner[selected];
        const int old = (s + 2) % 3;  // read by every block before the last barrier
        c->rebuild[old] = c->reselect[old] = 0;
      }
      selected = -1;
    }
    if (rebuild) {
      if (!resident_rebuild(g, d, c, r, row_lanes)) {
        halted = true;
        break;
      }
      rebuilds++;
      reselect = true;
    }
    const int slot = s % 3, next = (s + 1) % 3;
    // this step's row total was last read two barriers ago
    double ke;
    const unsigned long long lang = lang0 + (unsigned long long)s;
    if (reselect) {
      ke = resident_step<FORM, THERMO, COMPAT, LANES, THREADS, true>(g, d, r.par, lo, hi, exp1, lang, &c->rebuild[next], &c->reselect[next],
                                                            &c->inner[slot]);
      prunes++;
      selected = slot;
    } else {
      ke = resident_step<FORM, THERMO, COMPAT, LANES, THREADS, false>(g, d, r.par, lo, hi, exp1, lang, &c->rebuild[next], &c->reselect[next],
                                                             nullptr);
    }
    r.stale = g.local_pos != 0;
    r.par ^= 1;
    // sums of consecutive steps in alternate halves: a block may be a step ahead of a reader
    double *part = d.partials + (s & 1) * gridDim.x;
    if (THERMO == MDG_NOSEHOOVER && threadIdx.x == 0) part[blockIdx.x] = ke;
    if (!grid_barrier(c, ++r.barriers)) {
      lost = true;
      break;
    }
    if (first) c->inner[(s + 2) % 3] = 0;  // its reader (step s at the latest) is this thread
    if (THERMO == MDG_NOSEHOOVER) {  // k_nh_update, by one thread of every block
      __shared__ double nh[4];
      double v = 0.0;
      for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads) v += part[b];
      v = resident_sum(v);
      if (threadIdx.x == 0) {
        const double now = v / (double)g.n / 1.5, dt2 = g.dt * 0.5, t1 = (now - g.temperature) / (g.tau * g.tau);
        nh[0] = now;
        nh[1] = zeta_a + t1 * dt2;
        nh[2] = nh[1] + t1 * dt2;
        nh[3] = exp(-dt2 * nh[2]);
      }
      __syncthreads();
      T = nh[0];
      zeta = nh[1];
      zeta_a = nh[2];
      exp1 = nh[3];
    }
  }
  // every block is past its last barrier before the last one to leave writes
  // the state back and clears the control words for the next launch
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&c->left, 1u) == gridDim.x - 1 ? 1 : 0;
    __threadfence();
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  if (lost || *(volatile int *)&c->failed) halt_with(f, kHaltBarrier);
  const int done = halted ? s + 1 : s;  // a halted step counts as begun
  f->steps += (unsigned long long)done;
  if (THERMO == MDG_LANGEVIN) f->lang = lang0 + (unsigned long long)done;
  f->rebuilds += rebuilds;
  f->prunes += prunes;
  f->end_stale = r.stale ? 1 : 0;
  if (halted) {
    f->rebuild = 1;
    f->prune_next = 0;
  } else {
    f->rebuild = *(volatile int *)&c->rebuild[s % 3];
    f->prune_next = *(volatile int *)&c->reselect[s % 3];
    if (selected >= 0) f->inner_pairs = *(volatile unsigned long long *)&c->inner[selected];
  }
  f->prune_now = 0;
  if (THERMO == MDG_NOSEHOOVER) {
    f->zeta = zeta;
    f->zeta_a = zeta_a;
    f->exp1 = exp1;
    f->t_cur = T;
  }
  for (int k = 0; k < 3; k++) {
    c->rebuild[k] = c->reselect[k] = 0;
    c->inner[k] = 0;
  }
  c->failed = 0;
  c->left = 0;
  __threadfence();
  c->arrived = 0;
}

using Kernel = void (*)(const Geom, const Dev, ResidentCtl *, int, int, int, int);

template <int FORM, int LANES, int THREADS>
Kernel kernel_of(int thermostat, int compat) {
  if (thermostat == MDG_LANGEVIN)
    return compat ? k_resident<FORM, MDG_LANGEVIN, 1, LANES, THREADS> : k_resident<FORM, MDG_LANGEVIN, 0, LANES, THREADS>;
  if (thermostat == MDG_NOSEHOOVER) return k_resident<FORM, MDG_NOSEHOOVER, 0, LANES, THREADS>;
  return k_resident<FORM, MDG_NVE, 0, LANES, THREADS>;
}

}  // namespace

// Particles per SM up to which a box takes the resident kernel.  us per step,
// resident against graphs (density 0.6, dt 0.002, 200 steps with their
// rebuilds): FP64 864 atoms 8.1 / 20.1, 4,000 9.8 / 21.6, 32,000 23.6 / 34.7,
// 70,304 35.8 / 53.6, 108,000 65.0 / 66.9, 157,216 97.9 / 88.8 (a second pass
// over the block's 512 threads); mixed 864 9.2 / 28.6, 32,000 14.6 / 33.9,
// 108,000 27.1 / 39.3, 157,216 47.1 / 48.1, 256,000 54.9 / 66.7, 389,344 84.9 / 89.7.
constexpr int kResidentFixed = 512, kResidentMixed = 2048;

// Beside other handles.  A block of 512 threads has an SM's registers to itself
// and a launch takes nearly every SM, so the launches of several handles run one
// after the other, where step graphs overlap.  In the mixed forms a call made while
// other handles have steps outstanding therefore takes, up to 256 particles per SM,
// a narrow launch: kNarrowRows particles a block (a warp on each sub-partition),
// which shares the SMs out up to 64 per SM, and above that blocks of 256 threads, two
// of which fit an SM.  Larger boxes step by graphs where those are faster (crowded in
// mdg_api.cu).  us per step of all handles, density 0.6, dt 0.002, one / four / eight, now
// (wide launches only; graphs only): 864 9.5 / 9.9 / 10.1 (9.4 / 9.8 / 16.7; 30 / 40 / 79),
// 4,000 10.3 / 13.2 / 23.3 (10.2 / 40.7 / 82; 32 / 39 / 78), 16,384 11.4 / 30.5 / 58.7 (11.4 /
// 43.9 / 90; 34 / 42 / 84), 32,000 14.4 / 40 / 77 (14.3 / 57 / 114; 35 / 47 / 93), 108,000
// 27.8 / 82 / 155 (27.7 / 111 / 221; 40 / 79 / 158), 300,000 60.8 / 189 / 372 (60.5 / 242 / 482;
// 78 / 189 / 376).  Not narrow always: fewer threads make the rebuild longer, and one
// handle 5-14 % slower at dt 0.005 (1,500 13.2 -> 15.2, 16,384 16.4 -> 17.4).  The
// particles' arithmetic is the same, bit for bit; Nose-Hoover, whose kinetic sum
// goes by blocks, stays with the wide launch, and FP64 handles side by side are
// faster than their graphs at every size (four of 32,000 95, 272).
constexpr int kNarrowRows = 128;
bool narrow_box(const Geom &g, int thermostat, int precision, int num_sms) {
  return precision != MDG_FP64 && thermostat != MDG_NOSEHOOVER && g.n <= 256 * num_sms;
}

size_t resident_ctl_bytes() { return sizeof(ResidentCtl); }

bool resident_box(const Geom &g, int precision, int num_sms) {
  return g.rebuild_policy == MDG_REBUILD_HALFMARGIN && (precision != MDG_FP64 || g.fixed) && num_sms <= 2048 &&
         g.n <= (precision == MDG_FP64 ? kResidentFixed : kResidentMixed) * num_sms;
}

cudaError_t launch_resident(const Geom &g, const Dev &d, void *ctl, int par, int nsteps, int thermostat, int compat, int precision,
                            int num_sms, bool beside, cudaStream_t s) {
  Kernel k;
  const bool narrow = beside && narrow_box(g, thermostat, precision, num_sms);
  int threads = 512, lanes = 1;
  if (precision == MDG_FP64) {
    // as many lanes as the block has threads for
    const int share = (g.n + num_sms - 1) / num_sms;
    while (lanes < 32 && 2 * lanes * share <= threads) lanes *= 2;
    k = lanes == 32   ? kernel_of<kFixedForm, 32, 512>(thermostat, compat)
        : lanes == 16 ? kernel_of<kFixedForm, 16, 512>(thermostat, compat)
        : lanes == 8  ? kernel_of<kFixedForm, 8, 512>(thermostat, compat)
        : lanes == 4  ? kernel_of<kFixedForm, 4, 512>(thermostat, compat)
        : lanes == 2  ? kernel_of<kFixedForm, 2, 512>(thermostat, compat)
                      : kernel_of<kFixedForm, 1, 512>(thermostat, compat);
  } else if (narrow && 2 * g.n > kNarrowRows * num_sms) {
    threads = 256;
    k = precision == MDG_MIXED ? kernel_of<MDG_MIXED, 1, 256>(thermostat, compat)
                               : kernel_of<MDG_MIXED_PLAIN, 1, 256>(thermostat, compat);
  } else if (g.n <= 512 * num_sms) {
    k = precision == MDG_MIXED ? kernel_of<MDG_MIXED, 1, 512>(thermostat, compat)
                               : kernel_of<MDG_MIXED_PLAIN, 1, 512>(thermostat, compat);
  } else {
    threads = 1024;
    k = precision == MDG_MIXED ? kernel_of<MDG_MIXED, 1, 1024>(thermostat, compat)
                               : kernel_of<MDG_MIXED_PLAIN, 1, 1024>(thermostat, compat);
  }
  // whole warps of particles per block
  const int unit = 32 / lanes;
  int share = (g.n + num_sms - 1) / num_sms;
  if (narrow && share < kNarrowRows) share = kNarrowRows;
  share = (share + unit - 1) / unit * unit;
  int grid = (g.n + share - 1) / share;
  Geom gg = g;
  Dev dd = d;
  ResidentCtl *c = static_cast<ResidentCtl *>(ctl);
  int row_lanes = lanes_per_row(g.n, (long long)grid * threads) ? 1 : 0;
  void *args[] = {&gg, &dd, &c, &par, &nsteps, &share, &row_lanes};
  size_t shared = 0;
  if (!row_lanes) {
    shared = threads / 32 * sizeof(CellRows<kResidentTile>);
    if (shared > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void *>(k), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k), dim3(grid), dim3(threads), args, shared, s);
}

}  // namespace mdg

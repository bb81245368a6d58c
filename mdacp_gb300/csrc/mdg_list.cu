// Pair-list rebuild, part 2: the padded neighbour list.
//
// Replaces MeshList::SearchMesh / AppendList / RegisterPair and the COO->CSR
// step of MeshList::MakeList (meshlist.cc:57-87, 207-310) together with the
// ghost images of MDManager::MakePairList (mdmanager.cc:262-280,
// mdunit.cc:125-191).  Instead of ghost copies each slot scans the 27 cells
// around its own with periodic wrap and records every partner image within
// the search length rc + margin: a full (both directions) list, so the force
// kernel gathers without atomics.
//
// Acceptance is decided exactly as the reference decides it: the image
// position is formed first, q_j +- L (mdunit.cc:167), then the difference and
// r2 = dx*dx + dy*dy + dz*dz with every operation rounded separately
// (meshlist.cc:262-266), accepted when r2 <= SL^2.  Candidates are first
// measured in float from home-cell-local positions, whose r2 is within 1e-5
// of the exact value; only those within 1e-4 of SL^2 take the double test,
// so the result is the exact set at float cost.  The order of the entries in
// a row (stencil cell by cell, near side first) carries no meaning.
#include "mdg_rebuild.cuh"

namespace mdg {

namespace {

// Threads per block of the list build.  A block's slots are consecutive in
// cell order, so larger blocks keep more neighbouring cells on one SM and
// their candidate loads hit L1 (forced rebuild of the 4M-atom liquid box: 128
// threads 3.55 ms, 256 3.44, 384 3.21); below a million particles the grid
// has too few of them for the SMs (256,000 atoms: 128 threads 0.366 ms, 384 0.404).
constexpr int kListThreads = 384, kListThreadsSmall = 128, kListLarge = 1000000;
// Below this many particles nine lanes share a slot: forced rebuild of 864
// atoms 124 -> 95 us, of 32,000 143 -> 120; 108,000 atoms have warps enough
// (174 us with one thread per slot, 230 with nine lanes).
constexpr int kLanesBelow = 49152;

// One thread per slot (LANES = 1), or LANES = 9 lanes of a warp per slot.
template <int LANES, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) k_build_list(Geom g, Dev d) {
  DevFlags *f = d.flags;
  // one read for the whole block: another block may set the halt meanwhile
  __shared__ int s_run;
  if (threadIdx.x == 0) s_run = f->halt == 0 && f->rebuild != 0;
  __syncthreads();
  if (!s_run) return;
  constexpr int kPerWarp = LANES == 1 ? 32 : 32 / LANES;  // slots of a warp
  const int wl = threadIdx.x & 31;
  const int lane = LANES == 1 ? 0 : wl % LANES;
  const int i = LANES == 1 ? blockIdx.x * blockDim.x + threadIdx.x
                           : (blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5)) * kPerWarp + wl / LANES;
  const bool active = i < g.n && wl < kPerWarp * LANES;
  const int cap = g.list_cap;
  const int cnt = build_slot_row<LANES>(g, d, i, active, lane, wl - lane);
  unsigned long long tot = 0;
  int mx = 0;
  if (active && lane == 0) {
    d.ncount[i] = cnt < cap ? cnt : cap;
    if (cnt > cap) {
      atomicMax(&f->overflow_max, cnt);
      halt_with(f, kHaltOverflow);
    }
    tot = (unsigned long long)(cnt < cap ? cnt : cap);
    mx = cnt;
  }
  // block totals -> one atomic each
  __shared__ unsigned long long s_sum[THREADS / 32];
  __shared__ int s_max[THREADS / 32];
  unsigned long long v = tot;
  int m = mx;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_down_sync(0xffffffffu, v, o);
    m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  }
  if ((threadIdx.x & 31) == 0) { s_sum[threadIdx.x >> 5] = v; s_max[threadIdx.x >> 5] = m; }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tv = 0;
    int tm = 0;
    for (int w = 0; w < THREADS / 32; w++) { tv += s_sum[w]; tm = max(tm, s_max[w]); }
    atomicAdd(&f->pairs, tv);
    atomicMax(&f->max_count, tm);
  }
}

// A new outer list always gets a fresh inner list: in this step's kernel
// when the rebuild ran inside a step, otherwise in the next step's.
__global__ void k_rebuild_done(DevFlags *f, int in_step) {
  if (f->halt == 0 && f->rebuild) {
    f->rebuild = 0;
    f->rebuilds += 1;
    if (!in_step) {
      f->prune_next = 1;
    } else if (!f->prune_now) {
      f->prune_now = 1;
      f->prunes += 1;
      f->inner_pairs = 0;
    }
  }
}

__global__ void k_list_prepare(DevFlags *f) {
  if (f->halt == 0 && f->rebuild) {
    f->pairs = 0;
    f->max_count = 0;
  }
}

}  // namespace

void launch_build_list(const Geom &g, const Dev &d, int num_sms, cudaStream_t s, bool in_step) {
  k_list_prepare<<<1, 1, 0, s>>>(d.flags);
  // one slot per thread, or per nine lanes: the blocks' work is uneven
  // (denser regions have more candidates), and many blocks balance it where
  // resident blocks striding over the slots did not (4M atoms, one wave: 25 % slower)
  (void)num_sms;
  auto grid = [&](int slots) { return g.n > 0 ? (g.n + slots - 1) / slots : 1; };
  if (g.n < kLanesBelow)
    k_build_list<kRowLanes, kListThreadsSmall><<<grid(kListThreadsSmall / 32 * (32 / kRowLanes)), kListThreadsSmall, 0, s>>>(g, d);
  else if (g.n < kListLarge)
    k_build_list<1, kListThreadsSmall><<<grid(kListThreadsSmall), kListThreadsSmall, 0, s>>>(g, d);
  else
    k_build_list<1, kListThreads><<<grid(kListThreads), kListThreads, 0, s>>>(g, d);
  k_rebuild_done<<<1, 1, 0, s>>>(d.flags, in_step ? 1 : 0);
}

}  // namespace mdg

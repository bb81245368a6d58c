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

// One warp per home cell, or two below kSplitBelow cells an SM: forced rebuild of
// 32,000 atoms 159 us with one, 149 with two, 158 with four; of 131,072 (about
// 4,900 cells) 201, 213, 248.  The blocks' work is uneven (denser regions have
// more candidates): many small blocks balance it.
constexpr int kListWarps = 8;
constexpr long long kSplitBelow = 20;
__global__ void __launch_bounds__(32 * kListWarps, 4) k_build_list(Geom g, Dev d, int split) {
  DevFlags *f = d.flags;
  // one read for the whole block: another block may set the halt meanwhile
  __shared__ int s_run;
  __shared__ CellRows<kTileChunks> s_rows[kListWarps];
  if (threadIdx.x == 0) s_run = f->halt == 0 && f->rebuild != 0;
  __syncthreads();
  if (!s_run) return;
  const int warp = threadIdx.x >> 5, item = blockIdx.x * kListWarps + warp, home = item / split, part = item % split;
  int v = 0, mx = 0;
  if (home < g.nrank) build_cell_rows(g, d, s_rows[warp], home, part, split, v, mx);
  // block totals -> one atomic each
  __shared__ int s_sum[kListWarps], s_max[kListWarps];
  v = __reduce_add_sync(0xffffffffu, v);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) { s_sum[warp] = v; s_max[warp] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tv = 0;
    int tm = 0;
    for (int w = 0; w < kListWarps; w++) { tv += s_sum[w]; tm = max(tm, s_max[w]); }
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
  const long long cells = (long long)g.nc[0] * g.nc[1] * g.nc[2];
  const int split = cells >= kSplitBelow * num_sms ? 1 : 2;
  k_build_list<<<(g.nrank * split + kListWarps - 1) / kListWarps, 32 * kListWarps, 0, s>>>(g, d, split);
  k_rebuild_done<<<1, 1, 0, s>>>(d.flags, in_step ? 1 : 0);
}

}  // namespace mdg

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

// A block's listed pairs and longest row from each lane's, one atomic each.
__device__ __forceinline__ void add_totals(DevFlags *f, int v, int mx) {
  __shared__ int s_sum[32], s_max[32];
  const int warp = threadIdx.x >> 5;
  v = __reduce_add_sync(0xffffffffu, v);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) { s_sum[warp] = v; s_max[warp] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tv = 0;
    int tm = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) { tv += s_sum[w]; tm = max(tm, s_max[w]); }
    atomicAdd(&f->pairs, tv);
    atomicMax(&f->max_count, tm);
  }
}

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
  add_totals(f, v, mx);
}

// One thread per particle, for boxes of few particles a cell: the 27 stencil
// cells in turn, kRowUnroll candidates at a time, each accepted one appended as
// it is found.  A warp per cell has too little to do there, and most of the
// cells of a gas are empty.  Forced rebuild, thread per particle / warp per cell
// (cut-off 2.5, margin 0.5), us: 1M at density 0.005 328 / 3,670, 0.05 339 / 855, 0.1
// 354 / 606, 0.2 474 / 498, 0.25 536 / 499; 100,000 at 0.05 94 / 135, 0.15 104 / 105, 0.2
// 106 / 105; 30,000 at 0.05 81 / 91, 0.1 85 / 83; 10,000 at 0.005 (74,000 cells) 78 / 101, 0.02
// (18,500) 78 / 77, 0.05 82 / 79: the line lies at 6 particles a cell, and at 16,000
// cells, which one wave of warps works off.  (Bound by the chain of loads cell by
// cell; 78 registers, so that the loads of three cells are in flight.)
constexpr double kDilute = 6.0;
constexpr long long kDiluteCells = 16000;
constexpr int kRowThreads = 384, kRowUnroll = 4;
__global__ void __launch_bounds__(kRowThreads, 1) k_build_rows(Geom g, Dev d) {
  DevFlags *f = d.flags;
  // one read for the whole block: another block may set the halt meanwhile
  __shared__ int s_run;
  if (threadIdx.x == 0) s_run = f->halt == 0 && f->rebuild != 0;
  __syncthreads();
  if (!s_run) return;
  int v = 0, mx = 0;
  const float acc_lo = g.acc_lo, acc_hi = g.acc_hi;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) {
    int cnt = 0;
    const float4 fi = d.qf[i];
    int cx, cy, cz;
    cell_unpack(fi.w, cx, cy, cz);
    uint32_t *row = d.nl + i;
    const size_t stride = (size_t)g.stride;
    const int cap = g.list_cap;
    for (int oz = -1; oz <= 1; oz++) {
      int nz = cz + oz, sz = 0;
      if (nz < 0) { nz += g.nc[2]; sz = -1; } else if (nz >= g.nc[2]) { nz -= g.nc[2]; sz = 1; }
      // offset of the partner cell's centre: oz*w + sz*(L - nc*w)
      const float fz = (float)oz * g.w32[2] + (float)sz * g.dl32[2] - fi.z;
      for (int oy = -1; oy <= 1; oy++) {
        int ny = cy + oy, sy = 0;
        if (ny < 0) { ny += g.nc[1]; sy = -1; } else if (ny >= g.nc[1]) { ny -= g.nc[1]; sy = 1; }
        const float fy = (float)oy * g.w32[1] + (float)sy * g.dl32[1] - fi.y;
        for (int ox = -1; ox <= 1; ox++) {
          int nx = cx + ox, sx = 0;
          if (nx < 0) { nx += g.nc[0]; sx = -1; } else if (nx >= g.nc[0]) { nx -= g.nc[0]; sx = 1; }
          const float fx = (float)ox * g.w32[0] + (float)sx * g.dl32[0] - fi.x;
          const int cc = cell_rank(g, nx, ny, nz);
          if (!MDG_IN_RANGE(f, kCheckBuildCell, cc, g.nrank)) continue;
          int a = d.cell_start[cc], b = d.cell_start[cc + 1];
          if (!MDG_IN_RANGE(f, kCheckBuildRange, b, g.n + 1) || !MDG_IN_RANGE(f, kCheckBuildRange, a, b + 1)) a = b = 0;
          const uint32_t code = entry_pack(0, ox, oy, oz);
          for (int j0 = a; j0 < b; j0 += kRowUnroll) {
            float4 fj[kRowUnroll];
#pragma unroll
            for (int u = 0; u < kRowUnroll; u++)
              fj[u] = j0 + u < b ? d.qf[j0 + u] : make_float4(1e30f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < kRowUnroll; u++) {
              const int j = j0 + u;
              const float ex = fj[u].x + fx, ey = fj[u].y + fy, ez = fj[u].z + fz;
              const float r2f = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
              if (r2f > acc_hi || j == i) continue;
              bool take = r2f < acc_lo;
              if (!take) take = image_within(d.q_end[i], d.q_end[j], g.L, sx, sy, sz, g.sl2);
              if (take) {
                if (cnt < cap) row[(size_t)cnt * stride] = ((uint32_t)j << kCodeBits) | code;
                cnt++;
              }
            }
          }
        }
      }
    }
    keep_row_length(g, d, i, cnt, v, mx);
  }
  add_totals(f, v, mx);
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
  if (cells >= kDiluteCells && (double)g.n < kDilute * (double)cells) {
    k_build_rows<<<(g.n + kRowThreads - 1) / kRowThreads, kRowThreads, 0, s>>>(g, d);
  } else {
    const int split = cells >= kSplitBelow * num_sms ? 1 : 2;
    k_build_list<<<(g.nrank * split + kListWarps - 1) / kListWarps, 32 * kListWarps, 0, s>>>(g, d, split);
  }
  k_rebuild_done<<<1, 1, 0, s>>>(d.flags, in_step ? 1 : 0);
}

}  // namespace mdg

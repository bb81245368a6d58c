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
// more candidates): many small blocks balance it, resident ones striding over
// the cells did not (4M atoms, one wave: 25 % slower).
constexpr int kListWarps = 8;
constexpr long long kSplitBelow = 20;
__global__ void __launch_bounds__(32 * kListWarps, 4) k_build_list(Geom g, Dev d, int split) {
  DevFlags *f = d.flags;
  // one read for the whole block: another block may set the halt meanwhile
  __shared__ int s_run;
  __shared__ CellRows s_rows[kListWarps];
  if (threadIdx.x == 0) s_run = f->halt == 0 && f->rebuild != 0;
  __syncthreads();
  if (!s_run) return;
  const int warp = threadIdx.x >> 5, item = blockIdx.x * kListWarps + warp, home = item / split, part = item % split;
  const int cap = g.list_cap;
  int a = 0, b = 0;
  if (home < g.nrank) {
    a = d.cell_start[home];
    b = d.cell_start[home + 1];
  }
  if (!MDG_IN_RANGE(f, kCheckBuildRange, b, g.n + 1) || !MDG_IN_RANGE(f, kCheckBuildRange, a, b + 1)) a = b = 0;
  int v = 0, mx = 0;
  const int from = a + (b - a) * part / split, to = a + (b - a) * (part + 1) / split;
  if (from < to) {
    int cx, cy, cz;
    cell_unpack(d.qf[a].w, cx, cy, cz);
    cell_rows(
        s_rows[warp], d.qf, a, from, to, g.acc_lo, g.acc_hi, cap,
        [&](int l, int &first, int &count, float3 &shift, uint32_t &code) {
          const int ox = l % 3 - 1, oy = l / 3 % 3 - 1, oz = l / 9 - 1;
          int sx, sy, sz;
          const int nx = wrap_cell(cx, ox, g.nc[0], sx), ny = wrap_cell(cy, oy, g.nc[1], sy), nz = wrap_cell(cz, oz, g.nc[2], sz);
          // offset of the partner cell's centre: o*w + s*(L - nc*w)
          shift.x = (float)ox * g.w32[0] + (float)sx * g.dl32[0];
          shift.y = (float)oy * g.w32[1] + (float)sy * g.dl32[1];
          shift.z = (float)oz * g.w32[2] + (float)sz * g.dl32[2];
          code = entry_pack(0, ox, oy, oz);
          const int cc = cell_rank(g, nx, ny, nz);
          if (!MDG_IN_RANGE(f, kCheckBuildCell, cc, g.nrank)) return;
          int lo = d.cell_start[cc], hi = d.cell_start[cc + 1];
          if (!MDG_IN_RANGE(f, kCheckBuildRange, hi, g.n + 1) || !MDG_IN_RANGE(f, kCheckBuildRange, lo, hi + 1)) return;
          first = lo;
          count = hi - lo;
        },
        [&](int i, int j, int l) {
          int sx, sy, sz;
          wrap_cell(cx, l % 3 - 1, g.nc[0], sx);
          wrap_cell(cy, l / 3 % 3 - 1, g.nc[1], sy);
          wrap_cell(cz, l / 9 - 1, g.nc[2], sz);
          return image_within(d.q_end[i], d.q_end[j], g.L, sx, sy, sz, g.sl2);
        },
        RowSink{d.nl, (size_t)g.stride, nullptr},
        [&](int i, int cnt) {
          d.ncount[i] = cnt < cap ? cnt : cap;
          if (cnt > cap) {
            atomicMax(&f->overflow_max, cnt);
            halt_with(f, kHaltOverflow);
          }
          v += cnt < cap ? cnt : cap;
          mx = max(mx, cnt);
        });
  }
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

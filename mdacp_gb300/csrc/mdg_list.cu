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
#include "mdg_build.cuh"

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

// Exact acceptance of a candidate in the float band: the reference's image
// and rounding order (mdunit.cc:167, meshlist.cc:262-266).
__device__ __forceinline__ bool exact_within(const Geom &g, const double4_32a &qi, const double4_32a &qj, int sx, int sy,
                                             int sz) {
  const double xj = sx ? __dadd_rn(qj.x, sx > 0 ? g.L[0] : -g.L[0]) : qj.x;
  const double yj = sy ? __dadd_rn(qj.y, sy > 0 ? g.L[1] : -g.L[1]) : qj.y;
  const double zj = sz ? __dadd_rn(qj.z, sz > 0 ? g.L[2] : -g.L[2]) : qj.z;
  const double dx = __dsub_rn(qi.x, xj), dy = __dsub_rn(qi.y, yj), dz = __dsub_rn(qi.z, zj);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return r2 <= g.sl2;
}

// One thread per slot (LANES = 1), or LANES = 9 lanes of a warp per slot, one for
// each (y, z) row of three stencil cells: a row's candidates then take a
// ninth of the time one after the other, which is what a small box waits for.
// The rows' entries are in stencil order (z, y, x), candidates ascending, either way.
constexpr int kRowLanes = 9;
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
  const float acc_lo = g.acc_lo, acc_hi = g.acc_hi;
  const int cap = g.list_cap;
  const size_t stride = (size_t)g.stride;
  uint32_t *row = d.nl + i;
  int cnt = 0;
  float4 fi = make_float4(0.f, 0.f, 0.f, 0.f);
  int cx = 0, cy = 0, cz = 0;
  if (active) {
    fi = d.qf[i];
    cell_unpack(fi.w, cx, cy, cz);
  }
  // candidates of stencil cell (ox, oy, oz): emit(mask, j0, code) for every 32
  auto scan = [&](int ox, int oy, int oz, auto &&emit) {
    int sx, sy, sz;
    const int nx = wrap_cell(cx, ox, g.nc[0], sx), ny = wrap_cell(cy, oy, g.nc[1], sy), nz = wrap_cell(cz, oz, g.nc[2], sz);
    // offset of the partner cell's centre: o*w + s*(L - nc*w)
    const float fx = (float)ox * g.w32[0] + (float)sx * g.dl32[0] - fi.x;
    const float fy = (float)oy * g.w32[1] + (float)sy * g.dl32[1] - fi.y;
    const float fz = (float)oz * g.w32[2] + (float)sz * g.dl32[2] - fi.z;
    const int cc = cell_rank(g, nx, ny, nz);
    if (!MDG_IN_RANGE(f, kCheckBuildCell, cc, g.nrank)) return;
    int a = d.cell_start[cc], b = d.cell_start[cc + 1];
    if (!MDG_IN_RANGE(f, kCheckBuildRange, b, g.n + 1) || !MDG_IN_RANGE(f, kCheckBuildRange, a, b + 1)) a = b = 0;
    const uint32_t code = entry_pack(0, ox, oy, oz);
    for (int j0 = a; j0 < b; j0 += 32) {
      uint32_t in, sure;
      chunk_masks(d.qf, j0, min(b - j0, 32), fx, fy, fz, acc_lo, acc_hi, in, sure);
      if ((unsigned)(i - j0) < 32u) in &= ~(1u << (i - j0));  // the particle itself (its images are a box away)
      for (uint32_t band = in & ~sure; band; band &= band - 1u) {
        const int u = __ffs(band) - 1;
        if (!exact_within(g, d.q_end[i], d.q_end[j0 + u], sx, sy, sz)) in &= ~(1u << u);
      }
      emit(in, j0, code);
    }
  };
  auto append = [&](uint32_t in, int j0, uint32_t code) {
    for (; in; in &= in - 1u) {
      const int j = j0 + __ffs(in) - 1;
      if (cnt < cap) row[(size_t)cnt * stride] = ((uint32_t)j << kCodeBits) | code;
      cnt++;
    }
  };
  if (LANES == 1) {
    if (active)
      for (int oz = -1; oz <= 1; oz++)
        for (int oy = -1; oy <= 1; oy++)
          for (int ox = -1; ox <= 1; ox++) scan(ox, oy, oz, append);
  } else {
    // the first masks of each cell are kept between counting and writing;
    // cells of more than 32 particles are scanned again
    const int oy = lane % 3 - 1, oz = lane / 3 - 1;
    int own = 0;
    uint32_t kept[3] = {0u, 0u, 0u};
    int first[3] = {0, 0, 0};
    bool again = false;
    if (active)
#pragma unroll
      for (int ox = -1; ox <= 1; ox++) {
        int chunk = 0;
        scan(ox, oy, oz, [&](uint32_t in, int j0, uint32_t) {
          own += __popc(in);
          if (chunk++ == 0) {
            kept[ox + 1] = in;
            first[ox + 1] = j0;
          } else {
            again = true;
          }
        });
      }
    // entries of the particle's lower lanes, and of all
    const int base = wl - lane;
    int before = 0, total = 0;
#pragma unroll
    for (int l = 0; l < LANES; l++) {
      const int v = __shfl_sync(0xffffffffu, own, min(base + l, 31));
      before += l < lane ? v : 0;
      total += v;
    }
    cnt = before;
    if (active) {
#pragma unroll
      for (int ox = -1; ox <= 1; ox++) {
        if (again) scan(ox, oy, oz, append);
        else append(kept[ox + 1], first[ox + 1], entry_pack(0, ox, oy, oz));
      }
    }
    cnt = total;
  }
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

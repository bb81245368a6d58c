// mdg_observe_noalloc: the observers of mdg_observe for callers that cannot
// allocate device memory.
//
// Who needs it: code that runs where cudaMalloc is unavailable or unsafe --
// inside a memory-pool-managed host application that forbids CUDA
// allocations, inside a host callback or a stream-ordered section that must
// not synchronise the device, or a caller that already owns its particle
// arrays on the device and has no mdg handle (creating one allocates the
// whole pair-list machinery).  Such a caller passes its own device arrays and
// receives the three observer sums in its own device buffer.
//
// How: instead of reading a handle's neighbour list the kernels bin the
// particles into cells of width >= cutoff and scan the 27 neighbouring cells:
// a warp per cell finds the pairs as the list build does (cell_rows) and, in
// place of writing them, adds the handle's fixed-point pair sums
// (mdg_fixed.cuh).  A cut-off outside 1.0 .. 3.9, nearly empty boxes and positions
// that cannot be wrapped into the box take the double expressions, a thread per
// particle.
// All working memory -- cell counts, cell starts, the particle order, the
// positions in it and the per-block partial sums -- is one file-scope
// __device__ array of fixed size, 62 MB (every GPU that loads this library
// holds it until the process exits).  Its device address
// is looked up once per device with cudaGetSymbolAddress on that device's
// first call; nothing is allocated or freed, ever.
#include <cuda_runtime.h>

#include <climits>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <mutex>

#include "mdg_build.cuh"

namespace mdg {
namespace noalloc {

constexpr int kMaxParticles = 1 << 20;  // 1,048,576
constexpr int kMaxCells = 1 << 18;      // 262,144
constexpr int kThreads = 128;
constexpr int kMaxBlocks = kMaxParticles / kThreads;
constexpr int kMaxDevices = 64;

// Layout of the scratch array, in 8-byte words.
constexpr size_t kOffCount = 0;                                   // int[kMaxCells]
constexpr size_t kOffStart = kOffCount + kMaxCells / 2;           // int[kMaxCells + 2]
constexpr size_t kOffFill = kOffStart + kMaxCells / 2 + 1;        // int[kMaxCells]
constexpr size_t kOffCellOf = kOffFill + kMaxCells / 2;           // int[kMaxParticles]
constexpr size_t kOffOrder = kOffCellOf + kMaxParticles / 2;      // int[kMaxParticles]
constexpr size_t kOffPartial = kOffOrder + kMaxParticles / 2;     // double[3 * kMaxBlocks]
constexpr size_t kOffFlag = kOffPartial + 3 * (size_t)kMaxBlocks;  // int
constexpr size_t kOffLocal = (kOffFlag + 32) / 32 * 32;            // float4[kMaxParticles]
constexpr size_t kOffFix = kOffLocal + 2 * (size_t)kMaxParticles;  // FixPos[kMaxParticles]
static_assert(sizeof(FixPos) == 32, "four words each");
constexpr size_t kWords = kOffFix + 4 * (size_t)kMaxParticles;     // 62 MB

static __device__ __align__(256) unsigned long long g_scratch[kWords];

struct Box {
  double L[3], inv_w[3];
  int nc[3], ncell, n;
  double rc2, c0, c2, c2x8;
  // fixed-point form: box sides, cut-off, the close pairs' bound, and the cell
  // widths and the float test's radius
  int fixed, fx_L[3];
  float fx_l[3];
  uint64_t fx_rc2;
  uint32_t fx_near;
  double w[3];
  float w32[3], hi;
};

struct Scratch {
  int *count, *start, *fill, *cell_of, *order, *flag;
  double *partial;
  float4 *local;  // positions from their cell's centre, in cell order
  FixPos *fix;
};

__global__ void k_clear(Box b, Scratch s) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < b.ncell; c += gridDim.x * blockDim.x) {
    s.count[c] = 0;
    s.fill[c] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *s.flag = 0;
}

__device__ __forceinline__ double wrap1(double x, double L) {
  if (x < 0.0) x += L;
  else if (x >= L) x -= L;
  if (x < 0.0 || x >= L) x -= L * floor(x / L);
  return x;
}

__global__ void k_bin(Box b, Scratch s, const double4_32a *q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n) return;
  const double4_32a v = q[i];
  const double x[3] = {wrap1(v.x, b.L[0]), wrap1(v.y, b.L[1]), wrap1(v.z, b.L[2])};
  int c[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (!(x[k] >= 0.0 && x[k] <= b.L[k])) *s.flag = 1;  // not a number
    int ci = (int)(x[k] * b.inv_w[k]);
    c[k] = ci < 0 ? 0 : (ci >= b.nc[k] ? b.nc[k] - 1 : ci);
  }
  const int cc = (c[2] * b.nc[1] + c[1]) * b.nc[0] + c[0];
  s.cell_of[i] = cc;
  atomicAdd(&s.count[cc], 1);
}

// One block of 1024 threads: exclusive scan over all cells, eight a thread as
// two 16-byte loads (77,000 cells: a tenth of the rounds of one each).
constexpr int kScanItems = 8;
__global__ void __launch_bounds__(1024) k_scan(Box b, Scratch s) {
  __shared__ int warp_tot[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int base = 0; base < b.ncell; base += 1024 * kScanItems) {
    const int c0 = base + threadIdx.x * kScanItems;
    int v[kScanItems], sum = 0;
    if (c0 + kScanItems <= b.ncell) {  // the counts start on a 16-byte boundary
#pragma unroll
      for (int k = 0; k < kScanItems; k += 4) {
        const int4 w = *reinterpret_cast<const int4 *>(s.count + c0 + k);
        v[k] = w.x, v[k + 1] = w.y, v[k + 2] = w.z, v[k + 3] = w.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; k++) v[k] = c0 + k < b.ncell ? s.count[c0 + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; k++) sum += v[k];
    int x = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
      int t = warp_tot[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += y;
      }
      warp_tot[lane] = t;
    }
    __syncthreads();
    int excl = carry + (wid ? warp_tot[wid - 1] : 0) + x - sum;
    int at[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      at[k] = excl;
      excl += v[k];
    }
    if (c0 + kScanItems <= b.ncell) {
#pragma unroll
      for (int k = 0; k < kScanItems; k += 4) *reinterpret_cast<int4 *>(s.start + c0 + k) = make_int4(at[k], at[k + 1], at[k + 2], at[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; k++)
        if (c0 + k < b.ncell) s.start[c0 + k] = at[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_tot[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) s.start[b.ncell] = carry;
}

__global__ void k_scatter(Box b, Scratch s, const double4_32a *q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.n) return;
  const int c = s.cell_of[i];
  const int k = s.start[c] + atomicAdd(&s.fill[c], 1);
  s.order[k] = i;
  if (!b.fixed) return;
  const double4_32a v = q[i];
  const double x = wrap1(v.x, b.L[0]), y = wrap1(v.y, b.L[1]), z = wrap1(v.z, b.L[2]);
  const int cx = c % b.nc[0], t = c / b.nc[0], cy = t % b.nc[1], cz = t / b.nc[1];
  s.local[k] = make_float4((float)(x - ((double)cx + 0.5) * b.w[0]), (float)(y - ((double)cy + 0.5) * b.w[1]),
                           (float)(z - ((double)cz + 0.5) * b.w[2]), 0.0f);
  s.fix[k] = fix_position(x, y, z, c);
}

__device__ __forceinline__ double block_sum(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
  __syncthreads();
  return t;
}

// Adds half the energy and virial of the pair (xi, yi, zi), (xj, yj, zj) when it
// lies within the cut-off (observer.cc:5-79; each pair is met from both sides).
__device__ __forceinline__ void pair_sums(const Box &b, double xi, double yi, double zi, double xj, double yj, double zj,
                                          double &pe, double &vir) {
  const double dx = __dsub_rn(xi, xj), dy = __dsub_rn(yi, yj), dz = __dsub_rn(zi, zj);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  if (r2 > b.rc2) return;
  const double r4 = __dmul_rn(r2, r2), r6 = __dmul_rn(r4, r2), r8 = __dmul_rn(r6, r2),
               r10 = __dmul_rn(r8, r2), r12 = __dmul_rn(r10, r2);
  const double e_ij = 4.0 * (1.0 / r12 - 1.0 / r6 + __dmul_rn(b.c2, r2) + b.c0);
  const double df = (__dsub_rn(__dmul_rn(24.0, r6), 48.0) / (__dmul_rn(__dmul_rn(r6, r6), r2)) + b.c2x8) * r2;
  pe += 0.5 * e_ij;
  vir += 0.5 * df;
}

__device__ __forceinline__ double image(double x, int s, double L) { return s ? __dadd_rn(x, s > 0 ? L : -L) : x; }

// Particle i's pairs in double.
__device__ void row_double(const Box &b, const Scratch &s, const double4_32a *q, int i, double &pe, double &vir) {
  const double4_32a qr = q[i];
  const double xi = wrap1(qr.x, b.L[0]), yi = wrap1(qr.y, b.L[1]), zi = wrap1(qr.z, b.L[2]);
  const int c = s.cell_of[i];
  const int cx = c % b.nc[0], t = c / b.nc[0], cy = t % b.nc[1], cz = t / b.nc[1];
  for (int oz = -1; oz <= 1; oz++) {
    int nz = cz + oz, sz = 0;
    if (nz < 0) { nz += b.nc[2]; sz = -1; } else if (nz >= b.nc[2]) { nz -= b.nc[2]; sz = 1; }
    for (int oy = -1; oy <= 1; oy++) {
      int ny = cy + oy, sy = 0;
      if (ny < 0) { ny += b.nc[1]; sy = -1; } else if (ny >= b.nc[1]) { ny -= b.nc[1]; sy = 1; }
      for (int ox = -1; ox <= 1; ox++) {
        int nx = cx + ox, sx = 0;
        if (nx < 0) { nx += b.nc[0]; sx = -1; } else if (nx >= b.nc[0]) { nx -= b.nc[0]; sx = 1; }
        const int cc = (nz * b.nc[1] + ny) * b.nc[0] + nx;
        const int a = s.start[cc], e = s.start[cc + 1];
        for (int k = a; k < e; k++) {
          const int j = s.order[k];
          if (j == i && !(sx | sy | sz)) continue;
          const double4_32a qj = q[j];
          pair_sums(b, xi, yi, zi, image(wrap1(qj.x, b.L[0]), sx, b.L[0]), image(wrap1(qj.y, b.L[1]), sy, b.L[1]),
                    image(wrap1(qj.z, b.L[2]), sz, b.L[2]), pe, vir);
        }
      }
    }
  }
}

// The observers in double, a thread per particle: cut-offs outside the fixed-point
// range, and boxes of less than kSparse particles a cell, where most warps of
// k_observe find nothing.  A whole call, this / that, us: 20,000 particles at 0.08
// a cell 150 / 204, at 0.16 144 / 159, at 0.34 170 / 139; 5,000 at 0.08 103 / 118, at 0.17 113
// / 105; 50,000 at 0.32 245 / 207.
constexpr double kSparse = 0.16;
__global__ void __launch_bounds__(kThreads) k_observe_rows(Box b, Scratch s, const double4_32a *q, const double4_32a *p) {
  __shared__ double sh[kThreads / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ke = 0.0, pe = 0.0, vir = 0.0;
  if (i < b.n) {
    const double4_32a pi = p[i];
    ke = 0.5 * pi.x * pi.x + 0.5 * pi.y * pi.y + 0.5 * pi.z * pi.z + 0.5 * pi.w * pi.w;
    row_double(b, s, q, i, pe, vir);
  }
  const double ta = block_sum(ke, sh), tb = block_sum(pe, sh), tc = block_sum(vir, sh);
  if (threadIdx.x == 0) {
    s.partial[3 * blockIdx.x + 0] = ta;
    s.partial[3 * blockIdx.x + 1] = tb;
    s.partial[3 * blockIdx.x + 2] = tc;
  }
}

// A lane's pairs in fixed point: the sums of mdg_fixed.cu's observers, added to
// the double ones at each new row and before they could overflow (361 pairs).
struct PairSink {
  const Box &b;
  const Scratch &s;
  const double4_32a *q;
  double pe, vir;
  FixPos own;
  int slot, m;
  uint64_t sz, szz, sr;

  __device__ __forceinline__ void flush() {
    const double u = 1.0 / (double)(1ull << 54), half = 0.5 * m;
    const double z = ((double)sz + half) * u, zz = ((double)szz + half) * u;
    const double r = b.c2 * (((double)sr + half) * (1.0 / (double)(1ull << 51)));
    // half of each pair's share: it is met from both sides
    pe += 2.0 * ((zz - z) + (r + b.c0 * (double)m));
    vir += 12.0 * (z - 2.0 * zz) + 4.0 * r;
    sz = szz = sr = 0;
    m = 0;
  }
  __device__ __forceinline__ void start(int i, int) {
    if (m) flush();
    slot = i;
    own = s.fix[i];
  }
  __device__ __forceinline__ void put(uint32_t e) {
    const int j = entry_slot(e);
    const FixPos x = ld_fix<false>(s.fix + j);
    int dx = x.x - own.x, dy = x.y - own.y, dz = x.z - own.z;
    float lx = x.lx - own.lx, ly = x.ly - own.ly, lz = x.lz - own.lz;
    const uint32_t ix = e & 3u, iy = (e >> 2) & 3u, iz = (e >> 4) & 3u;  // image step + 1
    if (ix != 1u) { dx += ix ? b.fx_L[0] : -b.fx_L[0]; lx += ix ? b.fx_l[0] : -b.fx_l[0]; }
    if (iy != 1u) { dy += iy ? b.fx_L[1] : -b.fx_L[1]; ly += iy ? b.fx_l[1] : -b.fx_l[1]; }
    if (iz != 1u) { dz += iz ? b.fx_L[2] : -b.fx_L[2]; lz += iz ? b.fx_l[2] : -b.fx_l[2]; }
    const uint64_t R = fix_r2(fix_sep(dx, dy, dz, lx, ly, lz));
    if (R > b.fx_rc2) return;
    if (fix_hi(R) < b.fx_near) {
      const double4_32a qi = q[s.order[slot]], qj = q[s.order[j]];
      pair_sums(b, wrap1(qi.x, b.L[0]), wrap1(qi.y, b.L[1]), wrap1(qi.z, b.L[2]),
                image(wrap1(qj.x, b.L[0]), (int)ix - 1, b.L[0]), image(wrap1(qj.y, b.L[1]), (int)iy - 1, b.L[1]),
                image(wrap1(qj.z, b.L[2]), (int)iz - 1, b.L[2]), pe, vir);
      return;
    }
    uint64_t y2, z;
    fix_powers(fix_recip(R), y2, z);
    const uint64_t zz = fix_sqrhi(z);  // 2^-58
    sz += z >> 7;
    szz += zz >> 4;
    sr += R >> 7;  // 2^-51
    if (++m == 360) flush();
  }
};

// Observers of observer.cc:5-79 over every image pair within the cut-off.
// A whole call, density 0.6, cut-off 2.5: 1,000 particles 1,191 -> 61 us, 8,000
// 926 -> 62, 60,000 2,791 -> 152, 600,000 21,096 -> 792 against a thread per
// particle with every candidate measured in double, which kept the FP64 pipe
// busy with candidates of which a sixth are pairs (and with three divisions a
// pair).  Now bound as the list build is, by issue; small calls by the six launches.
constexpr int kWarps = kThreads / 32;
__global__ void __launch_bounds__(kThreads) k_observe(Box b, Scratch s, const double4_32a *q, const double4_32a *p, int split) {
  __shared__ double sh[kThreads / 32];
  __shared__ CellRows<kTileChunks> s_rows[kWarps];
  double ke = 0.0;
  PairSink sink{b, s, q, 0.0, 0.0, {}, 0, 0, 0, 0, 0};
  const bool fixed = b.fixed && *s.flag == 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < b.n; i += gridDim.x * blockDim.x) {
    const double4_32a pi = p[i];
    ke += 0.5 * pi.x * pi.x + 0.5 * pi.y * pi.y + 0.5 * pi.z * pi.z + 0.5 * pi.w * pi.w;
    if (!fixed) row_double(b, s, q, i, sink.pe, sink.vir);
  }
  const int warp = threadIdx.x >> 5;
  if (fixed)
    for (int item = blockIdx.x * kWarps + warp; item < b.ncell * split; item += gridDim.x * kWarps) {
      const int c = item / split, part = item % split;
      const int lo = s.start[c], cnt = s.start[c + 1] - lo;
      const int from = lo + (int)((long long)cnt * part / split), to = lo + (int)((long long)cnt * (part + 1) / split);
      if (from == to) continue;
      const int cx = c % b.nc[0], t = c / b.nc[0], cy = t % b.nc[1], cz = t / b.nc[1];
      cell_rows(
          s_rows[warp], s.local, lo, from, to, b.hi, b.hi, INT_MAX,
          [&](int l, int &first, int &count, float3 &shift, uint32_t &code) {
            const int ox = l % 3 - 1, oy = l / 3 % 3 - 1, oz = l / 9 - 1;
            int sx, sy, sz;
            const int nx = wrap_cell(cx, ox, b.nc[0], sx), ny = wrap_cell(cy, oy, b.nc[1], sy), nz = wrap_cell(cz, oz, b.nc[2], sz);
            shift = make_float3((float)ox * b.w32[0], (float)oy * b.w32[1], (float)oz * b.w32[2]);
            code = entry_pack(0, sx, sy, sz);
            const int cc = (nz * b.nc[1] + ny) * b.nc[0] + nx;
            first = s.start[cc];
            count = s.start[cc + 1] - first;
          },
          [&](int, int, int) { return true; }, sink, [](int, int) {});
    }
  if (sink.m) sink.flush();
  const double ta = block_sum(ke, sh), tb = block_sum(sink.pe, sh), tc = block_sum(sink.vir, sh);
  if (threadIdx.x == 0) {
    s.partial[3 * blockIdx.x + 0] = ta;
    s.partial[3 * blockIdx.x + 1] = tb;
    s.partial[3 * blockIdx.x + 2] = tc;
  }
}

__global__ void k_final(Scratch s, int nparts, double *out) {
  __shared__ double sh[32];
  double a = 0.0, b2 = 0.0, c = 0.0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
    a += s.partial[3 * k + 0];
    b2 += s.partial[3 * k + 1];
    c += s.partial[3 * k + 2];
  }
  const double ta = block_sum(a, sh), tb = block_sum(b2, sh), tc = block_sum(c, sh);
  if (threadIdx.x == 0) {
    out[0] = ta;
    out[1] = tb;
    out[2] = tc / 3.0;
  }
}

std::mutex g_mu;
unsigned long long *g_addr[kMaxDevices] = {};

// Device address of g_scratch on the current device, looked up on the first call.
cudaError_t scratch_address(int dev, unsigned long long **out) {
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_addr[dev]) {
    void *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_scratch);
    if (e != cudaSuccess) return e;
    g_addr[dev] = static_cast<unsigned long long *>(ptr);
  }
  *out = g_addr[dev];
  return cudaSuccess;
}

}  // namespace noalloc
}  // namespace mdg

extern "C" int mdg_observe_noalloc(const double *q4_dev, const double *p4_dev, int32_t n, const double box[3],
                                   double cutoff, double *out3_dev, void *stream) {
  using namespace mdg::noalloc;
  if (!q4_dev || !p4_dev || !box || !out3_dev || n <= 0 || !(cutoff > 0.0)) return MDG_ERR_INVALID;
  // the state is read as 32-byte vectors, the sums written as doubles
  if ((((uintptr_t)q4_dev | (uintptr_t)p4_dev) & 31u) != 0 || ((uintptr_t)out3_dev & 7u) != 0) {
    fprintf(stderr, "mdg_observe_noalloc: q4_dev and p4_dev must be 32-byte aligned, out3_dev 8-byte aligned\n");
    return MDG_ERR_INVALID;
  }
  if (n > kMaxParticles) {
    fprintf(stderr, "mdg_observe_noalloc: %d particles exceed the fixed maximum of %d\n", n, kMaxParticles);
    return MDG_ERR_CAPACITY;
  }
  Box b;
  long long ncell = 1;
  for (int k = 0; k < 3; k++) {
    if (!(box[k] > 2.0 * cutoff) || !std::isfinite(box[k])) return MDG_ERR_INVALID;
    // the cell count is bounded before any conversion or product can overflow
    const double ratio = box[k] / cutoff;
    if (!(ratio <= (double)kMaxCells)) {
      fprintf(stderr, "mdg_observe_noalloc: box side %g / cutoff %g exceeds the fixed maximum of %d cells\n",
              box[k], cutoff, kMaxCells);
      return MDG_ERR_CAPACITY;
    }
    int nc = (int)ratio;
    while (nc > 0 && box[k] / (double)nc < cutoff * (1.0 + 1e-12)) nc--;
    if (nc < 2) return MDG_ERR_INVALID;
    b.L[k] = box[k];
    b.nc[k] = nc;
    b.inv_w[k] = 1.0 / (box[k] / (double)nc);
    if (ncell > kMaxCells / nc) {
      fprintf(stderr, "mdg_observe_noalloc: more cells than the fixed maximum of %d\n", kMaxCells);
      return MDG_ERR_CAPACITY;
    }
    ncell *= nc;
  }
  if (ncell > kMaxCells) {
    fprintf(stderr, "mdg_observe_noalloc: %lld cells exceed the fixed maximum of %d\n", ncell, kMaxCells);
    return MDG_ERR_CAPACITY;
  }
  b.ncell = (int)ncell;
  b.n = n;
  b.rc2 = cutoff * cutoff;
  const double s2 = 1.0 / (cutoff * cutoff);  // Variables::Variables (variables.cc:16-28)
  const double s6 = s2 * s2 * s2, s8 = s6 * s2, s12 = s6 * s6, s14 = s12 * s2;
  b.c2 = 6.0 * s14 - 3.0 * s8;
  b.c0 = -s12 + s6 - b.c2 / s2;
  b.c2x8 = b.c2 * 8.0;
  b.fixed = cutoff >= 1.0 && cutoff < 3.9 && n >= kSparse * b.ncell;
  b.fx_rc2 = b.fixed ? (uint64_t)std::ldexp(b.rc2, mdg::kFixR2Bits) : 0;
  b.fx_near = (uint32_t)(mdg::kFixNear * (double)(1u << (mdg::kFixR2Bits - 32))) + 1;
  for (int k = 0; k < 3; k++) {
    const int64_t L = mdg::fix_from_double(b.L[k]);
    b.fx_L[k] = mdg::fix_shi(L);
    b.fx_l[k] = mdg::fix_rest(L);
    b.w[k] = b.L[k] / (double)b.nc[k];
    b.w32[k] = (float)b.w[k];
  }
  // float positions from a cell's centre are within 1e-6: every pair within
  // the cut-off passes
  b.hi = (float)(b.rc2 + 1e-3);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return MDG_ERR_CUDA;
  unsigned long long *base = nullptr;
  if (scratch_address(dev, &base) != cudaSuccess) return MDG_ERR_CUDA;
  Scratch s;
  s.count = reinterpret_cast<int *>(base + kOffCount);
  s.start = reinterpret_cast<int *>(base + kOffStart);
  s.fill = reinterpret_cast<int *>(base + kOffFill);
  s.cell_of = reinterpret_cast<int *>(base + kOffCellOf);
  s.order = reinterpret_cast<int *>(base + kOffOrder);
  s.partial = reinterpret_cast<double *>(base + kOffPartial);
  s.flag = reinterpret_cast<int *>(base + kOffFlag);
  s.local = reinterpret_cast<float4 *>(base + kOffLocal);
  s.fix = reinterpret_cast<mdg::FixPos *>(base + kOffFix);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = (n + kThreads - 1) / kThreads;
  const auto *q = reinterpret_cast<const double4_32a *>(q4_dev);
  const auto *p = reinterpret_cast<const double4_32a *>(p4_dev);
  k_clear<<<(b.ncell + 255) / 256, 256, 0, st>>>(b, s);
  k_bin<<<grid, kThreads, 0, st>>>(b, s, q);
  k_scan<<<1, 1024, 0, st>>>(b, s);
  k_scatter<<<grid, kThreads, 0, st>>>(b, s, q);
  int blocks = grid;
  if (b.fixed) {
    // few cells: two or four warps each, as the list build
    const int split = b.ncell < 1500 ? 4 : (b.ncell < 12000 ? 2 : 1);
    const int warps = (b.ncell * split + kWarps - 1) / kWarps;
    const int most = warps > grid ? warps : grid;  // blocks of kThreads particles where the double sums run
    blocks = most < kMaxBlocks ? most : kMaxBlocks;
    k_observe<<<blocks, kThreads, 0, st>>>(b, s, q, p, split);
  } else {
    k_observe_rows<<<grid, kThreads, 0, st>>>(b, s, q, p);
  }
  k_final<<<1, 1024, 0, st>>>(s, blocks, out3_dev);
  return cudaGetLastError() == cudaSuccess ? MDG_OK : MDG_ERR_CUDA;
}

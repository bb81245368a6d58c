// Rows of the pair list, shared by the single box and the batch: the
// candidates of the 27 stencil cells tested in float from home-cell-local
// positions, the few inside the float band by the caller's exact test.
//
// The tests' results are kept as bit masks, and the accepted candidates, a
// seventh of them, are written from the masks: appending inside the test loop
// cost every candidate the append's instructions, since some lane of the
// warp almost always accepts (25 instructions a candidate).
#pragma once
#include "mdg_internal.cuh"

namespace mdg {

// Wraps the cell coordinate c + o; s the image step (-1, 0, 1).
__device__ __forceinline__ int wrap_cell(int c, int o, int nc, int &s) {
  int v = c + o;
  s = 0;
  if (v < 0) { v += nc; s = -1; }
  else if (v >= nc) { v -= nc; s = 1; }
  return v;
}

// Masks of the (at most 32) candidates qf[j0 .. j0 + m): `in` those whose r^2
// is at most hi, `sure` those below lo.
__device__ __forceinline__ void chunk_masks(const float4 *__restrict__ qf, int j0, int m, float fx, float fy, float fz,
                                            float lo, float hi, uint32_t &in, uint32_t &sure) {
  in = sure = 0u;
  const int last = j0 + m - 1;
  for (int u = 0; u < m; u += 4) {
    float4 f[4];
#pragma unroll
    for (int v = 0; v < 4; v++) f[v] = qf[min(j0 + u + v, last)];
    uint32_t a = 0u, b = 0u;
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const float ex = f[v].x + fx, ey = f[v].y + fy, ez = f[v].z + fz;
      const float r2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
      if (r2 <= hi) a |= 1u << v;
      if (r2 < lo) b |= 1u << v;
    }
    in |= a << u;
    sure |= b << u;
  }
  const uint32_t valid = m >= 32 ? 0xffffffffu : (1u << m) - 1u;
  in &= valid;
  sure &= valid;
}

// Exact acceptance of a candidate in the float band: the reference's image
// and rounding order (mdunit.cc:167, meshlist.cc:262-266).
__device__ __forceinline__ bool image_within(const double4_32a &qi, const double4_32a &qj, const double *L, int sx, int sy, int sz,
                                             double sl2) {
  const double xj = sx ? __dadd_rn(qj.x, sx > 0 ? L[0] : -L[0]) : qj.x;
  const double yj = sy ? __dadd_rn(qj.y, sy > 0 ? L[1] : -L[1]) : qj.y;
  const double zj = sz ? __dadd_rn(qj.z, sz > 0 ? L[2] : -L[2]) : qj.z;
  const double dx = __dsub_rn(qi.x, xj), dy = __dsub_rn(qi.y, yj), dz = __dsub_rn(qi.z, zj);
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return r2 <= sl2;
}

// The rows of a home cell's particles by one warp.  The 27 stencil cells'
// candidates are laid side by side and taken 32 at a time, one a lane; each
// home particle's position is then a broadcast, the test of 32 candidates six
// float operations and a vote, and the votes are kept as bit masks.  The
// entries are written from the masks by one lane per home particle (two or
// four where they are at most 16 or 8), so neighbouring slots' entries go out together.
// Bound by issue (76 % of the slots) and the float pipe; 372 warp instructions
// a particle at 1,000,188 atoms, density 0.5: 160 the tests, 100 the entries.
// Against a thread per particle with its own candidates (436 instructions, and
// loads from as many places as lanes): forced rebuild of 4M atoms 3.2 -> 2.2 ms,
// of 1M 0.80 -> 0.61; 50,000 rebuilding particles of a batch 80 us with nine lanes
// a particle, 64 with one warp a cell.  Tried: two home particles per packed
// float instruction (moves ate the gain), the next candidates' loads in flight
// during the tests (no faster: the other warps cover them).
// TILE: candidates whose masks are held at a time, in 32s.
constexpr int kTileChunks = 16;
template <int TILE>
struct CellRows {
  float4 home[32];  // positions relative to the home cell's centre
  float4 cell[32];  // a stencil cell's shift, and the offset from its candidates' places to their slots
  uint32_t code[32];
  uint32_t mask[TILE][32];   // [chunk][home particle]
  uint32_t entry[TILE][32];  // [chunk][candidate]
};

// Row entry k of slot i at row + i + k * stride.
struct RowSink {
  uint32_t *row;
  size_t stride;
  uint32_t *out;
  __device__ __forceinline__ void start(int i, int k) { out = row + i + (size_t)k * stride; }
  __device__ __forceinline__ void put(uint32_t e) {
    *out = e;
    out += stride;
  }
};

// Home slots a .. b - 1 of qf, of the cell that starts at a0.  stencil(l, first, count, shift, code): stencil cell l = 0 .. 26 in
// row order; exact(i, j, l): the exact test of a candidate in the float band;
// a lane's sink takes its entries: start(slot, k) ahead of entries k, k + 1, ...
// of a slot, put(entry); cap entries a row are kept; done(slot, count).
template <int TILE, class Stencil, class Exact, class Sink, class Done>
__device__ __forceinline__ void cell_rows(CellRows<TILE> &m, const float4 *__restrict__ qf, int a0, int a, int b, float lo, float hi,
                                          int cap, Stencil &&stencil, Exact &&exact, Sink &&sink, Done &&done) {
  const int lane = threadIdx.x & 31;
  const uint32_t all = 0xffffffffu;
  const float mid = 0.5f * (lo + hi), half = 0.5f * (hi - lo);
  int first = 0, count = 0;
  float3 shift = make_float3(0.f, 0.f, 0.f);
  uint32_t code = 0u;
  if (lane < 27) stencil(lane, first, count, shift, code);
  int end = count;  // of the cell's candidates in the sequence
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(all, end, o);
    if (lane >= o) end += v;
  }
  const int total = __shfl_sync(all, end, 31);
  const int self0 = __shfl_sync(all, end - count, 13);  // place of slot a0
  m.cell[lane] = make_float4(shift.x, shift.y, shift.z, __int_as_float(first - (end - count)));
  m.code[lane] = code;
  for (int h0 = a; h0 < b; h0 += 32) {
    const int H = min(b - h0, 32);
    __syncwarp();
    m.home[lane] = lane < H ? qf[h0 + lane] : make_float4(-1e15f, 0.f, 0.f, 0.f);
    __syncwarp();
    // home particle and chunks of this lane's writes
    const int wide = H <= 8 ? 8 : (H <= 16 ? 16 : 32), parts = 32 / wide;
    const int h = lane & (wide - 1), part = lane / wide;
    int cnt = 0;
    for (int t0 = 0; t0 < total; t0 += 32 * TILE) {
      const int chunks = min((total - t0 + 31) >> 5, TILE);
      for (int c = 0; c < chunks; c++) {
        const int f = t0 + 32 * c + 31 - lane;  // the first candidate at the top bit
        int k = 0;  // cells that end at or before f
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
          if (__shfl_sync(all, end, k + s - 1) <= f) k += s;
        const float4 cell = m.cell[k];
        const int j = f + __float_as_int(cell.w);
        float x = 1e15f, y = 0.f, z = 0.f;
        if (f < total) {
          const float4 q = qf[j];
          x = q.x + cell.x;
          y = q.y + cell.y;
          z = q.z + cell.z;
        }
        m.entry[c][lane] = ((uint32_t)j << kCodeBits) | m.code[k];
        // r^2 of home particle g, relative to the middle of the band
        auto test = [&](int g) {
          const float4 o = m.home[g];
          const float ex = x - o.x, ey = y - o.y, ez = z - o.z;
          return fmaf(ez, ez, fmaf(ey, ey, fmaf(ex, ex, -mid)));
        };
        float nearest = 1e30f;
#pragma unroll 2
        for (int g = 0; g < H; g += 2) {
          const float t0 = test(g), t1 = test(g + 1);
          nearest = fminf(nearest, fminf(fabsf(t0), fabsf(t1)));
          const uint32_t in0 = __ballot_sync(all, t0 <= half), in1 = __ballot_sync(all, t1 <= half);
          *reinterpret_cast<uint2 *>(&m.mask[c][g]) = make_uint2(in0, in1);
        }
        if (__any_sync(all, nearest <= half)) {
          __syncwarp();  // the masks above are written
          for (int g = 0; g < H; g++) {
            const float t = test(g);
            const uint32_t in = __ballot_sync(all, t < -half || (t <= half && exact(h0 + g, j, k)));
            if (lane == 0) m.mask[c][g] = in;
          }
        }
      }
      __syncwarp();
      // the particle itself
      const int self = self0 + (h0 - a0) + lane - t0;
      if (lane < H && self >= 0 && self < 32 * chunks) m.mask[self >> 5][lane] &= ~(0x80000000u >> (self & 31));
      __syncwarp();
      const int c0 = part * chunks / parts, c1 = (part + 1) * chunks / parts;
      int mine = 0, w = cnt;
      if (h < H)
        for (int c = c0; c < c1; c++) mine += __popc(m.mask[c][h]);
      for (int q = 0; q < parts; q++) {
        const int v = __shfl_sync(all, mine, q * wide + h);
        if (q < part) w += v;
        cnt += v;
      }
      mine = min(mine, cap - w);
      if (mine > 0) sink.start(h0 + h, w);
      const uint32_t *word = &m.mask[c0][h], *entry = m.entry[c0];
      uint32_t bits = mine > 0 ? *word : 0u;
      while (mine > 0) {
        if (bits == 0u) {
          word += 32;
          entry += 32;
          bits = *word;
        }
        if (bits != 0u) {
          const int u = 31 - __clz(bits);
          sink.put(entry[u]);
          bits ^= 1u << u;
          mine--;
        }
      }
      __syncwarp();
    }
    if (part == 0 && h < H) done(h0 + h, cnt);
  }
}

}  // namespace mdg

// Device functions of a rebuild, shared by its kernels (mdg_cells.cu,
// mdg_list.cu) and the resident kernel of small boxes.
#pragma once
#include "mdg_build.cuh"

namespace mdg {

// Step-boundary position of slot i in the mixed form from the home-cell-local
// mid-step position: the centre of the home cell plus (q_mid - p dt/2), the
// inverse of the step's last half-drift.
__device__ __forceinline__ double4_32a end_from_mid(const Geom &g, const Dev &d, int i, int mid) {
  const double4_32a u = d.q_mid[mid][i], p = d.p[i];
  int cx, cy, cz;
  cell_unkey(d.cell[i], cx, cy, cz);
  double4_32a q = u;
  q.x = cell_centre(g, 0, cx) + fma(-p.x, g.dt2, u.x);
  q.y = cell_centre(g, 1, cy) + fma(-p.y, g.dt2, u.y);
  q.z = cell_centre(g, 2, cz) + fma(-p.z, g.dt2, u.z);
  return q;
}

// Wraps slot i's q_end into the box (one +-L per component), bins it and counts
// it; a non-finite or escaped coordinate halts the run.
__device__ __forceinline__ void wrap_bin_one(const Geom &g, const Dev &d, int i, bool from_mid, int mid) {
  double4_32a q = from_mid ? end_from_mid(g, d, i, mid) : d.q_end[i];
  double x[3] = {q.x, q.y, q.z};
  int c[3];
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double v = x[k];
    if (v < 0.0) v += g.L[k];
    else if (v > g.L[k]) v -= g.L[k];
    if (!(v >= 0.0 && v <= g.L[k])) bad = true;  // also catches NaN
    x[k] = v;
    int ci = bad ? 0 : (int)(v * g.inv_w[k]);
    c[k] = ci < 0 ? 0 : (ci >= g.nc[k] ? g.nc[k] - 1 : ci);
  }
  if (bad) {
    halt_with(d.flags, kHaltBadState);
    atomicMin(&d.flags->bad_slot, i);
    return;
  }
  q.x = x[0]; q.y = x[1]; q.z = x[2];
  d.q_end[i] = q;
  d.cell[i] = cell_key(c[0], c[1], c[2]);
  atomicAdd(&d.cell_count[cell_rank(g, c[0], c[1], c[2])], 1);
}

// Sorted particle k of a new list (q and p in registers: loaded one by one
// between the stores they cost k_finalize 13 us of 46 at 1M): the state back in place, the build
// positions, and the positions of the next force evaluation in q_mid[q_mid_dst].
template <bool LOCAL, bool FIXED>
__device__ __forceinline__ void finalize_one(const Geom &g, const Dev &d, int k, double4_32a q, double4_32a p, int id,
                                             int c, int q_mid_dst) {
  d.q_end[k] = q;
  d.id[k] = id;
  d.cell[k] = c;
  d.inv[id] = k;
  int cx, cy, cz;
  cell_unkey(c, cx, cy, cz);
  const float cw = __int_as_float(c);
  const double ox = cell_centre(g, 0, cx), oy = cell_centre(g, 1, cy), oz = cell_centre(g, 2, cz);
  const float4 lb = make_float4((float)(q.x - ox), (float)(q.y - oy), (float)(q.z - oz), cw);
  d.qf[k] = lb;
  double4_32a m = q;
  if (LOCAL) {
    m.x = __dadd_rn(q.x - ox, __dmul_rn(p.x, g.dt2));
    m.y = __dadd_rn(q.y - oy, __dmul_rn(p.y, g.dt2));
    m.z = __dadd_rn(q.z - oz, __dmul_rn(p.z, g.dt2));
    // the build reference (for the rebuild test) in q_mid's padding word, and
    // the same position as the prune reference in p's until the step's
    // re-selection records its own
    m.w = pack_ref(g, lb.x, lb.y, lb.z);
    p.w = m.w;
    d.q_mid[q_mid_dst][k] = m;
    d.p[k] = p;
    d.loc[q_mid_dst][k] = make_float4((float)m.x, (float)m.y, (float)m.z, cw);
  } else {
    d.p[k] = p;
    d.q_build[k] = q;
    m.x = __dadd_rn(q.x, __dmul_rn(p.x, g.dt2));
    m.y = __dadd_rn(q.y, __dmul_rn(p.y, g.dt2));
    m.z = __dadd_rn(q.z, __dmul_rn(p.z, g.dt2));
    d.q_mid[q_mid_dst][k] = m;
    if (FIXED) {
      d.xq[q_mid_dst][k] = fix_position(m.x, m.y, m.z, c);
      const FixPos b = fix_position(q.x, q.y, q.z, c);
      d.xb[k] = make_int4(b.x, b.y, b.z, c);
      // the first half-drift must stay inside the modulus's guard too
      const double far = fmax(fmax(fabs(p.x), fabs(p.y)), fabs(p.z)) * g.dt2;
      if (!(far <= (double)g.fx_guard)) d.flags->fx_wide[q_mid_dst] = 1;
    } else {
      d.loc[q_mid_dst][k] = make_float4((float)(m.x - ox), (float)(m.y - oy), (float)(m.z - oz), cw);
    }
  }
}

constexpr int kRowLanes = 9;

// The length `cnt` of slot i's row, which may exceed the capacity: kept, or the
// run halted; the kept entries added to `pairs`, the longest row to `longest`.
__device__ __forceinline__ void keep_row_length(const Geom &g, const Dev &d, int i, int cnt, int &pairs, int &longest) {
  const int kept = min(cnt, g.list_cap);
  d.ncount[i] = kept;
  if (cnt > g.list_cap) {
    atomicMax(&d.flags->overflow_max, cnt);
    halt_with(d.flags, kHaltOverflow);
  }
  pairs += kept;
  longest = max(longest, cnt);
}

// The row of slot i by kRowLanes neighbouring lanes of a warp (`base` the first
// of them), one for each (y, z) row of three stencil cells: a row's candidates
// then take a ninth of the time one after the other, which is what a small box
// waits for.  The entries are in stencil order (z, y, x), candidates ascending, as
// cell_rows writes them.  Every lane of the warp calls it; returns the row's
// length, which may exceed the capacity.
__device__ __forceinline__ int build_slot_row(const Geom &g, const Dev &d, int i, bool active, int lane, int base) {
  DevFlags *f = d.flags;
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
        if (!image_within(d.q_end[i], d.q_end[j0 + u], g.L, sx, sy, sz, g.sl2)) in &= ~(1u << u);
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
  int before = 0, total = 0;
#pragma unroll
  for (int l = 0; l < kRowLanes; l++) {
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
  return total;
}

// The rows of part `part` of `split` of cell `home`'s particles, by a warp: the kept
// entries added to this lane's `pairs`, its longest row to `longest`.
template <int TILE>
__device__ __forceinline__ void build_cell_rows(const Geom &g, const Dev &d, CellRows<TILE> &rows, int home, int part, int split,
                                                int &pairs, int &longest) {
  DevFlags *f = d.flags;
  const int cap = g.list_cap;
  int a = d.cell_start[home], b = d.cell_start[home + 1];
  if (!MDG_IN_RANGE(f, kCheckBuildRange, b, g.n + 1) || !MDG_IN_RANGE(f, kCheckBuildRange, a, b + 1)) a = b = 0;
  const int from = a + (b - a) * part / split, to = a + (b - a) * (part + 1) / split;
  if (from >= to) return;
  int cx, cy, cz;
  cell_unpack(d.qf[a].w, cx, cy, cz);
  cell_rows(
      rows, d.qf, a, from, to, g.acc_lo, g.acc_hi, cap,
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
      [&](int i, int cnt) { keep_row_length(g, d, i, cnt, pairs, longest); });
}

}  // namespace mdg

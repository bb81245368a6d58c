// Device functions of the fixed-point form (mdg_fixed.cu), shared with the
// resident kernel of small boxes.
#pragma once
#include "mdg_fixed.cuh"
#include "mdg_step.cuh"

namespace mdg {

// List rows requested into L2 this many entries ahead with one thread per
// particle (1.073 ms; 24 ahead 1.083, none 1.090; observers 1.35 against 1.53).
constexpr int kRowsAhead = 12;
// Pairs per trip of the row walk (2: no moves for the entries in flight;
// 1.073 ms, 1 pair 1.095, 4 pairs 1.130).
constexpr int kPairsPerTrip = 2;
// Pairs a lane of the resident kernel works on together (FP64 864 / 16,384 /
// 70,304 atoms, us per step: 2 8.1 / 17.8 / 35.9, 3 8.4 / 18.7 / 36.4, 4 8.9 / 19.3 / 37.3).
constexpr int kInFlight = 2;

// Lanes per particle for n particles outside the resident kernel.  A row's
// pairs take about half a microsecond one after the other, so a GPU that one
// thread per particle does not fill (152 SMs x 24 warps) is better used by
// several.  Step kernel with 1 / 2 / 8 / 32 lanes, us (density 0.6): 864 atoms 29.9 /
// 23.9 / 19.0 / 17.5, 2,400 31.3 / 24.7 / 18.9 / 18.8, 5,000 31.4 / 24.7 / 19.9 / 25.7, 9,700
// 31.8 / 24.9 / 20.4 / 32.0, 16,000 31.8 / 25.3 / 25.9, 38,900 34.4 / 29.9 / 38.5, 64,000
// 45.5 / 43.5, 110,000 57.8 / 57.8 (two lanes still gain a little where the line puts
// one; by 256,000 they cost 187 for 141).  The lines are 16, 64 and 256 particles
// per SM of 152.
inline int fx_lanes(int n) { return n < 2432 ? 32 : (n < 9728 ? 8 : (n < 38912 ? 2 : 1)); }

// Image shifts of a particle at the box faces: per axis the step code (after
// entry ^ 0x15: 1 = step -1, 3 = step +1) that crosses the face, 2 = none,
// and the shift of the partner, -L or +L.
struct Faces {
  uint32_t kx, ky, kz;
  int sx, sy, sz;
  float lx, ly, lz;
};

__device__ __forceinline__ Faces faces_of(const Geom &g, const CellPos &cp) {
  Faces f;
  f.kx = cp.cx == 0 ? 1u : (cp.cx == g.nc[0] - 1 ? 3u : 2u);
  f.ky = (cp.cy == 0 ? 1u : (cp.cy == g.nc[1] - 1 ? 3u : 2u)) << 2;
  f.kz = (cp.cz == 0 ? 1u : (cp.cz == g.nc[2] - 1 ? 3u : 2u)) << 4;
  f.sx = cp.cx == 0 ? -g.fx_L[0] : g.fx_L[0];
  f.sy = cp.cy == 0 ? -g.fx_L[1] : g.fx_L[1];
  f.sz = cp.cz == 0 ? -g.fx_L[2] : g.fx_L[2];
  f.lx = cp.cx == 0 ? -g.fx_l[0] : g.fx_l[0];
  f.ly = cp.cy == 0 ? -g.fx_l[1] : g.fx_l[1];
  f.lz = cp.cz == 0 ? -g.fx_l[2] : g.fx_l[2];
  return f;
}

// Walks every LANES-th entry of the row of particle i from `lane` on: hands
// pair(valid, e, sep, R) the separation and R = r^2; where it returns true,
// close(e) follows.  One position and two entries are in flight (COH:
// kInFlight of each).  ALL: every thread of the warp calls pair the same
// number of times (for ballots), with valid = false past its row.
template <bool EDGE, int LANES, bool ALL, int SITE, bool COH, class Pair, class Close>
__device__ __forceinline__ void walk_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                           const FixPos &own, int i, const CellPos &cp,
                                           const uint32_t *__restrict__ list, int cnt, int lane, Pair &&pair, Close &&close) {
  Faces fc;
  if (EDGE) fc = faces_of(g, cp);
  const uint32_t *row = list + i;
  const size_t stride = (size_t)g.stride;
  const uint32_t none = entry_pack(i, 0, 0, 0);  // a valid address past the row's end
  auto entry = [&](int k) { return k < cnt ? ld_ro<COH>(row + (size_t)k * stride) : none; };
  int end = cnt;
  if (ALL) end = __reduce_max_sync(0xffffffffu, cnt);
  auto sep_of = [&](uint32_t e, const FixPos &q) {
    int dx = q.x - own.x, dy = q.y - own.y, dz = q.z - own.z;
    float lx = q.lx - own.lx, ly = q.ly - own.ly, lz = q.lz - own.lz;
    if (EDGE) {
      const uint32_t s = e ^ 0x15u;
      if ((s & 0x03u) == fc.kx) { dx += fc.sx; lx += fc.lx; }
      if ((s & 0x0Cu) == fc.ky) { dy += fc.sy; ly += fc.ly; }
      if ((s & 0x30u) == fc.kz) { dz += fc.sz; lz += fc.lz; }
    }
    return fix_sep(dx, dy, dz, lx, ly, lz);
  };
  if (COH) {
    // the resident kernel waits for each round of loads: kInFlight at a time
    uint32_t en[kInFlight];
#pragma unroll
    for (int u = 0; u < kInFlight; u++) en[u] = entry(lane + u * LANES);
    for (int k = lane; k - lane < end && (ALL || k < cnt); k += kInFlight * LANES) {
      uint32_t e[kInFlight];
      FixPos q[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; u++) {
        e[u] = en[u];
        if (!MDG_IN_RANGE(d.flags, SITE, entry_slot(e[u]), g.n)) e[u] = none;
        q[u] = ld_fix<COH>(xq + entry_slot(e[u]));
      }
#pragma unroll
      for (int u = 0; u < kInFlight; u++) en[u] = entry(k + (kInFlight + u) * LANES);
      // the rare branch after all pairs of the round, so that they overlap
      unsigned rare = 0u;
#pragma unroll
      for (int u = 0; u < kInFlight; u++) {
        const FixSep sep = sep_of(e[u], q[u]);
        if (pair(k + u * LANES < cnt, e[u], sep, fix_r2(sep))) rare |= 1u << u;
      }
      if (rare) {
#pragma unroll
        for (int u = 0; u < kInFlight; u++)
          if (rare >> u & 1u) close(e[u]);
      }
    }
    return;
  }
  uint32_t e0 = entry(lane), e1 = entry(lane + LANES);
  if (!MDG_IN_RANGE(d.flags, SITE, entry_slot(e0), g.n)) e0 = none;
  FixPos q0 = ld_fix<COH>(xq + entry_slot(e0));
#pragma unroll kPairsPerTrip
  for (int k = lane; k - lane < end && (ALL || k < cnt); k += LANES) {
    if (!MDG_IN_RANGE(d.flags, SITE, entry_slot(e1), g.n)) e1 = none;
    const FixPos q1 = ld_fix<COH>(xq + entry_slot(e1));
    const uint32_t e2 = entry(k + 2 * LANES);
    if (LANES == 1 && kRowsAhead > 0 && k + kRowsAhead < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (size_t)(k + kRowsAhead) * stride));
    const FixSep sep = sep_of(e0, q0);
    if (pair(k < cnt, e0, sep, fix_r2(sep))) close(e0);
    e0 = e1;
    q0 = q1;
    e1 = e2;
  }
}

// The double expression for one entry of the row of i (pairs closer than
// kFixNear), as force_fp64 evaluates it.
template <bool COH>
__device__ __noinline__ double3 near_force(const Geom &g, const double4_32a *pos, int i, int key, uint32_t e) {
  const double4_32a qi = COH ? ld_ro<true>(pos + i) : pos[i];
  double4_32a qj = COH ? ld_ro<true>(pos + entry_slot(e)) : pos[entry_slot(e)];
  apply_image(g, cell_pos(g, key), e, qj);
  const double dx = qj.x - qi.x, dy = qj.y - qi.y, dz = qj.z - qi.z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double inv = rcp_hh3(r2);
  const double i6 = inv * inv * inv;
  const double df = (i6 * inv) * fma(-48.0, i6, 24.0) + g.c2x8;
  return make_double3(df * dx, df * dy, df * dz);
}

struct RowForce {
  FixForce f;
  double nx, ny, nz;  // the pairs closer than kFixNear
  bool near;
};

template <bool PRUNE, bool EDGE, int LANES, bool COH>
__device__ __forceinline__ void row_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                          const double4_32a *__restrict__ pos, const FixPos &own, int i,
                                          const CellPos &cp, const uint32_t *__restrict__ list, int cnt, int lane,
                                          RowForce &r, int &kept) {
  const uint64_t rc2 = g.fx_rc2;
  const int64_t c8 = g.fx_c8;
  const uint32_t near = g.fx_near, keep = g.fx_keep;
  const size_t stride = (size_t)g.stride;
  walk_fixed<EDGE, LANES, PRUNE && (LANES > 1), kCheckStepSlot, COH>(
      g, d, xq, own, i, cp, list, cnt, lane, [&](bool valid, uint32_t e, const FixSep &sep, uint64_t R) {
        if (PRUNE) {
          const bool in = valid && fix_hi(R) <= keep;
          if (LANES == 1) {
            if (in) d.pl[(size_t)(kept++) * stride + i] = e;
          } else {
            // this group's lanes in row order
            const unsigned m = (__ballot_sync(0xffffffffu, in) >> ((threadIdx.x & 31) - lane)) & (LANES == 32 ? 0xffffffffu : (1u << (LANES & 31)) - 1u);
            if (in) d.pl[(size_t)(kept + __popc(m & ((1u << lane) - 1u))) * stride + i] = e;
            kept += __popc(m);
          }
        }
        const bool in = R <= rc2 && (valid || !(COH || (PRUNE && LANES > 1)));
        const bool close = in && fix_hi(R) < near;
        // evaluated for every entry and masked: no divergent branch per pair
        int64_t df = fix_force(R, c8);
        df = in && !close ? df : 0;
        fix_add(r.f, df, sep);
        return close;
      },
      [&](uint32_t e) {
        const double3 f = near_force<COH>(g, pos, i, (int)own.w, e);
        r.nx += f.x;
        r.ny += f.y;
        r.nz += f.z;
        r.near = true;
      });
}

// The force on particle i in units of 2^-52 as doubles, from LANES lanes
// (every lane of the group receives it); *kept the new inner row's length.
template <bool PRUNE, int LANES, bool COH>
__device__ __forceinline__ double3 force_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                               const double4_32a *__restrict__ pos, const FixPos &own, int i,
                                               bool wide, const uint32_t *__restrict__ list,
                                               const int *__restrict__ counts, bool active, int lane, int &kept) {
  const double up = (double)(1ull << kFixSumBits);
  const CellPos cp = cell_pos(g, (int)own.w);
  if (wide) {  // uniform over the grid
    double3 F = make_double3(0.0, 0.0, 0.0);
    if (active && lane == 0) F = force_fp64<PRUNE, COH>(g, d, pos, i, cp, list, counts, &kept);
    return make_double3(F.x * up, F.y * up, F.z * up);
  }
  int cnt = active ? ld_ro<COH>(counts + i) : 0;
  if (!MDG_IN_RANGE(d.flags, kCheckStepRow, cnt, g.list_cap + 1)) cnt = 0;
  RowForce r{{0, 0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f}, 0.0, 0.0, 0.0, false};
  if (__all_sync(0xffffffffu, !cp.edge || !active))
    row_fixed<PRUNE, false, LANES, COH>(g, d, xq, pos, own, i, cp, list, cnt, lane, r, kept);
  else
    row_fixed<PRUNE, true, LANES, COH>(g, d, xq, pos, own, i, cp, list, cnt, lane, r, kept);
  __syncwarp();
  if (LANES > 1) {
#pragma unroll
    for (int o = 1; o < LANES; o <<= 1) {
      r.f.x += __shfl_xor_sync(0xffffffffu, r.f.x, o);
      r.f.y += __shfl_xor_sync(0xffffffffu, r.f.y, o);
      r.f.z += __shfl_xor_sync(0xffffffffu, r.f.z, o);
      r.f.mx += __shfl_xor_sync(0xffffffffu, r.f.mx, o);
      r.f.my += __shfl_xor_sync(0xffffffffu, r.f.my, o);
      r.f.mz += __shfl_xor_sync(0xffffffffu, r.f.mz, o);
      r.f.cx += __shfl_xor_sync(0xffffffffu, r.f.cx, o);
      r.f.cy += __shfl_xor_sync(0xffffffffu, r.f.cy, o);
      r.f.cz += __shfl_xor_sync(0xffffffffu, r.f.cz, o);
      r.f.s += __shfl_xor_sync(0xffffffffu, r.f.s, o);
    }
  }
  double3 F;
  if (LANES == 1 || lane == 0) 
    F = make_double3(fix_sum(r.f.x, r.f.mx, r.f.cx), fix_sum(r.f.y, r.f.my, r.f.cy), fix_sum(r.f.z, r.f.mz, r.f.cz));
  if (__any_sync(0xffffffffu, r.near)) {
    if (LANES > 1) {
#pragma unroll
      for (int o = 1; o < LANES; o <<= 1) {
        r.nx += __shfl_xor_sync(0xffffffffu, r.nx, o);
        r.ny += __shfl_xor_sync(0xffffffffu, r.ny, o);
        r.nz += __shfl_xor_sync(0xffffffffu, r.nz, o);
      }
    }
    F.x += r.nx * up;
    F.y += r.ny * up;
    F.z += r.nz * up;
  }
  // sums that may have left their range: the row again in double
  if (active && lane == 0 && !fix_sum_fits(r.f, cnt)) {
    F = force_fp64<false, COH>(g, d, pos, i, cp, list, counts, nullptr);
    F = make_double3(F.x * up, F.y * up, F.z * up);
  }
  return F;
}

// A momentum component that carries a particle too far for the modulus in one
// step, or is not a number.
__device__ __forceinline__ bool fast(const Geom &g, const double4_32a &p) {
  const int m = 0x7fffffff;
  return (__double2hiint(p.x) & m) >= g.fx_pmax || (__double2hiint(p.y) & m) >= g.fx_pmax ||
         (__double2hiint(p.z) & m) >= g.fx_pmax;
}

// The rest of particle i's step after its force F (units of 2^-52), as step_one.
template <int THERMO, int COMPAT>
__device__ __forceinline__ double step_one_fixed(const Geom &g, const Dev &d, int par, int i, bool prune, int kept,
                                                 const double3 &F, double exp1, unsigned long long lang, int *rebuild,
                                                 int *reselect) {
  const double dt = g.dt, dts = g.dt * (1.0 / (double)(1ull << kFixSumBits));  // F is in units of 2^-52
  double4_32a p = d.p[i];
  if (THERMO == MDG_NOSEHOOVER) {
    const double e1 = exp1;
    p.x *= e1; p.y *= e1; p.z *= e1;
    p.x += F.x * dts; p.y += F.y * dts; p.z += F.z * dts;
    p.x *= e1; p.y *= e1; p.z *= e1;
  } else {
    p.x += F.x * dts; p.y += F.y * dts; p.z += F.z * dts;
  }
  if (THERMO == MDG_LANGEVIN) {
    double z[3];
    langevin_normals(g.seed, (uint32_t)d.id[i], lang, z);
    p.x += (-g.gamma * p.x + g.hb_d * z[0]) * dt;
    p.y += (-g.gamma * p.y + g.hb_d * z[1]) * dt;
    p.z += (-g.gamma * p.z + g.hb_d * z[2]) * dt;
  }
  const double4_32a q0 = d.q_mid[par][i];
  // the reference's separate product and sum in each half-drift
  const double hx = __dmul_rn(p.x, g.dt2), hy = __dmul_rn(p.y, g.dt2), hz = __dmul_rn(p.z, g.dt2);
  double4_32a qe = q0, q1;
  if (!(THERMO == MDG_LANGEVIN && COMPAT)) {
    qe.x = __dadd_rn(q0.x, hx);
    qe.y = __dadd_rn(q0.y, hy);
    qe.z = __dadd_rn(q0.z, hz);
  }
  q1 = qe;
  q1.x = __dadd_rn(qe.x, hx);
  q1.y = __dadd_rn(qe.y, hy);
  q1.z = __dadd_rn(qe.z, hz);
  const int4 xb = d.xb[i];
  const FixPos xn = fix_position(q1.x, q1.y, q1.z, xb.w);
  const float u = 1.0f / (float)(1 << (kFixPosBits - 32));
  // displacement since the build, from the high words (1.9e-9 sigma): the
  // rebuild test in float, within 1e-6 of the threshold in double
  const float bx = (float)(xn.x - xb.x) * u, by = (float)(xn.y - xb.y) * u, bz = (float)(xn.z - xb.z) * u;
  const float b2 = bx * bx + by * by + bz * bz;
  const bool far = fast(g, p);
  if (g.rebuild_policy == MDG_REBUILD_HALFMARGIN) {
    bool moved = far || b2 > g.fx_moved_hi;
    if (!moved && b2 >= g.fx_moved_lo) {
      const double4_32a qb = d.q_build[i];
      const double ux = q1.x - qb.x, uy = q1.y - qb.y, uz = q1.z - qb.z;
      moved = ux * ux + uy * uy + uz * uz > g.half_margin2;
    }
    if (moved) *rebuild = 1;
  }
  if (far && !(q1.x == q1.x && q1.y == q1.y && q1.z == q1.z)) *rebuild = 1;
  if (far || fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz))) > g.fx_guard) d.flags->fx_wide[par ^ 1] = 1;
  // inner-list reference: this force evaluation's positions when the rows
  // were re-selected now, else those of the last selection
  int4 xp;
  if (prune) {
    const FixPos x0 = d.xq[par][i];
    xp = make_int4(x0.x, x0.y, x0.z, 0);
    d.xp[i] = xp;
    d.pcount[i] = kept;
  } else {
    xp = d.xp[i];
  }
  const float vx = (float)(xn.x - xp.x) * u, vy = (float)(xn.y - xp.y) * u, vz = (float)(xn.z - xp.z) * u;
  if (vx * vx + vy * vy + vz * vz > g.half_prune2) *reselect = 1;
  d.xq[par ^ 1][i] = xn;
  d.p[i] = p;
  d.q_end[i] = qe;
  d.q_mid[par ^ 1][i] = q1;
  return THERMO == MDG_NOSEHOOVER ? 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z : 0.0;
}

}  // namespace mdg

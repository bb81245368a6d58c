// The FP64 form's step, observers and forces with the pair arithmetic in
// 64-bit fixed point (mdg_fixed.cuh): the same step as k_step (mdg_step.cu),
// the same state and integration in double, rounding for rounding; only the
// pair separation, distance and force run on the integer units.
//
// Used when Geom::fixed is set: search length + margin below 4 sigma (the
// positions are kept modulo 8 sigma) and a cut-off of at least one sigma;
// anything else keeps the double pair loop of k_step.  So does a step whose
// positions are not safe modulo 8 (flags->fx_wide: a particle further from
// its place at the build than Geom::fx_guard allows for two of them), and a
// row whose force sums might leave their range (fix_sum_fits); a pair closer
// than r^2 = kFixNear takes the double expression by itself.
//
// Extra state: xq[2] the fixed-point positions of q_mid[2] (what partners
// gather, 32 bytes, the w word holds the home cell), xb the high words at the
// last build and xp at the last inner-list selection (displacement tests).
#include "mdg_step.cuh"
#include "mdg_fixed.cuh"

namespace mdg {

namespace {

// Threads per block: one thread per particle, or kWide threads whose LANES
// neighbours share a particle's row.
constexpr int kOne = 128, kWide = 256;
// Blocks per SM asked for with one thread per particle (80 registers; the
// integer multiply-adds keep their pipe about 80 % busy): 4M atoms, step kernel
// 1.073 ms with 6 blocks, 1.115 with 5.
constexpr int kOneBlocks = 6;
// List rows requested into L2 this many entries ahead with one thread per
// particle (1.073 ms; 24 ahead 1.083, none 1.090; observers 1.35 against 1.53).
constexpr int kRowsAhead = 12;
// Pairs per trip of the row walk (2: no moves for the entries in flight;
// 1.073 ms, 1 pair 1.095, 4 pairs 1.130).
constexpr int kPairsPerTrip = 2;

template <int LANES>
__host__ __device__ constexpr int fx_threads() { return LANES == 1 ? kOne : kWide; }
template <int LANES>
__host__ __device__ constexpr int fx_particles() { return fx_threads<LANES>() / LANES; }

// Lanes per particle for n particles.  A row's pairs take about half a
// microsecond one after the other, so a GPU that one thread per particle does
// not fill (152 SMs x 24 warps) is better used by several: step kernel of 864
// atoms 34.0, 26.2, 21.7, 19.1 us with 1, 2, 4, 8 lanes; 32,000 atoms 32.3,
// 28.3, 30.8, 36.1; 256,000 atoms 141, 187, 229, 304 (of which about 8 us are
// the graph's hand-over).
inline int fx_lanes(int n) { return n < 12288 ? 8 : (n < 65536 ? 2 : 1); }

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
// pair(valid, e, sep, R) the separation and R = r^2.  One position and two
// entries are in flight.  ALL: every thread of the warp calls pair the same number
// of times (for ballots), with valid = false past its row.
template <bool EDGE, int LANES, bool ALL, int SITE, class Pair>
__device__ __forceinline__ void walk_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                           const FixPos &own, int i, const CellPos &cp,
                                           const uint32_t *__restrict__ list, int cnt, int lane, Pair &&pair) {
  Faces fc;
  if (EDGE) fc = faces_of(g, cp);
  const uint32_t *row = list + i;
  const size_t stride = (size_t)g.stride;
  const uint32_t none = entry_pack(i, 0, 0, 0);  // a valid address past the row's end
  auto entry = [&](int k) { return k < cnt ? __ldg(row + (size_t)k * stride) : none; };
  int end = cnt;
  if (ALL) end = __reduce_max_sync(0xffffffffu, cnt);
  uint32_t e0 = entry(lane), e1 = entry(lane + LANES);
  if (!MDG_IN_RANGE(d.flags, SITE, entry_slot(e0), g.n)) e0 = none;
  FixPos q0 = ld_fix(xq + entry_slot(e0));
#pragma unroll kPairsPerTrip
  for (int k = lane; k - lane < end && (ALL || k < cnt); k += LANES) {
    if (!MDG_IN_RANGE(d.flags, SITE, entry_slot(e1), g.n)) e1 = none;
    const FixPos q1 = ld_fix(xq + entry_slot(e1));
    const uint32_t e2 = entry(k + 2 * LANES);
    if (LANES == 1 && kRowsAhead > 0 && k + kRowsAhead < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (size_t)(k + kRowsAhead) * stride));
    int dx = q0.x - own.x, dy = q0.y - own.y, dz = q0.z - own.z;
    float lx = q0.lx - own.lx, ly = q0.ly - own.ly, lz = q0.lz - own.lz;
    if (EDGE) {
      const uint32_t s = e0 ^ 0x15u;
      if ((s & 0x03u) == fc.kx) { dx += fc.sx; lx += fc.lx; }
      if ((s & 0x0Cu) == fc.ky) { dy += fc.sy; ly += fc.ly; }
      if ((s & 0x30u) == fc.kz) { dz += fc.sz; lz += fc.lz; }
    }
    const FixSep sep = fix_sep(dx, dy, dz, lx, ly, lz);
    pair(k < cnt, e0, sep, fix_r2(sep));
    e0 = e1;
    q0 = q1;
    e1 = e2;
  }
}

// The double expression for one entry of the row of i (pairs closer than
// kFixNear), as force_fp64 evaluates it.
__device__ __noinline__ double3 near_force(const Geom &g, const double4_32a *pos, int i, int key, uint32_t e) {
  const double4_32a qi = pos[i];
  double4_32a qj = pos[entry_slot(e)];
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

template <bool PRUNE, bool EDGE, int LANES>
__device__ __forceinline__ void row_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                          const double4_32a *__restrict__ pos, const FixPos &own, int i,
                                          const CellPos &cp, const uint32_t *__restrict__ list, int cnt, int lane,
                                          RowForce &r, int &kept) {
  const uint64_t rc2 = g.fx_rc2;
  const int64_t c8 = g.fx_c8;
  const uint32_t near = g.fx_near, keep = g.fx_keep;
  const size_t stride = (size_t)g.stride;
  walk_fixed<EDGE, LANES, PRUNE && (LANES > 1), kCheckStepSlot>(
      g, d, xq, own, i, cp, list, cnt, lane, [&](bool valid, uint32_t e, const FixSep &sep, uint64_t R) {
        if (PRUNE) {
          const bool in = valid && fix_hi(R) <= keep;
          if (LANES == 1) {
            if (in) d.pl[(size_t)(kept++) * stride + i] = e;
          } else {
            // this group's lanes in row order
            const unsigned m = (__ballot_sync(0xffffffffu, in) >> ((threadIdx.x & 31) - lane)) & ((1u << LANES) - 1u);
            if (in) d.pl[(size_t)(kept + __popc(m & ((1u << lane) - 1u))) * stride + i] = e;
            kept += __popc(m);
          }
        }
        const bool in = R <= rc2 && (valid || !(PRUNE && LANES > 1));
        const bool close = in && fix_hi(R) < near;
        // evaluated for every entry and masked: no divergent branch per pair
        int64_t df = fix_force(R, c8);
        df = in && !close ? df : 0;
        fix_add(r.f, df, sep);
        if (close) {
          const double3 f = near_force(g, pos, i, (int)own.w, e);
          r.nx += f.x;
          r.ny += f.y;
          r.nz += f.z;
          r.near = true;
        }
      });
}

// The force on particle i in units of 2^-52 as doubles, from LANES lanes
// (every lane of the group receives it); *kept the new inner row's length.
template <bool PRUNE, int LANES>
__device__ __forceinline__ double3 force_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                               const double4_32a *__restrict__ pos, const FixPos &own, int i,
                                               bool wide, const uint32_t *__restrict__ list,
                                               const int *__restrict__ counts, bool active, int lane, int &kept) {
  const double up = (double)(1ull << kFixSumBits);
  const CellPos cp = cell_pos(g, (int)own.w);
  if (wide) {  // uniform over the grid
    double3 F = make_double3(0.0, 0.0, 0.0);
    if (active && lane == 0) F = force_fp64<PRUNE>(g, d, pos, i, cp, list, counts, &kept);
    return make_double3(F.x * up, F.y * up, F.z * up);
  }
  int cnt = active ? counts[i] : 0;
  if (!MDG_IN_RANGE(d.flags, kCheckStepRow, cnt, g.list_cap + 1)) cnt = 0;
  RowForce r{{0, 0, 0, 0, 0, 0, 0.f, 0.f, 0.f, 0.f}, 0.0, 0.0, 0.0, false};
  if (__all_sync(0xffffffffu, !cp.edge || !active))
    row_fixed<PRUNE, false, LANES>(g, d, xq, pos, own, i, cp, list, cnt, lane, r, kept);
  else
    row_fixed<PRUNE, true, LANES>(g, d, xq, pos, own, i, cp, list, cnt, lane, r, kept);
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
    F = force_fp64<false>(g, d, pos, i, cp, list, counts, nullptr);
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

// The step of k_step (mdg_step.cu) on the fixed-point positions; PMODE as there.
template <int THERMO, int COMPAT, int PMODE, int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>(), LANES == 1 ? kOneBlocks : 2) k_step_fixed(Geom g, Dev d, int par) {
  constexpr int kThreads = fx_threads<LANES>(), kParticles = fx_particles<LANES>();
  const DevFlags *f = d.flags;
  if (f->halt != 0) return;
  if (PMODE == 1 && f->prune_now != 0) return;
  if (PMODE == 2 && f->prune_now == 0) return;
  const bool prune = PMODE == 2 ? true : (PMODE == 1 ? false : f->prune_now != 0);
  const bool wide = f->fx_wide[par] != 0;
  const double4_32a *qm = d.q_mid[par];
  double4_32a *qn = d.q_mid[par ^ 1];
  const FixPos *xq = d.xq[par];
  const int first = blockIdx.x * kParticles;
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  int i = first + threadIdx.x / LANES;
  bool active = i < g.n;
  int kept = 0;
  double3 F = make_double3(0.0, 0.0, 0.0);
  {
    const int ia = active ? i : g.n - 1;
    const FixPos own = xq[ia];
    if (prune) F = force_fixed<true, LANES>(g, d, xq, qm, own, ia, wide, d.nl, d.ncount, active, lane, kept);
    else F = force_fixed<false, LANES>(g, d, xq, qm, own, ia, wide, d.pl, d.pcount, active, lane, kept);
  }
  if (LANES > 1) {
    // the block's particles move on to its first threads, one each
    __shared__ double3 sF[kParticles];
    __shared__ int sk[kParticles];
    if (lane == 0) {
      sF[threadIdx.x / LANES] = F;
      sk[threadIdx.x / LANES] = kept;
    }
    __syncthreads();
    i = first + threadIdx.x;
    active = threadIdx.x < kParticles && i < g.n;
    kept = 0;
    if (active) {
      F = sF[threadIdx.x];
      kept = sk[threadIdx.x];
    }
  }
  double ke = 0.0;
  if (active) {
    const double dt = g.dt, dts = g.dt * (1.0 / (double)(1ull << kFixSumBits));  // F is in units of 2^-52
    double4_32a p = d.p[i];
    if (THERMO == MDG_NOSEHOOVER) {
      const double e1 = f->exp1;
      p.x *= e1; p.y *= e1; p.z *= e1;
      p.x += F.x * dts; p.y += F.y * dts; p.z += F.z * dts;
      p.x *= e1; p.y *= e1; p.z *= e1;
    } else {
      p.x += F.x * dts; p.y += F.y * dts; p.z += F.z * dts;
    }
    if (THERMO == MDG_LANGEVIN) {
      double z[3];
      langevin_normals(g.seed, (uint32_t)d.id[i], f->lang - 1ull, z);
      p.x += (-g.gamma * p.x + g.hb_d * z[0]) * dt;
      p.y += (-g.gamma * p.y + g.hb_d * z[1]) * dt;
      p.z += (-g.gamma * p.z + g.hb_d * z[2]) * dt;
    }
    const double4_32a q0 = qm[i];
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
      if (moved) d.flags->rebuild = 1;
    }
    if (far && !(q1.x == q1.x && q1.y == q1.y && q1.z == q1.z)) d.flags->rebuild = 1;
    if (far || fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz))) > g.fx_guard) d.flags->fx_wide[par ^ 1] = 1;
    // inner-list reference: this force evaluation's positions when the rows
    // were re-selected now, else those of the last selection
    int4 xp;
    if (prune) {
      const FixPos x0 = xq[i];
      xp = make_int4(x0.x, x0.y, x0.z, 0);
      d.xp[i] = xp;
      d.pcount[i] = kept;
    } else {
      xp = d.xp[i];
    }
    const float vx = (float)(xn.x - xp.x) * u, vy = (float)(xn.y - xp.y) * u, vz = (float)(xn.z - xp.z) * u;
    if (vx * vx + vy * vy + vz * vz > g.half_prune2) d.flags->prune_next = 1;
    d.xq[par ^ 1][i] = xn;
    d.p[i] = p;
    d.q_end[i] = qe;
    qn[i] = q1;
    if (THERMO == MDG_NOSEHOOVER) ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
  }
  if (THERMO == MDG_NOSEHOOVER) {
    __shared__ double sh[kThreads / 32];
    const double t = block_sum(ke, sh);
    if (threadIdx.x == 0) d.partials[blockIdx.x] = t;
  }
  if (prune) {  // inner-list size for the statistics (uniform branch)
    unsigned long long v = (unsigned long long)kept;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&d.flags->inner_pairs, v);
  }
}

// Fixed-point positions of q_end into xq[dst] (the buffer the next step
// overwrites before reading it); a particle too far from its place at the
// build marks fx_wide_end with this call's number.
__global__ void k_fix_end(Geom g, Dev d, int dst, int call) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.n) return;
  const int4 xb = d.xb[i];
  const double4_32a q = d.q_end[i];
  const FixPos x = fix_position(q.x, q.y, q.z, xb.w);
  const float u = 1.0f / (float)(1 << (kFixPosBits - 32));
  const float bx = (float)(x.x - xb.x) * u, by = (float)(x.y - xb.y) * u, bz = (float)(x.z - xb.z) * u;
  if (fast(g, d.p[i]) || fmaxf(fabsf(bx), fmaxf(fabsf(by), fabsf(bz))) > g.fx_guard) d.flags->fx_wide_end = call;
  d.xq[dst][i] = x;
}

template <int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>()) k_forces_fixed(Geom g, Dev d, int src, int call) {
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  const int i = blockIdx.x * fx_particles<LANES>() + threadIdx.x / LANES;
  const bool active = i < g.n;
  const int ia = active ? i : g.n - 1;
  int kept = 0;
  const double3 F = force_fixed<false, LANES>(g, d, d.xq[src], d.q_end, d.xq[src][ia], ia, d.flags->fx_wide_end == call,
                                              d.nl, d.ncount, active, lane, kept);
  const double s = 1.0 / (double)(1ull << kFixSumBits);
  if (active && lane == 0) d.io4[d.id[i]] = make_double4_32a(F.x * s, F.y * s, F.z * s, 0.0);
}

// Longest row whose sums of z^2 (2.83 at most each, units of 2^-54) fit.
constexpr int kFixObserveRow = 361;

// Observers (observer.cc:5-79) at q_end: a row's pair energies are
// 4 (sum z^2 - sum z + C2 sum r^2 + C0 count) and its virial terms
// 24 sum z - 48 sum z^2 + 8 C2 sum r^2 with z = r^-6, summed as integers (the
// cut bits' mean, half a unit, added back); each pair is listed from both sides
// and weighted 1/2.
template <bool EDGE, int LANES>
__device__ __forceinline__ void observe_fixed(const Geom &g, const Dev &d, const FixPos *__restrict__ xq,
                                              const FixPos &own, int i, const CellPos &cp, int cnt, int lane,
                                              uint64_t &sz, uint64_t &szz, uint64_t &sr, int &m, double &ne, double &nv) {
  const uint64_t rc2 = g.fx_rc2;
  const uint32_t near = g.fx_near;
  walk_fixed<EDGE, LANES, false, kCheckObserve>(
      g, d, xq, own, i, cp, d.nl, cnt, lane, [&](bool, uint32_t e, const FixSep &, uint64_t R) {
        const bool in = R <= rc2, close = in && fix_hi(R) < near, take = in && !close;
        uint64_t y2, z;
        fix_powers(fix_recip(R), y2, z);
        const uint64_t zz = fix_sqrhi(z);  // 2^-58
        sz += take ? z >> 7 : 0;
        szz += take ? zz >> 4 : 0;
        sr += take ? R >> 7 : 0;  // 2^-51
        m += take ? 1 : 0;
        if (close) {
          double4_32a qj = d.q_end[entry_slot(e)];
          const double4_32a qi = d.q_end[i];
          apply_image(g, cp, e, qj);
          const double dx = __dsub_rn(qi.x, qj.x), dy = __dsub_rn(qi.y, qj.y), dz = __dsub_rn(qi.z, qj.z);
          const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
          double a, b;
          pair_observables(g, r2, a, b);
          ne += a;
          nv += b;
        }
      });
}

template <int LANES>
__global__ void __launch_bounds__(fx_threads<LANES>()) k_observe_fixed(Geom g, Dev d, int src, int call) {
  __shared__ double sh[fx_threads<LANES>() / 32];
  const int lane = LANES == 1 ? 0 : threadIdx.x % LANES;
  const int i = blockIdx.x * fx_particles<LANES>() + threadIdx.x / LANES;
  const bool active = i < g.n;
  double ke = 0.0, pe = 0.0, vir = 0.0;
  const int ia = active ? i : g.n - 1;
  const FixPos own = d.xq[src][ia];
  const CellPos cp = cell_pos(g, (int)own.w);
  int cnt = active ? d.ncount[ia] : 0;
  if (!MDG_IN_RANGE(d.flags, kCheckObserve, cnt, g.list_cap + 1)) cnt = 0;
  if (active && lane == 0) {
    const double4_32a p = d.p[ia];
    ke = 0.5 * p.x * p.x + 0.5 * p.y * p.y + 0.5 * p.z * p.z;
  }
  if (d.flags->fx_wide_end == call || cnt > kFixObserveRow) {
    if (active && lane == 0) observe_row_fp64(g, d, ia, cp, cnt, pe, vir);
  } else {
    uint64_t sz = 0, szz = 0, sr = 0;
    int m = 0;
    double ne = 0.0, nv = 0.0;
    if (__all_sync(__activemask(), !cp.edge)) observe_fixed<false, LANES>(g, d, d.xq[src], own, ia, cp, cnt, lane, sz, szz, sr, m, ne, nv);
    else observe_fixed<true, LANES>(g, d, d.xq[src], own, ia, cp, cnt, lane, sz, szz, sr, m, ne, nv);
    const double u = 1.0 / (double)(1ull << 54), half = 0.5 * m;
    const double z = ((double)sz + half) * u, zz = ((double)szz + half) * u;
    const double r = g.c2 * (((double)sr + half) * (1.0 / (double)(1ull << 51)));
    pe = ne + 2.0 * ((zz - z) + (r + g.c0 * (double)m));
    vir = nv + 12.0 * (z - 2.0 * zz) + 4.0 * r;
  }
  const double a = block_sum(ke, sh);
  const double b = block_sum(pe, sh);
  const double c = block_sum(vir, sh);
  if (threadIdx.x == 0) {
    d.partials[3 * blockIdx.x + 0] = a;
    d.partials[3 * blockIdx.x + 1] = b;
    d.partials[3 * blockIdx.x + 2] = c;
  }
}

template <int LANES>
int fx_grid(int n) { return n > 0 ? (n + fx_particles<LANES>() - 1) / fx_particles<LANES>() : 1; }

template <int T, int C, int LANES>
int launch_lanes(const Geom &g, const Dev &d, int par, int pmode, cudaStream_t s) {
  constexpr int t = fx_threads<LANES>();
  const int grid = fx_grid<LANES>(g.n);
  if (pmode == 0) k_step_fixed<T, C, 0, LANES><<<grid, t, 0, s>>>(g, d, par);
  if (pmode == 1 || pmode == 3) k_step_fixed<T, C, 1, LANES><<<grid, t, 0, s>>>(g, d, par);
  if (pmode == 2 || pmode == 3) k_step_fixed<T, C, 2, LANES><<<grid, t, 0, s>>>(g, d, par);
  return grid;
}

template <int T, int C>
int launch_thermo(const Geom &g, const Dev &d, int par, int pmode, cudaStream_t s) {
  const int lanes = fx_lanes(g.n);
  return lanes == 8   ? launch_lanes<T, C, 8>(g, d, par, pmode, s)
         : lanes == 2 ? launch_lanes<T, C, 2>(g, d, par, pmode, s)
                      : launch_lanes<T, C, 1>(g, d, par, pmode, s);
}

}  // namespace

int launch_step_fixed(const Geom &g, const Dev &d, int par, int thermostat, int compat, int pmode, cudaStream_t s) {
  if (thermostat == MDG_LANGEVIN)
    return compat ? launch_thermo<MDG_LANGEVIN, 1>(g, d, par, pmode, s) : launch_thermo<MDG_LANGEVIN, 0>(g, d, par, pmode, s);
  if (thermostat == MDG_NOSEHOOVER) return launch_thermo<MDG_NOSEHOOVER, 0>(g, d, par, pmode, s);
  return launch_thermo<MDG_NVE, 0>(g, d, par, pmode, s);
}

void launch_forces_fixed(const Geom &g, const Dev &d, int par, int call, cudaStream_t s) {
  const int dst = par ^ 1, lanes = fx_lanes(g.n);
  k_fix_end<<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  if (lanes == 8) k_forces_fixed<8><<<fx_grid<8>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 2) k_forces_fixed<2><<<fx_grid<2>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else k_forces_fixed<1><<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
}

int launch_observe_fixed(const Geom &g, const Dev &d, int par, int call, cudaStream_t s) {
  const int dst = par ^ 1, lanes = fx_lanes(g.n);
  k_fix_end<<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  if (lanes == 8) k_observe_fixed<8><<<fx_grid<8>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else if (lanes == 2) k_observe_fixed<2><<<fx_grid<2>(g.n), kWide, 0, s>>>(g, d, dst, call);
  else k_observe_fixed<1><<<fx_grid<1>(g.n), kOne, 0, s>>>(g, d, dst, call);
  return lanes == 8 ? fx_grid<8>(g.n) : lanes == 2 ? fx_grid<2>(g.n) : fx_grid<1>(g.n);
}

}  // namespace mdg

// The fixed-point pair arithmetic built for the host (tests/test_fixed.py).
#include "../mdacp_gb300/csrc/mdg_fixed.cuh"

using namespace mdg;

// out: high words and rests of n coordinates as doubles (their sum is the coordinate modulo 8)
extern "C" void fixed_positions(const double *x, int n, double *out) {
  for (int k = 0; k < n; k++) {
    const FixPos p = fix_position(x[k], 0.0, 0.0, 0);
    out[2 * k] = (double)p.x / 536870912.0;
    out[2 * k + 1] = (double)p.lx / 268435456.0;
  }
}

// f[3n]: the force on each qi from its qj; r2[n]
extern "C" void fixed_forces(const double *qi, const double *qj, int n, double c2x8, double *f, double *r2) {
  const int64_t c8 = fix_c8(c2x8);
  for (int k = 0; k < n; k++) {
    const FixPos a = fix_position(qi[3 * k], qi[3 * k + 1], qi[3 * k + 2], 0);
    const FixPos b = fix_position(qj[3 * k], qj[3 * k + 1], qj[3 * k + 2], 0);
    const FixSep s = fix_sep(b.x - a.x, b.y - a.y, b.z - a.z, b.lx - a.lx, b.ly - a.ly, b.lz - a.lz);
    const uint64_t R = fix_r2(s);
    FixForce F{};
    fix_add(F, fix_force(R, c8), s);
    const double u = 1.0 / 4503599627370496.0;
    f[3 * k] = fix_sum(F.x, F.mx, F.cx) * u;
    f[3 * k + 1] = fix_sum(F.y, F.my, F.cy) * u;
    f[3 * k + 2] = fix_sum(F.z, F.mz, F.cz) * u;
    r2[k] = (double)R / 288230376151711744.0;
  }
}

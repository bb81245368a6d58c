// r^2 of image pairs in fixed point built for the host (tests/test_fixed_faces.py).
#include "../mdacp_gb300/csrc/mdg_fixed.cuh"

using namespace mdg;

// out[2k], out[2k + 1]: r^2 of the pair qi[k], qj[k] + s[k] L (s = -1, 0, 1 per axis) in units of 2^-58, as its two words
extern "C" void fixed_image_r2(const double *qi, const double *qj, const int *s, const double *L, int n, double *out) {
  for (int k = 0; k < n; k++) {
    const FixPos a = fix_position(qi[3 * k], qi[3 * k + 1], qi[3 * k + 2], 0);
    const FixPos b = fix_position(qj[3 * k], qj[3 * k + 1], qj[3 * k + 2], 0);
    uint32_t d[3] = {(uint32_t)b.x - (uint32_t)a.x, (uint32_t)b.y - (uint32_t)a.y, (uint32_t)b.z - (uint32_t)a.z};
    float l[3] = {b.lx - a.lx, b.ly - a.ly, b.lz - a.lz};
    for (int c = 0; c < 3; c++) {
      const int64_t side = fix_from_double(L[3 * k + c]);
      d[c] += (uint32_t)s[3 * k + c] * (uint32_t)fix_shi(side);
      l[c] += (float)s[3 * k + c] * fix_rest(side);
    }
    const uint64_t R = fix_r2(fix_sep((int32_t)d[0], (int32_t)d[1], (int32_t)d[2], l[0], l[1], l[2]));
    out[2 * k] = (double)fix_hi(R);
    out[2 * k + 1] = (double)fix_lo(R);
  }
}

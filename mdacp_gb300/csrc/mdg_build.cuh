// One particle's row of the pair list, shared by the single box and the
// batch: the candidates of the 27 stencil cells tested in float from
// home-cell-local positions, the few inside the float band by the caller's
// exact test.
//
// A cell's candidates are tested 32 at a time into bit masks (eleven
// instructions each, no branch) and the accepted ones, a seventh of them, are
// written from the masks: appending inside the test loop cost every
// candidate the append's instructions, since some lane of the warp almost always
// accepts (25 instructions a candidate).
#pragma once
#include "mdg_internal.cuh"

namespace mdg {

// The cells around home cell (cx, cy, cz) of a periodic box: number of cells
// and, per axis, the float offsets between cell centres.
struct Stencil {
  int nc[3];
  float w[3], dl[3];
};

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

}  // namespace mdg

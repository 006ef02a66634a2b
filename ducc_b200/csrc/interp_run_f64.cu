// Double-precision 2D interpolation with register windows.
#include "interp_run.cuh"

namespace dnufft {

void launch_interp_run(const PointsDesc &pts, const uint32_t *sel, uint32_t npts,
                       const Geometry &g, const KernelPoly<double> &kp, const void *grid,
                       int64_t gtrans, void *out, int64_t os, int64_t otrans, int ntrans,
                       cudaStream_t st) {
  if (npts == 0 || ntrans == 0) return;
#define DN_CASE(WW)                                                                             \
  case WW:                                                                                      \
    if (pts.coord_f64)                                                                          \
      interp_run_w<double, WW>(pts, sel, npts, g, kp, grid, gtrans, out, os, otrans, ntrans, st); \
    else                                                                                        \
      interp_run_w<float, WW>(pts, sel, npts, g, kp, grid, gtrans, out, os, otrans, ntrans, st); \
    return;
  switch (g.W) { DN_FOR_W_DOUBLE(DN_CASE) }
#undef DN_CASE
  throw Error(ST_UNSUPPORTED, "kernel support not supported by this build");
}

}  // namespace dnufft

// Single-precision 3D interpolation with register windows.
#include "interp_run3.cuh"

namespace dnufft {

void launch_interp_run3(const PointsDesc &pts, const Geometry &g, const KernelPoly<float> &kp,
                        const void *grid, int64_t gtrans, void *out, int64_t os, int64_t otrans,
                        int ntrans, cudaStream_t st) {
  if (pts.npts == 0 || ntrans == 0) return;
  // the one support for which interp3_in_windows (capi.cpp) holds in single precision
  if (g.W == 8) {
    if (pts.coord_f64)
      interp_run3f_w<double, 8>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);
    else
      interp_run3f_w<float, 8>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);
    return;
  }
  throw Error(ST_UNSUPPORTED, "kernel support not supported by this build");
}

}  // namespace dnufft

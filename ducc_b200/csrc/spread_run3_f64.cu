// 3D spreading with register windows, double precision (complex128 data).
#include "spread_run3.cuh"

namespace dnufft {

template <typename T>
void launch_spread_run3(const PointsDesc &pts, const Geometry &g, const KernelPoly<T> &kp,
                        const void *values, int64_t vs, int64_t vtrans, void *grid,
                        int64_t gtrans, int ntrans, cudaStream_t st) {
  launch_spread_run3_impl<T>(pts, g, kp, values, vs, vtrans, grid, gtrans, ntrans, st);
}

template void launch_spread_run3<double>(const PointsDesc &, const Geometry &,
                                         const KernelPoly<double> &, const void *, int64_t, int64_t,
                                         void *, int64_t, int, cudaStream_t);

}  // namespace dnufft

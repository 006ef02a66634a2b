// 2D spreading with register accumulators, double precision (complex128 data).
#include "spread_run.cuh"

namespace dnufft {

template <typename T>
void launch_spread_run(const PointsDesc &pts, const uint32_t *sel, uint32_t npts, const Geometry &g,
                       const KernelPoly<T> &kp, const void *values, int64_t vs, int64_t vtrans,
                       void *grid, int64_t gtrans, int ntrans, cudaStream_t st) {
  launch_spread_run_impl<T>(pts, sel, npts, g, kp, values, vs, vtrans, grid, gtrans, ntrans, st);
}

template void launch_spread_run<double>(const PointsDesc &, const uint32_t *, uint32_t,
                                        const Geometry &, const KernelPoly<double> &, const void *,
                                        int64_t, int64_t, void *, int64_t, int, cudaStream_t);

}  // namespace dnufft

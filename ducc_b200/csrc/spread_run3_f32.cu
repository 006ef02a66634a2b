// 3D spreading with register windows, single precision (complex64 data).
#include "spread_run3.cuh"

namespace dnufft {

template <typename T>
void launch_spread_run3(const PointsDesc &pts, const Geometry &g, const KernelPoly<T> &kp,
                        const void *values, int64_t vs, int64_t vtrans, void *grid,
                        int64_t gtrans, int ntrans, cudaStream_t st) {
  launch_spread_run3_impl<T>(pts, g, kp, values, vs, vtrans, grid, gtrans, ntrans, st);
}

template void launch_spread_run3<float>(const PointsDesc &, const Geometry &,
                                         const KernelPoly<float> &, const void *, int64_t, int64_t,
                                         void *, int64_t, int, cudaStream_t);

int spread_run3_bin_log2(int W) { return run3_bin_log2(W); }

}  // namespace dnufft

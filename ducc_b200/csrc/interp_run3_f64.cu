// Double-precision 3D interpolation.
#include "interp_run3.cuh"

namespace dnufft {

// supports of the direct kernel
#define DN_FOR_W_DIRECT3(M) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(11) M(12) M(13) M(14) M(15)

// The direct kernel or the windows?  A point costs the direct kernel W^3 reads
// through L1, and the windows FP64 matrix instructions over the whole window,
// plus its share of loading the window (16 to 24 cells per axis) once per bin: the
// direct kernel is the faster one for small supports, and for larger ones where
// points are few per bin of 8^3 cells.  Measured (us, windows / direct; p: points
// per 8^3 cells):
//   W = 6   p = 300: 257 / 106, p = 512: 1550 / 541
//   W = 8   p = 5: 1 / 0.44-0.69, p = 50: 1 / 0.78-0.86, p = 500: 1 / 0.62
//   W = 10  p = 5: 1 / 0.61-0.78, p = 50: 1 / 0.99-1.06, p = 500: 1 / 0.75
//   W = 11  p = 5: 1 / 0.74-0.91, p = 17-170: 1 / 1.1-1.26, p = 500: 1 / 0.94
//   W = 12  p = 5: 1 / 0.91, p = 15-500: 1 / 1.2-1.57
//   W = 14  (bins of 4^3 cells) p = 15-22: 1 / 0.72-0.80, p = 50: 1 / 1.0-1.08
//   W = 15  p = 5-17: 1 / 0.73-0.96, p = 50: 1 / 1.2-1.3
//   W = 16  p = 7: 1 / 0.85, else more
// A few thousand points are latency: from W = 8 the windows' many warps per point
// finish sooner (1000 points: 1 / 1.03-1.2 at W = 8, 1 / 2.5 at W = 14).
bool interp3_direct(const Geometry &g, uint32_t npts) {
  const int W = g.W;
  if (W > 15 || (W >= 8 && npts < (W <= 10 ? 4096u : 16384u))) return false;
  if (W <= 10) return true;
  const double p = double(npts) * 512. / (double(g.nover[0]) * double(g.nover[1]) * double(g.nover[2]));
  if (W == 11) return p < 8. || p > 500.;
  if (W == 12) return p < 6.;
  return p < (W <= 14 ? 30. : 18.);
}

void launch_interp_run3(const PointsDesc &pts, const Geometry &g, const KernelPoly<double> &kp,
                        const void *grid, int64_t gtrans, void *out, int64_t os, int64_t otrans,
                        int ntrans, cudaStream_t st) {
  if (pts.npts == 0 || ntrans == 0) return;
  if (interp3_direct(g, pts.npts)) {
#define DN_CASE(WW)                                                                           \
  case WW:                                                                                    \
    if (pts.coord_f64)                                                                        \
      interp_direct3_w<double, WW>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);    \
    else                                                                                      \
      interp_direct3_w<float, WW>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);     \
    return;
    switch (g.W) { DN_FOR_W_DIRECT3(DN_CASE) }
#undef DN_CASE
  }
#define DN_CASE(WW)                                                                           \
  case WW:                                                                                    \
    if (pts.coord_f64)                                                                        \
      interp_run3_w<double, WW>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);       \
    else                                                                                      \
      interp_run3_w<float, WW>(pts, g, kp, grid, gtrans, out, os, otrans, ntrans, st);        \
    return;
  switch (g.W) { DN_FOR_W_DOUBLE(DN_CASE) }
#undef DN_CASE
  throw Error(ST_UNSUPPORTED, "kernel support not supported by this build");
}

}  // namespace dnufft

// Double-precision 2D interpolation (type 2) with the window of a bin in
// registers: the transpose of spread_run.cuh.
//
// A warp takes consecutive sorted points.  Per bin of 8 x 8 cells it loads the
// window of 8 MT x 4 NT grid cells that the footprints of the bin's points lie in
// into the fragments of FP64 matrix instructions (mma m8n8k4), and eight points
// at a time multiplies their column weights (zero-filled to the window) with it:
// T[point][row] = sum over columns of kv * G[row][column], both components.  The
// accumulator fragments hold one point per four lanes; these multiply them with
// the point's row weights and add up.
//
// Staging a tile in shared memory and reading W^2 cells of 16 bytes per point
// took 132 SM cycles per point at W = 15 (28 of shared-memory bandwidth, the rest
// bank conflicts and latency at 255 registers); this takes 18 cycles of matrix
// instructions per point, and the window's loads come from L2 once per bin: 5e6
// points 2.32 -> 0.80 ms, 46 cycles in all (12 warps per SM; the matrix pipe is
// active 39 % of the cycles, the rest is the latency of staging and of the loads).
//
// A window with a value that is not finite is not multiplied (zero weights
// would spread it to points that do not touch it): its points read their own
// W x W cells.
//
// Mirrors HelperU2nu / interpolation_helper (src/ducc0/nufft/nufft.h:995-1272).
#pragma once

#include "spread_run.cuh"

namespace dnufft {

template <int W> struct InterpShape {
  static constexpr int SPAN = 7 + W;
  static constexpr int RT = (SPAN + 3) / 4, KT = (SPAN + 3) / 4;   // 4-row blocks, 4-column steps
  static constexpr int ROWS = 4 * RT, COLS = 4 * KT;
  // stride between staged points: 4 or 12 modulo 16 doubles (fragment reads of
  // 4 points x 4 columns of a half-warp hit all banks)
  static constexpr int ST0 = ROWS + COLS;
  static constexpr int ST = ST0 % 8 == 4 ? ST0 : ST0 + 4;
  static constexpr int BATCH = 16;
  static constexpr size_t WARP_BYTES = size_t(BATCH) * ST * sizeof(double);
};

constexpr int IR_THREADS = 128;

template <typename Tc, int W>
__global__ void __launch_bounds__(IR_THREADS, W <= 9 ? 4 : 3)
    k_interp_run(const __grid_constant__ PointsDesc pts, const uint32_t *__restrict__ sel,
                 uint32_t npts, uint32_t ppw,
                 const __grid_constant__ Geometry g, const __grid_constant__ KernelPoly<double> kp,
                 const double2 *__restrict__ grid, int64_t gtrans, double2 *__restrict__ out,
                 int64_t os, int64_t otrans) {
  using R = InterpShape<W>;
  constexpr int B = R::BATCH;
  extern __shared__ __align__(16) unsigned char smraw_run[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t first64 = (uint64_t(blockIdx.x) * (IR_THREADS / 32) + warp) * ppw;
  if (first64 >= npts) return;
  const uint32_t first = uint32_t(first64);
  const uint32_t last = uint32_t(min(uint64_t(npts), first64 + ppw));
  grid += int64_t(blockIdx.y) * gtrans;
  out += int64_t(blockIdx.y) * otrans;
  double *st = reinterpret_cast<double *>(smraw_run + warp * R::WARP_BYTES);
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]);
  // window fragments: column 4 k + lane % 4, row 4 r + lane / 8, component
  // (lane / 4) % 2
  double G[R::RT][R::KT];
  int cu = -1, cv = -1;
  bool finite = true;
  auto load_window = [&]() {
    bool ok = true;
    const int u0 = cu * 8 - g.nsafe, v0 = cv * 8 - g.nsafe;
    const double *gd = reinterpret_cast<const double *>(grid) + ((lane >> 2) & 1);
#pragma unroll
    for (int r = 0; r < R::RT; ++r) {
      const double *row = gd + 2 * int64_t(wrap3(u0 + 4 * r + (lane >> 3), n0)) * n1;
#pragma unroll
      for (int k = 0; k < R::KT; ++k) {
        G[r][k] = __ldg(row + 2 * wrap3(v0 + 4 * k + (lane & 3), n1));
        ok = ok && isfinite(G[r][k]);
      }
    }
    finite = __all_sync(0xffffffffu, ok);
  };
  const int q = lane & (B - 1), ax = lane >> 4;   // lane = 16 * axis + point
  Tc x = Tc(0);
  uint32_t j = 0;
  auto fetch = [&](uint32_t i) {
    if (i < last) {
      if (sel) i = sel[i];
      j = pts.perm[i];
      const Tc *c = static_cast<const Tc *>(pts.coord);
      x = pts.sorted ? c[uint64_t(i) * 2 + ax]
                     : c[int64_t(j) * pts.cs0 + int64_t(ax) * pts.cs1];
    }
  };
  fetch(first + q);
  for (uint32_t base = first; base < last; base += B) {
    const int np = int(min(uint32_t(B), last - base));
    {
      double2 *z = reinterpret_cast<double2 *>(st);
      constexpr int NZ = B * R::ST / 2;
#pragma unroll 4
      for (int i = lane; i < NZ; i += 32) z[i] = make_double2(0., 0.);
    }
    __syncwarp();
    int t = 0;
    if (q < np) {
      int i0;
      double frac, w[W];
      fold<Tc>(x, ax ? g.coordfct[1] : g.coordfct[0], ax ? n1 : n0, ax ? g.shift[1] : g.shift[0],
               ax ? g.maxi0[1] : g.maxi0[0], i0, frac);
      t = i0 + g.nsafe;
      kernel_weights<double, W>(kp, double(W - 1) - 2.0 * frac, w);
      double *sp = st + q * R::ST + (ax ? R::ROWS : 0) + (t & 7);
#pragma unroll
      for (int a = 0; a < W; ++a) sp[a] = w[a];
    }
    const uint32_t jq = j;
    const int bu = __shfl_sync(0xffffffffu, t, q) >> 3, bv = __shfl_sync(0xffffffffu, t, q + B) >> 3;
    fetch(base + B + q);
    int pu = __shfl_up_sync(0xffffffffu, bu, 1), pv = __shfl_up_sync(0xffffffffu, bv, 1);
    if (lane == 0) {
      pu = cu;
      pv = cv;
    }
    const unsigned bins = __ballot_sync(0xffffffffu, lane < np && (bu != pu || bv != pv));
    unsigned rest = bins & ~1u;
    __syncwarp();
    for (int s = 0; s < np;) {
      if ((bins >> s) & 1u) {
        cu = __shfl_sync(0xffffffffu, bu, s);
        cv = __shfl_sync(0xffffffffu, bv, s);
        load_window();
      }
      const int e = rest ? __ffs(rest) - 1 : np;
      rest &= rest - 1;
      if (!finite) {
        for (int p = s; p < e; ++p) {
          const int tu = __shfl_sync(0xffffffffu, t, p), tv = __shfl_sync(0xffffffffu, t, p + B);
          const double *f = st + p * R::ST;
          double sx = 0., sy = 0.;
          for (int c = lane; c < W * W; c += 32) {
            const int a = c / W, b = c - a * W;
            const double wt = f[(tu & 7) + a] * f[R::ROWS + (tv & 7) + b];
            const double2 gv = __ldg(grid + int64_t(wrap3(tu - g.nsafe + a, n0)) * n1 +
                                     wrap3(tv - g.nsafe + b, n1));
            sx += wt * gv.x;
            sy += wt * gv.y;
          }
#pragma unroll
          for (int o = 16; o; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
          }
          const uint32_t jo = __shfl_sync(0xffffffffu, jq, p);
          if (lane == 0) out[int64_t(jo) * os] = make_double2(sx, sy);
        }
        s = e;
        continue;
      }
      for (int p = s; p < e; p += 8) {
        const int pt = p + (lane >> 2);
        const bool on = pt < e;
        const double *f = st + (on ? pt : s) * R::ST;
        double a[R::KT];
#pragma unroll
        for (int k = 0; k < R::KT; ++k) a[k] = f[R::ROWS + 4 * k + (lane & 3)];
        double sx = 0., sy = 0.;
#pragma unroll
        for (int r = 0; r < R::RT; ++r) {
          double c0 = 0., c1 = 0.;
#pragma unroll
          for (int k = 0; k < R::KT; ++k)
            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                : "+d"(c0), "+d"(c1)
                : "d"(a[k]), "d"(G[r][k]));
          const double ku = f[4 * r + (lane & 3)];
          sx += ku * c0;
          sy += ku * c1;
        }
        sx += __shfl_xor_sync(0xffffffffu, sx, 1);
        sy += __shfl_xor_sync(0xffffffffu, sy, 1);
        sx += __shfl_xor_sync(0xffffffffu, sx, 2);
        sy += __shfl_xor_sync(0xffffffffu, sy, 2);
        const uint32_t jo = __shfl_sync(0xffffffffu, jq, min(pt, 15));
        if (on && (lane & 3) == 0) out[int64_t(jo) * os] = make_double2(sx, sy);
      }
      s = e;
    }
    __syncwarp();
  }
}

template <typename Tc, int W>
void interp_run_w(const PointsDesc &pts, const uint32_t *sel, uint32_t npts, const Geometry &g,
                  const KernelPoly<double> &kp, const void *grid, int64_t gtrans, void *out,
                  int64_t os, int64_t otrans, int ntrans, cudaStream_t st) {
  constexpr uint32_t NW = IR_THREADS / 32;
  const size_t sm = NW * InterpShape<W>::WARP_BYTES;
  auto kern = k_interp_run<Tc, W>;
  allow_smem(kern, sm);
  const uint32_t ppw = run_points_per_warp(uint64_t(npts) * uint64_t(ntrans), true);
  const uint64_t per = uint64_t(NW) * ppw;
  dim3 grd(unsigned((npts + per - 1) / per), ntrans);
  kern<<<grd, IR_THREADS, sm, st>>>(pts, sel, npts, ppw, g, kp, static_cast<const double2 *>(grid),
                                    gtrans, static_cast<double2 *>(out), os, otrans);
  DN_LAUNCHED();
}

}  // namespace dnufft

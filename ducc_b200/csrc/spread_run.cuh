// 2D spreading (type 1) with the window of a bin in registers.
//
// A warp takes consecutive sorted points.  The lanes fold a batch of them,
// evaluate the W weights per axis and stage, per point, the row weights ku and
// the products value * kv in shared memory, each placed in a zero-filled window
// of ROWS rows / CELLS columns.  As long as the points lie in the same bin of
// 8 x 8 grid cells, their footprints lie in that window, and the sum over the
// points of the outer products ku x (value * kv) stays in the lanes' registers:
// FP32 multiply-adds (packed in pairs) for complex64, FP64 matrix instructions
// (mma m8n8k4, four points each) for complex128.  When the bin changes the
// window is added to the grid with reductions (red.global.add) and starts
// again at zero.  Nothing is shared between warps, so there are no other
// atomics and no barriers, and any order of the points is correct; the sort
// (tile, bin: launch_fold_keys) makes the runs long.
//
// Why this split.  Per-point shared-memory atomics cost 4.3 SM cycles per warp
// operation of 32 floats (6.1 for doubles, both measured): 33 SM cycles per
// point for W = 8 in single and 404 for W = 15 in double precision.  The
// window is larger than the footprint (16 x 16 cells for 8 x 8, 24 x 24 for
// 15 x 15), but a window that starts at a fixed cell needs no indexing:
// 4 SM cycles of FP32 multiply-adds and 4 of shared-memory reads per point
// (each lane reads 4 row weights and 2 cells' products), 18 cycles of FP64 and
// 4.5 of reads.  The same with exact rows, one loop per row offset and
// compile-time registers, ran at a quarter of the speed in double precision:
// the eight loops did not fit the instruction cache.  The reductions reach
// 745 G float2 cells/s (342 G double2, measured), 96 SM cycles of L2 time per
// 16 x 16 window; cells that no point touched are not sent, so a bin with one
// point costs about the same as adding its footprint directly.
//
// Measured (spreading alone, per-point shared atomics before): 5e7 clustered
// points, 8400^2 cells, complex64, W = 8: 5.9 -> 2.02 ms (3.49 ms in the
// tensor-core spreader), 87 % of the shared-memory pipe's cycles; 5e6 points,
// 2880^2 cells, complex128, W = 15: 7.18 -> 0.96 ms.
//
// A point whose value is not finite is added to its footprint alone: zero
// weights times an infinite value would spoil the rest of the window.
//
// Mirrors HelperNu2u / spreading_helper (src/ducc0/nufft/nufft.h:917-1204).
#pragma once

#include <algorithm>

#include "spread_impl.cuh"

namespace dnufft {

template <typename T, int W> struct RunShape {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int SPAN = 7 + W;                            // cells a bin's points touch per axis
  static constexpr int MT = (SPAN + 7) / 8, NT = (SPAN + 3) / 4;   // 8-row, 4-cell blocks
  static constexpr int ROWS = F32 ? 16 : 8 * MT;
  static constexpr int CELLS = F32 ? 16 : 4 * NT;
  // stride between staged points.  float: an odd number of 16-byte words
  // (conflict-free zeroing); double: 4 or 12 modulo 16 words, so that the 4
  // points x 4 rows of a half-warp's fragment reads hit all banks
  static constexpr int ST = ROWS + 2 * CELLS + 4;
  static constexpr int BATCH = F32 ? 32 : 16;                   // points staged at a time
  static constexpr size_t WARP_BYTES = size_t(BATCH) * ST * sizeof(T);
  // registers of the window: float: 8 rows x 2 components (row pairs packed);
  // double: the MT x NT accumulator fragments
  static constexpr int NACC = F32 ? 8 : 2 * MT * NT;
};

template <typename T> constexpr int run_threads() { return sizeof(T) == 4 ? 256 : 128; }
// CTAs per SM the registers must allow: float 3 (77 registers; at 4 the window
// spills, 2.31 against 2.02 ms at 5e7 points, W = 8), double 4 (of 4 warps, 128
// registers; 3: 1.00 against 0.96 ms at 5e6 points, W = 15)
template <typename T> constexpr int run_min_ctas() { return sizeof(T) == 4 ? 3 : 4; }

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}

// The window of the current bin: adds points [s, e) of the staged batch,
// flushes itself to the grid.  A window starts in [-nsafe, n + 1 - nsafe], n >= 2
// nsafe, and is at most 24 cells wide, so its cells lie in [-n, 4n); beyond 3n only
// those of 16 cells at n = 4, which only W = 4 has.
template <typename T, int W> struct RunWindow;

template <int W> __host__ __device__ __forceinline__ int run_wrap(int i, int n) {
  return W == 4 ? wrap3(i, n) : wrap2(i, n);
}

// float: each lane has rows 4 rg .. + 3 of the cells cg and cg + 8, with rg =
// lane bit 0 and bit 4, cg = lane bits 1..3: at most two addresses among four
// neighbouring lanes, so that a 16-byte read takes 2 SM cycles and an 8-byte
// one 1 (half of what distinct addresses take)
template <int W> struct RunWindow<float, W> {
  using R = RunShape<float, W>;
  unsigned long long c[2][4];   // (re, im) of a cell packed, [cell][row]
  static __device__ __forceinline__ int row0(int lane) { return 4 * ((lane & 1) | ((lane >> 4) << 1)); }
  static __device__ __forceinline__ int cell0(int lane) { return (lane >> 1) & 7; }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 4; ++i) c[0][i] = c[1][i] = 0ull;
  }
  __device__ __forceinline__ void add(const float *st, int s, int e, int lane) {
    const float *kr = st + row0(lane), *tc = st + R::ROWS + 2 * cell0(lane);
#pragma unroll 4
    for (int p = s; p < e; ++p) {
      const float4 k = *reinterpret_cast<const float4 *>(kr + p * R::ST);
      const unsigned long long t0 = *reinterpret_cast<const unsigned long long *>(tc + p * R::ST);
      const unsigned long long t1 =
          *reinterpret_cast<const unsigned long long *>(tc + p * R::ST + 16);
      const unsigned long long kk[4] = {pack2(k.x, k.x), pack2(k.y, k.y), pack2(k.z, k.z),
                                        pack2(k.w, k.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[0][i]) : "l"(kk[i]), "l"(t0));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[1][i]) : "l"(kk[i]), "l"(t1));
      }
    }
  }
  __device__ __forceinline__ void flush(float2 *grid, int u0, int v0, int n0, int n1, bool inside,
                                        int lane) {
    const int ru = u0 + row0(lane), va = v0 + cell0(lane);
    float2 *pa = grid + (inside ? va : run_wrap<W>(va, n1)), *pb = grid + (inside ? va + 8 : run_wrap<W>(va + 8, n1));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t off = int64_t(inside ? ru + i : run_wrap<W>(ru + i, n0)) * n1;
      const float2 a = unpack2(c[0][i]), b = unpack2(c[1][i]);
      if (a.x != 0.f || a.y != 0.f) atomicAdd(pa + off, a);
      if (b.x != 0.f || b.y != 0.f) atomicAdd(pb + off, b);
    }
    clear();
  }
};

// double: accumulator fragments of the row block m and the cell block n: row
// 8 m + lane / 4, cell 4 n + lane % 4 (both components)
template <int W> struct RunWindow<double, W> {
  using R = RunShape<double, W>;
  double c[R::MT][R::NT][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int m = 0; m < R::MT; ++m)
#pragma unroll
      for (int n = 0; n < R::NT; ++n) c[m][n][0] = c[m][n][1] = 0.;
  }
  __device__ __forceinline__ void add(const double *st, int s, int e, int lane) {
    const double *fr = st + (lane & 3) * R::ST + (lane >> 2);
#pragma unroll 1
    for (int p = s; p < e; p += 4) {
      const bool on = p + (lane & 3) < e;
      const double *f = fr + p * R::ST;
      double a[R::MT], b[R::NT];
#pragma unroll
      for (int m = 0; m < R::MT; ++m) a[m] = on ? f[8 * m] : 0.;
#pragma unroll
      for (int n = 0; n < R::NT; ++n) b[n] = on ? f[R::ROWS + 8 * n] : 0.;
#pragma unroll
      for (int m = 0; m < R::MT; ++m)
#pragma unroll
        for (int n = 0; n < R::NT; ++n)
          asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
              : "+d"(c[m][n][0]), "+d"(c[m][n][1])
              : "d"(a[m]), "d"(b[n]));
    }
  }
  __device__ __forceinline__ void flush(double2 *grid, int u0, int v0, int n0, int n1, bool inside,
                                        int lane) {
    const int ru = u0 + (lane >> 2), cv = v0 + (lane & 3);
#pragma unroll
    for (int m = 0; m < R::MT; ++m) {
      double2 *row = grid + int64_t(inside ? ru + 8 * m : wrap3(ru + 8 * m, n0)) * n1;
#pragma unroll
      for (int n = 0; n < R::NT; ++n) {
        double2 *q = row + (inside ? cv + 4 * n : wrap3(cv + 4 * n, n1));
        if (c[m][n][0] != 0.) atomicAdd(&q->x, c[m][n][0]);
        if (c[m][n][1] != 0.) atomicAdd(&q->y, c[m][n][1]);
      }
    }
    clear();
  }
};

// points [first, last) of the sorted order, by one warp; sel (may be null):
// sorted position of the i-th point to spread
template <typename T, typename Tc, int W>
__device__ __forceinline__ void spread_run(const PointsDesc &pts, const uint32_t *__restrict__ sel,
                                           const Geometry &g, const KernelPoly<T> &kp,
                                           const cplx<T> *__restrict__ values, int64_t vs,
                                           cplx<T> *__restrict__ grid, uint32_t first,
                                           uint32_t last, unsigned char *sm) {
  using R = RunShape<T, W>;
  constexpr int B = R::BATCH;
  const int lane = threadIdx.x & 31;
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]);
  T *st = reinterpret_cast<T *>(sm);
  RunWindow<T, W> win;
  win.clear();
  int cu = -1, cv = -1;   // bin of the window
  auto flush = [&]() {
    const int u0 = cu * 8 - g.nsafe, v0 = cv * 8 - g.nsafe;
    const bool inside = u0 >= 0 && u0 + R::ROWS <= n0 && v0 >= 0 && v0 + R::CELLS <= n1;
    win.flush(grid, u0, v0, n0, n1, inside, lane);
  };
  // float: lane = point; double: lane = 16 * axis + point
  const int q = lane & (B - 1);
  const int ax = R::F32 ? 0 : lane >> 4;
  Tc x[2] = {Tc(0), Tc(0)};
  cplx<T> v = mkc<T>(T(0), T(0));
  auto fetch = [&](uint32_t i) {
    if (i < last) {
      const uint32_t j = load_point<Tc, 2>(pts, sel ? sel[i] : i, x);
      // a gather through the permutation: cached in L2 only, so a miss
      // brings one 32-byte sector instead of a whole L1 line
      v = __ldcg(values + int64_t(j) * vs);
    }
  };
  fetch(first + q);
  for (uint32_t base = first; base < last; base += B) {
    const int np = int(min(uint32_t(B), last - base));
    // zero windows
    {
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 *z4 = reinterpret_cast<float4 *>(st);
      constexpr int NZ = int(R::WARP_BYTES / 16);
#pragma unroll 4
      for (int i = lane; i < NZ; i += 32) z4[i] = z;
    }
    __syncwarp();
    const bool bad = q < np && !(isfinite(v.x) && isfinite(v.y));
    const cplx<T> val = bad ? mkc<T>(T(1), T(0)) : v;
    int tu = 0, tv = 0;
    if (q < np) {
      T *sp = st + q * R::ST;
      int i0;
      double frac;
      T w[W];
      if constexpr (R::F32) {
        fold<Tc>(x[0], g.coordfct[0], n0, g.shift[0], g.maxi0[0], i0, frac);
        tu = i0 + g.nsafe;
        kernel_weights<T, W>(kp, T(double(W - 1) - 2.0 * frac), w);
        T *sr = sp + (tu & 7);
#pragma unroll
        for (int a = 0; a < W; ++a) sr[a] = w[a];
        fold<Tc>(x[1], g.coordfct[1], n1, g.shift[1], g.maxi0[1], i0, frac);
        tv = i0 + g.nsafe;
        kernel_weights<T, W>(kp, T(double(W - 1) - 2.0 * frac), w);
        cplx<T> *sc = reinterpret_cast<cplx<T> *>(sp + R::ROWS) + (tv & 7);
#pragma unroll
        for (int a = 0; a < W; ++a) sc[a] = mkc<T>(w[a] * val.x, w[a] * val.y);
      } else {
        fold<Tc>(ax ? x[1] : x[0], ax ? g.coordfct[1] : g.coordfct[0], ax ? n1 : n0,
                 ax ? g.shift[1] : g.shift[0], ax ? g.maxi0[1] : g.maxi0[0], i0, frac);
        tu = i0 + g.nsafe;
        kernel_weights<T, W>(kp, T(double(W - 1) - 2.0 * frac), w);
        if (ax == 0) {
          T *sr = sp + (tu & 7);
#pragma unroll
          for (int a = 0; a < W; ++a) sr[a] = w[a];
        } else {
          cplx<T> *sc = reinterpret_cast<cplx<T> *>(sp + R::ROWS) + (tu & 7);
#pragma unroll
          for (int a = 0; a < W; ++a) sc[a] = mkc<T>(w[a] * val.x, w[a] * val.y);
        }
      }
    }
    if constexpr (!R::F32) {
      // both axes' cells to every lane of the point
      const int t = tu;
      tu = __shfl_sync(0xffffffffu, t, q);
      tv = __shfl_sync(0xffffffffu, t, q + B);
    }
    unsigned badmask = __ballot_sync(0xffffffffu, bad && lane < B);
    while (badmask) {
      // not finite (staged with value 1): straight into the grid, then zero
      // row weights
      __syncwarp();
      const int p = __ffs(badmask) - 1;
      badmask &= badmask - 1;
      const int su = __shfl_sync(0xffffffffu, tu, p), sv = __shfl_sync(0xffffffffu, tv, p);
      const T vx = __shfl_sync(0xffffffffu, v.x, p), vy = __shfl_sync(0xffffffffu, v.y, p);
      T *sp = st + p * R::ST;
      for (int c = lane; c < W * W; c += 32) {
        const int a = c / W, b = c - a * W;
        const T wt = sp[(su & 7) + a] * sp[R::ROWS + 2 * ((sv & 7) + b)];
        global_add<T>(grid + int64_t(wrap2(su - g.nsafe + a, n0)) * n1 +
                          wrap2(sv - g.nsafe + b, n1),
                      wt * vx, wt * vy);
      }
      __syncwarp();
      if (lane < R::ROWS) sp[lane] = T(0);
    }
    fetch(base + B + q);   // the next batch, while this one is added
    // points whose bin differs from the one before
    const int bu = tu >> 3, bv = tv >> 3;
    int pu = __shfl_up_sync(0xffffffffu, bu, 1), pv = __shfl_up_sync(0xffffffffu, bv, 1);
    if (lane == 0) {
      pu = cu;
      pv = cv;
    }
    const unsigned bins = __ballot_sync(0xffffffffu, lane < np && (bu != pu || bv != pv));
    __syncwarp();
    int s = 0;
    unsigned rest = bins;
    while (s < np) {
      if ((bins >> s) & 1u) {
        if (cu >= 0) flush();
        cu = __shfl_sync(0xffffffffu, bu, s);
        cv = __shfl_sync(0xffffffffu, bv, s);
        rest &= ~(1u << s);
      }
      const int e = rest ? __ffs(rest) - 1 : np;
      win.add(st, s, e, lane);
      s = e;
    }
    __syncwarp();
  }
  if (cu >= 0) flush();
}

// Points per warp: about 24 warps per SM get work before longer runs save flushes; a
// multiple of 32 from 32 up, at least 8 (few points: a warp adds its points one after
// the other, so more warps finish sooner).  waves: where runs of 128 points and more
// would make little more than one wave of warps, a third of that length: warps in
// thin and in dense places take times of their own, and a wave lasts as long as its
// slowest (1e6 points, one wave / three, us: complex64 spreading of clustered points
// on 2420^2 cells 188 / 96, 4116^2 222 / 121, evenly spread 203 / 167, complex128
// interpolation of clustered points on 1890^2 211 / 109).  Not for complex128
// spreading, whose flushes cost more (clustered on 224^2: 118 / 211; thinly spread
// ones would gain, 248 / 139 on 1890^2), nor for fewer points (3e5 on 1050^2: 50 / 53).
inline uint32_t run_points_per_warp(uint64_t npts, bool waves) {
  uint64_t p = npts / (148 * 24);
  if (waves && p >= 128) p = std::max<uint64_t>(64, p / 3);
  return uint32_t(p < 32 ? std::max<uint64_t>(8, p & ~uint64_t(7))
                         : std::min<uint64_t>(256, p & ~uint64_t(31)));
}

template <typename T, typename Tc, int W>
__global__ void __launch_bounds__(run_threads<T>(), run_min_ctas<T>())
    k_spread_run(const __grid_constant__ PointsDesc pts, const uint32_t *__restrict__ sel,
                 uint32_t npts, uint32_t ppw, const __grid_constant__ Geometry g,
                 const __grid_constant__ KernelPoly<T> kp, const cplx<T> *__restrict__ values,
                 int64_t vs, int64_t vtrans, cplx<T> *__restrict__ grid, int64_t gtrans) {
  extern __shared__ __align__(16) unsigned char smraw_run[];
  constexpr uint32_t NW = run_threads<T>() / 32;
  const uint32_t warp = threadIdx.x >> 5;
  const uint64_t first = (uint64_t(blockIdx.x) * NW + warp) * ppw;
  if (first >= npts) return;
  spread_run<T, Tc, W>(pts, sel, g, kp, values + int64_t(blockIdx.y) * vtrans, vs,
                       grid + int64_t(blockIdx.y) * gtrans, uint32_t(first),
                       uint32_t(min(uint64_t(npts), first + ppw)),
                       smraw_run + warp * RunShape<T, W>::WARP_BYTES);
}

template <typename T, typename Tc, int W>
void spread_run_w(const PointsDesc &pts, const uint32_t *sel, uint32_t npts, const Geometry &g,
                  const KernelPoly<T> &kp, const void *values, int64_t vs, int64_t vtrans,
                  void *grid, int64_t gtrans, int ntrans, cudaStream_t st) {
  constexpr uint32_t NW = run_threads<T>() / 32;
  const size_t sm = NW * RunShape<T, W>::WARP_BYTES;
  auto kern = k_spread_run<T, Tc, W>;
  allow_smem(kern, sm);
  const uint32_t ppw = run_points_per_warp(uint64_t(npts) * uint64_t(ntrans), sizeof(T) == 4);
  const uint64_t per = uint64_t(NW) * ppw;
  dim3 grd(unsigned((npts + per - 1) / per), ntrans);
  kern<<<grd, run_threads<T>(), sm, st>>>(pts, sel, npts, ppw, g, kp,
                                          static_cast<const cplx<T> *>(values), vs, vtrans,
                                          static_cast<cplx<T> *>(grid), gtrans);
  DN_LAUNCHED();
}

template <typename T>
void launch_spread_run_impl(const PointsDesc &pts, const uint32_t *sel, uint32_t npts,
                            const Geometry &g, const KernelPoly<T> &kp, const void *values,
                            int64_t vs, int64_t vtrans, void *grid, int64_t gtrans, int ntrans,
                            cudaStream_t st) {
  if (npts == 0 || ntrans == 0) return;
#define DN_CASE(WW)                                                                              \
  case WW:                                                                                       \
    if (pts.coord_f64)                                                                           \
      spread_run_w<T, double, WW>(pts, sel, npts, g, kp, values, vs, vtrans, grid, gtrans,       \
                                  ntrans, st);                                                   \
    else                                                                                         \
      spread_run_w<T, float, WW>(pts, sel, npts, g, kp, values, vs, vtrans, grid, gtrans,        \
                                 ntrans, st);                                                    \
    return;
  if constexpr (sizeof(T) == 4) {
    switch (g.W) { DN_FOR_W_FLOAT(DN_CASE) }
  } else {
    switch (g.W) { DN_FOR_W_DOUBLE(DN_CASE) }
  }
#undef DN_CASE
  throw Error(ST_UNSUPPORTED, "kernel support not supported by this build");
}

}  // namespace dnufft

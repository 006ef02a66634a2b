// 3D spreading (type 1) with the window of a bin in registers.
//
// The 3D form of spread_run.cuh: a point adds the plane ku[a] * (kv x (value *
// kw)) to W consecutive planes of the window of its bin (8^3 cells; 4^3 for
// W > 12, whose window would not fit the registers).  A CTA takes consecutive
// sorted points, stages a batch of them in shared memory (zero-filled windows of
// plane, row and column weights), and every warp adds all of the batch's points
// to its own planes, kept in registers:
//   complex64: 4 warps, warp r has planes r, r + 4, r + 8, r + 12; a point adds
//     to two neighbouring ones of them, sharing the row and column operands (FP32
//     multiply-adds packed in pairs, operand layout of the 2D form).  Which two
//     depends on its plane in the bin; the sort keeps points of equal plane
//     together, and a loop for each of the three pairs has no branches inside;
//   complex128: one warp per plane, FP64 matrix instructions over four points;
//     planes that none of the four touches are skipped (the sort keeps points of
//     equal u together).
// When the bin changes, every warp adds its planes to the grid with reductions.
// No other atomics; warps meet only when a batch is staged.
//
// Before, a W = 8 complex64 point cost 1024 shared-memory atomics (633 SM cycles)
// and a W = 12 complex128 point 3456 global ones (3090 SM cycles); here 40 SM
// cycles of FP32 and 175 of FP64 multiply-adds, 51 and 107 reductions of a cell at
// one point per 8 cells.  Measured in all: 94 (1e7 points, 256^3 cells, 3.3 ms) and
// 384 (1e6 points, 1.35 ms): the adding warps wait while a batch is staged (no
// overlap inside a CTA; 16 and 19 warps per SM), issue is active 58 % and 43 % of
// the cycles, the double-precision matrix pipe 48 %.
//
// Mirrors HelperNu2u / spreading_helper (src/ducc0/nufft/nufft.h:1391-1649).
#pragma once

#include "spread_run.cuh"

namespace dnufft {

// cells per axis of a bin (log2), by support
constexpr int run3_bin_log2(int W) { return W <= 12 ? 3 : 2; }

template <typename T, int W> struct Run3Shape {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int LB = run3_bin_log2(W), BIN = 1 << LB;
  static constexpr int SPAN = BIN - 1 + W;
  static constexpr int MT = (SPAN + 7) / 8, NT = (SPAN + 3) / 4;
  static constexpr int PLANES = F32 ? 16 : (SPAN + 1) / 2 * 2;   // staged plane weights
  static constexpr int ROWS = F32 ? 16 : 8 * MT;
  static constexpr int CELLS = F32 ? 16 : 4 * NT;
  static constexpr int WARPS = F32 ? 4 : SPAN;
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int BATCH = F32 ? 128 : (W <= 9 ? 64 : 128);
  // float: an odd number of 16-byte words; double: 4 or 12 modulo 16 words
  static constexpr int ST0 = PLANES + ROWS + 2 * CELLS;
  static constexpr int ST = F32 ? ST0 + 4 : ST0 + (ST0 % 8 == 4 ? 0 : (12 - ST0 % 8) % 8);
  static constexpr size_t SMEM = size_t(BATCH) * ST * sizeof(T) + size_t(BATCH) * sizeof(int4);
  static_assert(F32 || ST % 8 == 4, "fragment reads would conflict");
};

// float: planes of warp r; the rest as RunWindow<float>
template <typename T, int W> struct Run3Window;

template <int W> struct Run3Window<float, W> {
  using R = Run3Shape<float, W>;
  using L = RunWindow<float, W>;
  unsigned long long c[4][2][4];   // [plane][cell][row]
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) c[j][0][i] = c[j][1][i] = 0ull;
  }
  // slot of plane weight i (of 16): the four planes of a warp side by side
  static __device__ __forceinline__ int plane_slot(int i) { return (i & 3) * 4 + (i >> 2); }
  // the warp's first plane at or after plane ou of the window
  static __device__ __forceinline__ int first_plane(int ou, int warp) { return (ou - warp + 3) >> 2; }
  // points [s, e), whose footprints start at planes of the same first_plane
  __device__ __forceinline__ void add(const float *st, int s, int e, int ou, int warp, int lane) {
    const int j0 = first_plane(ou, warp);
    if (j0 == 0) add_pair<0>(st, s, e, warp, lane);
    else if (j0 == 1) add_pair<1>(st, s, e, warp, lane);
    else add_pair<2>(st, s, e, warp, lane);
  }
  // planes of a warp that a footprint touches: one at W = 4 (2e6 points, 112^3
  // cells: 527 us with the second, always zero one, 357 without)
  static constexpr int NP = W <= 4 ? 1 : 2;
  template <int J0>
  __device__ __forceinline__ void add_pair(const float *st, int s, int e, int warp, int lane) {
    const float *pk = st + 4 * warp + J0, *kr = st + R::PLANES + L::row0(lane),
                *tc = st + R::PLANES + R::ROWS + 2 * L::cell0(lane);
#pragma unroll 2
    for (int p = s; p < e; ++p) {
      float kj[NP];
#pragma unroll
      for (int j = 0; j < NP; ++j) kj[j] = pk[p * R::ST + j];
      const float4 k = *reinterpret_cast<const float4 *>(kr + p * R::ST);
      const unsigned long long t0 = *reinterpret_cast<const unsigned long long *>(tc + p * R::ST);
      const unsigned long long t1 =
          *reinterpret_cast<const unsigned long long *>(tc + p * R::ST + 16);
      const unsigned long long kk[4] = {pack2(k.x, k.x), pack2(k.y, k.y), pack2(k.z, k.z),
                                        pack2(k.w, k.w)};
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const unsigned long long m = pack2(kj[j], kj[j]);
        unsigned long long a0, a1;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(a0) : "l"(t0), "l"(m));
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(a1) : "l"(t1), "l"(m));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[J0 + j][0][i]) : "l"(kk[i]), "l"(a0));
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c[J0 + j][1][i]) : "l"(kk[i]), "l"(a1));
        }
      }
    }
  }
  __device__ __forceinline__ void flush(float2 *grid, int u0, int v0, int w0, int n0, int n1,
                                        int n2, int warp, int lane) {
    const int rv = v0 + L::row0(lane), wa = w0 + L::cell0(lane);
    const int ca = wrap3(wa, n2), cb = wrap3(wa + 8, n2);
    int64_t row[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) row[i] = int64_t(wrap3(rv + i, n1)) * n2;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 *pl = grid + int64_t(wrap3(u0 + warp + 4 * j, n0)) * n1 * n2;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = unpack2(c[j][0][i]), b = unpack2(c[j][1][i]);
        if (a.x != 0.f || a.y != 0.f) atomicAdd(pl + row[i] + ca, a);
        if (b.x != 0.f || b.y != 0.f) atomicAdd(pl + row[i] + cb, b);
      }
    }
    clear();
  }
};

// double: the fragments of one plane
template <int W> struct Run3Window<double, W> {
  using R = Run3Shape<double, W>;
  double c[R::MT][R::NT][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int m = 0; m < R::MT; ++m)
#pragma unroll
      for (int n = 0; n < R::NT; ++n) c[m][n][0] = c[m][n][1] = 0.;
  }
  static __device__ __forceinline__ int plane_slot(int i) { return i; }
  __device__ __forceinline__ void add(const double *st, int s, int e, int ou, int warp, int lane) {
    const double *pt = st + (lane & 3) * R::ST;
#pragma unroll 1
    for (int p = s; p < e; p += 4) {
      const bool on = p + (lane & 3) < e;
      const double *f = pt + p * R::ST;
      const double ku = on ? f[warp] : 0.;
      if (!__any_sync(0xffffffffu, ku != 0.)) continue;
      const double *fr = f + R::PLANES + (lane >> 2);
      double a[R::MT], b[R::NT];
#pragma unroll
      for (int m = 0; m < R::MT; ++m) a[m] = on ? fr[8 * m] * ku : 0.;
#pragma unroll
      for (int n = 0; n < R::NT; ++n) b[n] = on ? fr[R::ROWS + 8 * n] : 0.;
#pragma unroll
      for (int m = 0; m < R::MT; ++m)
#pragma unroll
        for (int n = 0; n < R::NT; ++n)
          asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
              : "+d"(c[m][n][0]), "+d"(c[m][n][1])
              : "d"(a[m]), "d"(b[n]));
    }
  }
  __device__ __forceinline__ void flush(double2 *grid, int u0, int v0, int w0, int n0, int n1,
                                        int n2, int warp, int lane) {
    double2 *pl = grid + int64_t(wrap3(u0 + warp, n0)) * n1 * n2;
    const int rv = v0 + (lane >> 2), cw = w0 + (lane & 3);
#pragma unroll
    for (int m = 0; m < R::MT; ++m) {
      double2 *row = pl + int64_t(wrap3(rv + 8 * m, n1)) * n2;
#pragma unroll
      for (int n = 0; n < R::NT; ++n) {
        double2 *q = row + wrap3(cw + 4 * n, n2);
        if (c[m][n][0] != 0.) atomicAdd(&q->x, c[m][n][0]);
        if (c[m][n][1] != 0.) atomicAdd(&q->y, c[m][n][1]);
      }
    }
    clear();
  }
};

template <typename T, typename Tc, int W>
__global__ void __launch_bounds__(Run3Shape<T, W>::THREADS)
    k_spread_run3(const __grid_constant__ PointsDesc pts, uint32_t ppb,
                  const __grid_constant__ Geometry g, const __grid_constant__ KernelPoly<T> kp,
                  const cplx<T> *__restrict__ values, int64_t vs, int64_t vtrans,
                  cplx<T> *__restrict__ grid, int64_t gtrans) {
  using R = Run3Shape<T, W>;
  constexpr int B = R::BATCH;
  extern __shared__ __align__(16) unsigned char smraw_run[];
  __shared__ int s_bad;
  T *st = reinterpret_cast<T *>(smraw_run);
  // every staged point: cell of the first axis, bins of the other two, and
  // whether its value is not finite
  int4 *info = reinterpret_cast<int4 *>(st + size_t(B) * R::ST);
  values += int64_t(blockIdx.y) * vtrans;
  grid += int64_t(blockIdx.y) * gtrans;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]), n2 = int(g.nover[2]);
  const uint32_t first = blockIdx.x * ppb;
  const uint32_t last = uint32_t(min(uint64_t(pts.npts), uint64_t(first) + ppb));
  Run3Window<T, W> win;
  win.clear();
  int cu = -1, cv = -1, cw = -1;   // bin of the window
  auto flush = [&]() {
    win.flush(grid, cu * R::BIN - g.nsafe, cv * R::BIN - g.nsafe, cw * R::BIN - g.nsafe, n0, n1,
              n2, warp, lane);
  };
  for (uint32_t base = first; base < last; base += B) {
    const int np = int(min(uint32_t(B), last - base));
    __syncthreads();   // the last batch has been added
    {
      float4 *z4 = reinterpret_cast<float4 *>(st);
      const int nz = np * (R::ST * int(sizeof(T)) / 16);
      for (int i = tid; i < nz; i += R::THREADS) z4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tid == 0) s_bad = 0;
    }
    __syncthreads();
    // one (point, axis) per thread and step
    for (int it = tid; it < 3 * B; it += R::THREADS) {
      const int ax = it / B, q = it - ax * B;
      if (q >= np) continue;
      const uint32_t i = base + uint32_t(q);
      const uint32_t j = pts.perm[i];
      const Tc *c = static_cast<const Tc *>(pts.coord);
      const Tc x = pts.sorted ? c[uint64_t(i) * 3 + ax]
                              : c[int64_t(j) * pts.cs0 + int64_t(ax) * pts.cs1];
      cplx<T> v = mkc<T>(T(1), T(0));
      bool bad = false;
      if (ax == 2) {
        v = __ldcg(values + int64_t(j) * vs);
        bad = !(isfinite(v.x) && isfinite(v.y));
        if (bad) {
          v = mkc<T>(T(1), T(0));
          s_bad = 1;
        }
      }
      int i0;
      double frac;
      T w[W];
      fold<Tc>(x, ax == 0 ? g.coordfct[0] : (ax == 1 ? g.coordfct[1] : g.coordfct[2]),
               ax == 0 ? n0 : (ax == 1 ? n1 : n2),
               ax == 0 ? g.shift[0] : (ax == 1 ? g.shift[1] : g.shift[2]),
               ax == 0 ? g.maxi0[0] : (ax == 1 ? g.maxi0[1] : g.maxi0[2]), i0, frac);
      kernel_weights<T, W>(kp, T(double(W - 1) - 2.0 * frac), w);
      const int t = i0 + g.nsafe,
                o = t & (R::BIN - 1);
      T *sp = st + q * R::ST;
      int *inf = reinterpret_cast<int *>(info + q);
      inf[ax] = ax == 0 ? t : t >> R::LB;
      if (ax == 0) {
#pragma unroll
        for (int a = 0; a < W; ++a) sp[Run3Window<T, W>::plane_slot(o + a)] = w[a];
      } else if (ax == 1) {
#pragma unroll
        for (int a = 0; a < W; ++a) sp[R::PLANES + o + a] = w[a];
      } else {
        inf[3] = bad ? 1 : 0;
        cplx<T> *sc = reinterpret_cast<cplx<T> *>(sp + R::PLANES + R::ROWS) + o;
#pragma unroll
        for (int a = 0; a < W; ++a) sc[a] = mkc<T>(w[a] * v.x, w[a] * v.y);
      }
    }
    __syncthreads();
    if (s_bad) {
      // values that are not finite (staged as 1): straight into the grid, the
      // nonzero weights of the window only, then zero plane weights
      for (int q = 0; q < np; ++q) {
        if (!info[q].w) continue;
        const T *sp = st + q * R::ST;
        const cplx<T> v = __ldcg(values + int64_t(pts.perm[base + q]) * vs);
        const int u0 = (info[q].x >> R::LB) * R::BIN - g.nsafe, v0 = info[q].y * R::BIN - g.nsafe,
                  w0 = info[q].z * R::BIN - g.nsafe;
        for (int c = tid; c < R::SPAN * R::SPAN * R::SPAN; c += R::THREADS) {
          const int a = c / (R::SPAN * R::SPAN), r = c - a * (R::SPAN * R::SPAN), b = r / R::SPAN,
                    e = r - b * R::SPAN;
          const T wt = sp[Run3Window<T, W>::plane_slot(a)] * sp[R::PLANES + b] *
                       sp[R::PLANES + R::ROWS + 2 * e];
          if (wt != T(0))
            global_add<T>(grid + (int64_t(wrap3(u0 + a, n0)) * n1 + wrap3(v0 + b, n1)) * n2 +
                              wrap3(w0 + e, n2),
                          wt * v.x, wt * v.y);
        }
      }
      __syncthreads();
      for (int i = tid; i < np * R::PLANES; i += R::THREADS) {
        const int q = i / R::PLANES;
        if (info[q].w) st[q * R::ST + (i - q * R::PLANES)] = T(0);
      }
      __syncthreads();
    }
    for (int s0 = 0; s0 < np; s0 += 32) {
      // points whose bin, or (float) first plane of this warp in it, differs from
      // the one before
      const int p = s0 + lane, ns = min(32, np - s0);
      const int4 b = info[min(p, np - 1)];
      int pu = __shfl_up_sync(0xffffffffu, b.x, 1), pv = __shfl_up_sync(0xffffffffu, b.y, 1),
          pw = __shfl_up_sync(0xffffffffu, b.z, 1);
      if (lane == 0) {
        pu = cu * R::BIN;
        pv = cv;
        pw = cw;
      }
      const unsigned bins = __ballot_sync(
          0xffffffffu, p < np && ((b.x >> R::LB) != (pu >> R::LB) || b.y != pv || b.z != pw));
      unsigned rest = bins;
      if constexpr (R::F32) {
        const int j0 = Run3Window<T, W>::first_plane(b.x & (R::BIN - 1), warp);
        const int pj = __shfl_up_sync(0xffffffffu, j0, 1);
        rest |= __ballot_sync(0xffffffffu, p < np && lane > 0 && j0 != pj);
      }
      rest &= ~1u;
      for (int s = 0; s < ns;) {
        if ((bins >> s) & 1u) {
          if (cu >= 0) flush();
          cu = __shfl_sync(0xffffffffu, b.x, s) >> R::LB;
          cv = __shfl_sync(0xffffffffu, b.y, s);
          cw = __shfl_sync(0xffffffffu, b.z, s);
        }
        const int e = rest ? __ffs(rest) - 1 : ns;
        rest &= rest - 1;
        const int ou = __shfl_sync(0xffffffffu, b.x, s) & (R::BIN - 1);
        win.add(st, s0 + s, s0 + e, ou, warp, lane);
        s = e;
      }
    }
  }
  if (cu >= 0) flush();
}

template <typename T, typename Tc, int W>
void spread_run3_w(const PointsDesc &pts, const Geometry &g, const KernelPoly<T> &kp,
                   const void *values, int64_t vs, int64_t vtrans, void *grid, int64_t gtrans,
                   int ntrans, cudaStream_t st) {
  using R = Run3Shape<T, W>;
  auto kern = k_spread_run3<T, Tc, W>;
  allow_smem(kern, R::SMEM);
  // points per CTA: up to eight batches where that leaves 8 CTAs per SM, down
  // to 16 points for few points (the CTAs walk them one after the other)
  const uint64_t per = uint64_t(pts.npts) * uint64_t(ntrans) / (148 * 8);
  const uint32_t ppb =
      per >= R::BATCH ? R::BATCH * uint32_t(std::min<uint64_t>(8, per / R::BATCH))
                      : std::max<uint32_t>(16, uint32_t(per) & ~15u);
  dim3 grd(unsigned((uint64_t(pts.npts) + ppb - 1) / ppb), ntrans);
  kern<<<grd, R::THREADS, R::SMEM, st>>>(pts, ppb, g, kp, static_cast<const cplx<T> *>(values), vs,
                                         vtrans, static_cast<cplx<T> *>(grid), gtrans);
  DN_LAUNCHED();
}

template <typename T>
void launch_spread_run3_impl(const PointsDesc &pts, const Geometry &g, const KernelPoly<T> &kp,
                             const void *values, int64_t vs, int64_t vtrans, void *grid,
                             int64_t gtrans, int ntrans, cudaStream_t st) {
  if (pts.npts == 0 || ntrans == 0) return;
#define DN_CASE(WW)                                                                            \
  case WW:                                                                                     \
    if (pts.coord_f64)                                                                         \
      spread_run3_w<T, double, WW>(pts, g, kp, values, vs, vtrans, grid, gtrans, ntrans, st);  \
    else                                                                                       \
      spread_run3_w<T, float, WW>(pts, g, kp, values, vs, vtrans, grid, gtrans, ntrans, st);   \
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

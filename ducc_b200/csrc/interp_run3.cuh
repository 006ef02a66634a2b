// 3D interpolation (type 2) with the window of a bin in registers: the
// transpose of spread_run3.cuh.  Double precision first, single below.
//
// A CTA takes consecutive sorted points and has one warp per plane of the window
// of their bin (8^3 cells, 4^3 for W > 12).  A batch of points is staged in
// shared memory (plane, row and column weights, zero-filled to the window); every
// warp keeps its plane of the grid in the fragments of FP64 matrix instructions
// (as k_interp_run), forms the points' sums over the plane eight at a time
// (skipping those whose footprints do not touch it) and leaves them, times the
// plane weight, in shared memory, where they are added over the planes.
//
// Reading W^3 cells of 16 bytes through L1 per point took 700 SM cycles per point
// at W = 12; the matrix instructions take 165, all of it 426 (1e6 points, 1.5 ms: the
// matrix pipe is active 45 % of the cycles, the warps of the one CTA that fits an SM
// wait for staging and at its barriers).  Small supports and thinly spread
// points are left to that direct form (k_interp_direct3).
//
// Mirrors HelperU2nu / interpolation_helper (src/ducc0/nufft/nufft.h:1508-1729).
#pragma once

#include "interp_run.cuh"
#include "spread_run3.cuh"

namespace dnufft {

template <int W> struct Interp3Shape {
  static constexpr int LB = run3_bin_log2(W), BIN = 1 << LB;
  static constexpr int SPAN = BIN - 1 + W;
  static constexpr int RT = (SPAN + 3) / 4, KT = (SPAN + 3) / 4;
  static constexpr int PLANES = (SPAN + 3) / 4 * 4, ROWS = 4 * RT, COLS = 4 * KT;
  static constexpr int THREADS = 32 * SPAN;
  static constexpr int BATCH = 64;
  static constexpr int ST0 = PLANES + ROWS + COLS;
  static constexpr int ST = ST0 % 8 == 4 ? ST0 : ST0 + 4;   // 4 or 12 modulo 16
  static constexpr size_t SMEM = size_t(BATCH) * ST * 8 + size_t(SPAN) * BATCH * 16 +
                                 size_t(BATCH) * sizeof(int4);
};

template <typename Tc, int W>
__global__ void __launch_bounds__(Interp3Shape<W>::THREADS)
    k_interp_run3(const __grid_constant__ PointsDesc pts, uint32_t ppb,
                  const __grid_constant__ Geometry g, const __grid_constant__ KernelPoly<double> kp,
                  const double2 *__restrict__ grid, int64_t gtrans, double2 *__restrict__ out,
                  int64_t os, int64_t otrans) {
  using R = Interp3Shape<W>;
  constexpr int B = R::BATCH;
  extern __shared__ __align__(16) unsigned char smraw_run[];
  double *st = reinterpret_cast<double *>(smraw_run);
  double2 *part = reinterpret_cast<double2 *>(st + B * R::ST);   // [plane][point]
  // every staged point: bins of the three axes, output index
  int4 *info = reinterpret_cast<int4 *>(part + R::SPAN * B);
  grid += int64_t(blockIdx.y) * gtrans;
  out += int64_t(blockIdx.y) * otrans;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]), n2 = int(g.nover[2]);
  const uint32_t first = blockIdx.x * ppb;
  const uint32_t last = uint32_t(min(uint64_t(pts.npts), uint64_t(first) + ppb));
  double G[R::RT][R::KT];
  int cu = -1, cv = -1, cw = -1;
  bool finite = true;
  auto load_window = [&]() {
    const int u = wrap3(cu * R::BIN - g.nsafe + warp, n0), v0 = cv * R::BIN - g.nsafe,
              w0 = cw * R::BIN - g.nsafe;
    const double *pl = reinterpret_cast<const double *>(grid + int64_t(u) * n1 * n2) +
                       ((lane >> 2) & 1);
    bool ok = true;
#pragma unroll
    for (int r = 0; r < R::RT; ++r) {
      const double *row = pl + 2 * int64_t(wrap3(v0 + 4 * r + (lane >> 3), n1)) * n2;
#pragma unroll
      for (int k = 0; k < R::KT; ++k) {
        G[r][k] = __ldg(row + 2 * wrap3(w0 + 4 * k + (lane & 3), n2));
        ok = ok && isfinite(G[r][k]);
      }
    }
    finite = __all_sync(0xffffffffu, ok);
  };
  for (uint32_t base = first; base < last; base += B) {
    const int np = int(min(uint32_t(B), last - base));
    {
      // (every thread is past the reads of the last batch: the barrier before
      // its sums)
      float4 *z4 = reinterpret_cast<float4 *>(st);
      const int nz = np * (R::ST / 2);
      for (int i = tid; i < nz; i += R::THREADS) z4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    for (int it = tid; it < 3 * np; it += R::THREADS) {
      const int ax = it / np, q = it - ax * np;
      const uint32_t i = base + uint32_t(q), j = pts.perm[i];
      const Tc *c = static_cast<const Tc *>(pts.coord);
      const Tc x = pts.sorted ? c[uint64_t(i) * 3 + ax]
                              : c[int64_t(j) * pts.cs0 + int64_t(ax) * pts.cs1];
      int i0;
      double frac, w[W];
      fold<Tc>(x, ax == 0 ? g.coordfct[0] : (ax == 1 ? g.coordfct[1] : g.coordfct[2]),
               ax == 0 ? n0 : (ax == 1 ? n1 : n2),
               ax == 0 ? g.shift[0] : (ax == 1 ? g.shift[1] : g.shift[2]),
               ax == 0 ? g.maxi0[0] : (ax == 1 ? g.maxi0[1] : g.maxi0[2]), i0, frac);
      kernel_weights<double, W>(kp, double(W - 1) - 2.0 * frac, w);
      const int t = i0 + g.nsafe;
      int *inf = reinterpret_cast<int *>(info + q);
      inf[ax] = t >> R::LB;
      if (ax == 0) inf[3] = int(j);
      double *sp = st + q * R::ST + (ax == 0 ? 0 : (ax == 1 ? R::PLANES : R::PLANES + R::ROWS)) +
                   (t & (R::BIN - 1));
#pragma unroll
      for (int a = 0; a < W; ++a) sp[a] = w[a];
    }
    __syncthreads();
    for (int s0 = 0; s0 < np; s0 += 32) {
      const int p0 = s0 + lane, ns = min(32, np - s0);
      const int4 b = info[min(p0, np - 1)];
      int pu = __shfl_up_sync(0xffffffffu, b.x, 1), pv = __shfl_up_sync(0xffffffffu, b.y, 1),
          pw = __shfl_up_sync(0xffffffffu, b.z, 1);
      if (lane == 0) {
        pu = cu;
        pv = cv;
        pw = cw;
      }
      const unsigned bins =
          __ballot_sync(0xffffffffu, p0 < np && (b.x != pu || b.y != pv || b.z != pw));
      unsigned rest = bins & ~1u;
      for (int s = 0; s < ns;) {
        if ((bins >> s) & 1u) {
          cu = __shfl_sync(0xffffffffu, b.x, s);
          cv = __shfl_sync(0xffffffffu, b.y, s);
          cw = __shfl_sync(0xffffffffu, b.z, s);
          load_window();
        }
        const int e = rest ? __ffs(rest) - 1 : ns;
        rest &= rest - 1;
        for (int p = s; p < e; p += 8) {
          const int pt = s0 + p + (lane >> 2);
          const bool on = p + (lane >> 2) < e;
          const double *f = st + (on ? pt : s0 + p) * R::ST;
          const double ku = on ? f[warp] : 0.;
          double sx = 0., sy = 0.;
          if (__any_sync(0xffffffffu, ku != 0.)) {
            if (finite) {
              double a[R::KT];
#pragma unroll
              for (int k = 0; k < R::KT; ++k) a[k] = f[R::PLANES + R::ROWS + 4 * k + (lane & 3)];
#pragma unroll
              for (int r = 0; r < R::RT; ++r) {
                double c0 = 0., c1 = 0.;
#pragma unroll
                for (int k = 0; k < R::KT; ++k)
                  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, "
                      "{%0, %1};"
                      : "+d"(c0), "+d"(c1)
                      : "d"(a[k]), "d"(G[r][k]));
                const double kv = f[R::PLANES + 4 * r + (lane & 3)];
                sx += kv * c0;
                sy += kv * c1;
              }
            } else if (ku != 0.) {
              // a value of the plane is not finite: the footprint's cells only
              const double2 *pl =
                  grid + int64_t(wrap3(cu * R::BIN - g.nsafe + warp, n0)) * n1 * n2;
              for (int r = lane & 3; r < R::SPAN; r += 4) {
                const double kv = f[R::PLANES + r];
                if (kv == 0.) continue;
                const double2 *row = pl + int64_t(wrap3(cv * R::BIN - g.nsafe + r, n1)) * n2;
                for (int c = 0; c < R::SPAN; ++c) {
                  const double wt = kv * f[R::PLANES + R::ROWS + c];
                  if (wt == 0.) continue;
                  const double2 gv = __ldg(row + wrap3(cw * R::BIN - g.nsafe + c, n2));
                  sx += wt * gv.x;
                  sy += wt * gv.y;
                }
              }
            }
            sx += __shfl_xor_sync(0xffffffffu, sx, 1);
            sy += __shfl_xor_sync(0xffffffffu, sy, 1);
            sx += __shfl_xor_sync(0xffffffffu, sx, 2);
            sy += __shfl_xor_sync(0xffffffffu, sy, 2);
          }
          // (a plane the point does not touch: exactly zero)
          if (on && (lane & 3) == 0)
            part[warp * B + pt] = ku != 0. ? make_double2(ku * sx, ku * sy) : make_double2(0., 0.);
        }
        s = e;
      }
    }
    __syncthreads();
    for (int q = tid; q < np; q += R::THREADS) {
      double sx = 0., sy = 0.;
      for (int pl = 0; pl < R::SPAN; ++pl) {
        const double2 v = part[pl * B + q];
        sx += v.x;
        sy += v.y;
      }
      out[int64_t(uint32_t(info[q].w)) * os] = make_double2(sx, sy);
    }
    // the next batch's zeroing touches st only; info and part are written after
    // its first barrier
  }
}

template <typename Tc, int W>
void interp_run3_w(const PointsDesc &pts, const Geometry &g, const KernelPoly<double> &kp,
                   const void *grid, int64_t gtrans, void *out, int64_t os, int64_t otrans,
                   int ntrans, cudaStream_t st) {
  using R = Interp3Shape<W>;
  auto kern = k_interp_run3<Tc, W>;
  allow_smem(kern, R::SMEM);
  // points per CTA: as the spreader
  const uint64_t per = uint64_t(pts.npts) * uint64_t(ntrans) / (148 * 8);
  const uint32_t ppb =
      per >= R::BATCH ? R::BATCH * uint32_t(std::min<uint64_t>(16, per / R::BATCH))
                      : std::max<uint32_t>(16, uint32_t(per) & ~15u);
  dim3 grd(unsigned((uint64_t(pts.npts) + ppb - 1) / ppb), ntrans);
  kern<<<grd, R::THREADS, R::SMEM, st>>>(pts, ppb, g, kp, static_cast<const double2 *>(grid),
                                         gtrans, static_cast<double2 *>(out), os, otrans);
  DN_LAUNCHED();
}

// The direct form (interp3_direct says when): one thread per point reads its W^3
// cells; the points are sorted by cell, so that a warp's reads hit few lines.  From
// W = 9 the compiler is told that one CTA per SM will do: left alone it keeps to 146
// to 188 registers and fewer loads in flight (2e6 points, 112^3 cells, W = 9: 1750
// us against 1262 with 255); below it is the faster form.
constexpr int ID3_THREADS = 128;

template <typename Tc, int W>
__global__ void __launch_bounds__(ID3_THREADS, W <= 8 ? 0 : 1)
    k_interp_direct3(const __grid_constant__ PointsDesc pts, const __grid_constant__ Geometry g,
                     const __grid_constant__ KernelPoly<double> kp,
                     const double2 *__restrict__ grid, int64_t gtrans, double2 *__restrict__ out,
                     int64_t os, int64_t otrans) {
  const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= pts.npts) return;
  grid += int64_t(blockIdx.y) * gtrans;
  out += int64_t(blockIdx.y) * otrans;
  Tc x[3];
  const uint32_t j = load_point<Tc, 3>(pts, uint32_t(i), x);
  double w[3][W];
  int c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double frac;
    fold<Tc>(x[d], g.coordfct[d], int(g.nover[d]), g.shift[d], g.maxi0[d], c[d], frac);
    kernel_weights<double, W>(kp, double(W - 1) - 2.0 * frac, w[d]);
  }
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]), n2 = int(g.nover[2]);
  int iw[W];
#pragma unroll
  for (int e = 0; e < W; ++e) iw[e] = wrap2(c[2] + e, n2);
  double ar = 0, ai = 0;
#pragma unroll 1
  for (int a = 0; a < W; ++a) {
    const double2 *plane = grid + int64_t(wrap2(c[0] + a, n0)) * n1 * n2;
    double pr = 0, pi = 0;
#pragma unroll
    for (int b = 0; b < W; ++b) {
      const double2 *row = plane + int64_t(wrap2(c[1] + b, n1)) * n2;
      double rr = 0, ri = 0;
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const double2 v = __ldg(row + iw[e]);
        rr += w[2][e] * v.x;
        ri += w[2][e] * v.y;
      }
      pr += w[1][b] * rr;
      pi += w[1][b] * ri;
    }
    ar += w[0][a] * pr;
    ai += w[0][a] * pi;
  }
  out[int64_t(j) * os] = make_double2(ar, ai);
}

template <typename Tc, int W>
void interp_direct3_w(const PointsDesc &pts, const Geometry &g, const KernelPoly<double> &kp,
                      const void *grid, int64_t gtrans, void *out, int64_t os, int64_t otrans,
                      int ntrans, cudaStream_t st) {
  // few points: one warp per CTA, so that they spread over the SMs
  const uint64_t all = uint64_t(pts.npts) * uint64_t(ntrans);
  const unsigned nt = all < 148u * 2u * ID3_THREADS ? 32u : unsigned(ID3_THREADS);
  const dim3 grd(unsigned((uint64_t(pts.npts) + nt - 1) / nt), ntrans);
  k_interp_direct3<Tc, W><<<grd, nt, 0, st>>>(pts, g, kp, static_cast<const double2 *>(grid),
                                              gtrans, static_cast<double2 *>(out), os, otrans);
  DN_LAUNCHED();
}

// ---------------------------------------------------------------- single precision
// The same with FP32 multiply-adds (packed in pairs), in the operand layout of
// Run3Window<float>: 4 warps, warp r has planes r, r + 4, r + 8, r + 12 of the
// window, a lane 4 rows x 2 cells of each.  A point uses two neighbouring planes
// of a warp (loops for the three pairs, as the spreader); the lanes' parts of
// four points are added over the warp together.
//
// One thread per point reading W^3 cells from a staged tile took 134 SM cycles at
// W = 8 (32 of shared-memory bandwidth; 16 warps per SM); this takes 46 issue
// cycles for the sums and their 12 shuffles per four points, 108 cycles in all (1e7
// points, 256^3 cells, 3.8 ms; issue active 59 %).
template <int W> struct Interp3fShape {
  static constexpr int PLANES = 16, ROWS = 16, CELLS = 16;
  static constexpr int THREADS = 128, BATCH = 128;
  static constexpr int ST = PLANES + ROWS + CELLS + 4;   // an odd number of 16-byte words
  static constexpr size_t SMEM = size_t(BATCH) * (ST * 4 + 4 * sizeof(float2) + sizeof(int4));
};

template <int W> struct Interp3fWindow {
  using R = Interp3fShape<W>;
  using L = RunWindow<float, W>;
  unsigned long long c[4][2][4];   // [plane][cell][row], (re, im)
  // sums of points p .. p + 3 (at most e) over planes J0, J0 + 1 to part
  template <int J0>
  __device__ __forceinline__ void points(const float *st, float2 *part, int s, int e, int warp,
                                         int lane) const {
    const float *pk = st + 4 * warp + J0, *kr = st + R::PLANES + L::row0(lane),
                *kc = st + R::PLANES + R::ROWS + L::cell0(lane);
#pragma unroll 1
    for (int p = s; p < e; p += 4) {
      float2 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int o = min(p + q, e - 1) * R::ST;
        const float4 k = *reinterpret_cast<const float4 *>(kr + o);
        const unsigned long long kk[4] = {pack2(k.x, k.x), pack2(k.y, k.y), pack2(k.z, k.z),
                                          pack2(k.w, k.w)};
        const float w0 = kc[o], w1 = kc[o + 8];
        const unsigned long long ww[2] = {pack2(w0, w0), pack2(w1, w1)};
        unsigned long long sum = 0ull;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          unsigned long long t = 0ull;
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            unsigned long long a;
            asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(a) : "l"(c[J0 + j][d][0]), "l"(kk[0]));
#pragma unroll
            for (int i = 1; i < 4; ++i)
              asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(c[J0 + j][d][i]), "l"(kk[i]));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t) : "l"(a), "l"(ww[d]));
          }
          const float kj = pk[o + j];
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum) : "l"(t), "l"(pack2(kj, kj)));
        }
        v[q] = unpack2(sum);
      }
      // lane bits 4 and 3 choose a point of the four, the others are added up
      const bool b4 = lane & 16, b3 = lane & 8;
      float2 x, y;
      x.x = (b4 ? v[2].x : v[0].x) + __shfl_xor_sync(0xffffffffu, b4 ? v[0].x : v[2].x, 16);
      x.y = (b4 ? v[2].y : v[0].y) + __shfl_xor_sync(0xffffffffu, b4 ? v[0].y : v[2].y, 16);
      y.x = (b4 ? v[3].x : v[1].x) + __shfl_xor_sync(0xffffffffu, b4 ? v[1].x : v[3].x, 16);
      y.y = (b4 ? v[3].y : v[1].y) + __shfl_xor_sync(0xffffffffu, b4 ? v[1].y : v[3].y, 16);
      float2 z;
      z.x = (b3 ? y.x : x.x) + __shfl_xor_sync(0xffffffffu, b3 ? x.x : y.x, 8);
      z.y = (b3 ? y.y : x.y) + __shfl_xor_sync(0xffffffffu, b3 ? x.y : y.y, 8);
#pragma unroll
      for (int o = 4; o; o >>= 1) {
        z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
        z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
      }
      const int q = p + 2 * (b4 ? 1 : 0) + (b3 ? 1 : 0);
      if ((lane & 7) == 0 && q < e) part[warp * R::BATCH + q] = z;
    }
  }
};

template <typename Tc, int W>
__global__ void __launch_bounds__(Interp3fShape<W>::THREADS, 4)
    k_interp_run3f(const __grid_constant__ PointsDesc pts, uint32_t ppb,
                   const __grid_constant__ Geometry g, const __grid_constant__ KernelPoly<float> kp,
                   const float2 *__restrict__ grid, int64_t gtrans, float2 *__restrict__ out,
                   int64_t os, int64_t otrans) {
  using R = Interp3fShape<W>;
  using L = RunWindow<float, W>;
  constexpr int B = R::BATCH;
  extern __shared__ __align__(16) unsigned char smraw_run[];
  float *st = reinterpret_cast<float *>(smraw_run);
  int4 *info = reinterpret_cast<int4 *>(st + B * R::ST);   // first-axis cell, bins, output index
  float2 *part = reinterpret_cast<float2 *>(info + B);     // [warp][point]
  grid += int64_t(blockIdx.y) * gtrans;
  out += int64_t(blockIdx.y) * otrans;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n0 = int(g.nover[0]), n1 = int(g.nover[1]), n2 = int(g.nover[2]);
  const uint32_t first = blockIdx.x * ppb;
  const uint32_t last = uint32_t(min(uint64_t(pts.npts), uint64_t(first) + ppb));
  Interp3fWindow<W> win;
  int cu = -1, cv = -1, cw = -1;
  bool finite = true;
  auto load_window = [&]() {
    const int u0 = cu * 8 - g.nsafe, rv = cv * 8 - g.nsafe + L::row0(lane),
              wa = cw * 8 - g.nsafe + L::cell0(lane);
    const int ca = wrap3(wa, n2), cb = wrap3(wa + 8, n2);
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 *pl = grid + int64_t(wrap3(u0 + warp + 4 * j, n0)) * n1 * n2;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 *row = pl + int64_t(wrap3(rv + i, n1)) * n2;
        const float2 a = __ldg(row + ca), b = __ldg(row + cb);
        win.c[j][0][i] = pack2(a.x, a.y);
        win.c[j][1][i] = pack2(b.x, b.y);
        ok = ok && isfinite(a.x) && isfinite(a.y) && isfinite(b.x) && isfinite(b.y);
      }
    }
    finite = __all_sync(0xffffffffu, ok);
  };
  for (uint32_t base = first; base < last; base += B) {
    const int np = int(min(uint32_t(B), last - base));
    {
      float4 *z4 = reinterpret_cast<float4 *>(st);
      const int nz = np * (R::ST / 4);
      for (int i = tid; i < nz; i += R::THREADS) z4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    for (int it = tid; it < 3 * B; it += R::THREADS) {
      const int ax = it / B, q = it - ax * B;
      if (q >= np) continue;
      const uint32_t i = base + uint32_t(q), j = pts.perm[i];
      const Tc *c = static_cast<const Tc *>(pts.coord);
      const Tc x = pts.sorted ? c[uint64_t(i) * 3 + ax]
                              : c[int64_t(j) * pts.cs0 + int64_t(ax) * pts.cs1];
      int i0;
      double frac;
      float w[W];
      fold<Tc>(x, ax == 0 ? g.coordfct[0] : (ax == 1 ? g.coordfct[1] : g.coordfct[2]),
               ax == 0 ? n0 : (ax == 1 ? n1 : n2),
               ax == 0 ? g.shift[0] : (ax == 1 ? g.shift[1] : g.shift[2]),
               ax == 0 ? g.maxi0[0] : (ax == 1 ? g.maxi0[1] : g.maxi0[2]), i0, frac);
      kernel_weights<float, W>(kp, float(double(W - 1) - 2.0 * frac), w);
      const int t = i0 + g.nsafe, o = t & 7;
      int *inf = reinterpret_cast<int *>(info + q);
      inf[ax] = ax == 0 ? t : t >> 3;
      float *sp = st + q * R::ST;
      if (ax == 0) {
        inf[3] = int(j);
#pragma unroll
        for (int a = 0; a < W; ++a) sp[Run3Window<float, W>::plane_slot(o + a)] = w[a];
      } else {
        sp += (ax == 1 ? R::PLANES : R::PLANES + R::ROWS) + o;
#pragma unroll
        for (int a = 0; a < W; ++a) sp[a] = w[a];
      }
    }
    __syncthreads();
    for (int s0 = 0; s0 < np; s0 += 32) {
      const int p0 = s0 + lane, ns = min(32, np - s0);
      const int4 b = info[min(p0, np - 1)];
      const int j0 = Run3Window<float, W>::first_plane(b.x & 7, warp);
      int pu = __shfl_up_sync(0xffffffffu, b.x >> 3, 1), pv = __shfl_up_sync(0xffffffffu, b.y, 1),
          pw = __shfl_up_sync(0xffffffffu, b.z, 1);
      const int pj = __shfl_up_sync(0xffffffffu, j0, 1);
      if (lane == 0) {
        pu = cu;
        pv = cv;
        pw = cw;
      }
      const unsigned bins = __ballot_sync(
          0xffffffffu, p0 < np && ((b.x >> 3) != pu || b.y != pv || b.z != pw));
      unsigned rest = bins | __ballot_sync(0xffffffffu, p0 < np && lane > 0 && j0 != pj);
      rest &= ~1u;
      for (int s = 0; s < ns;) {
        if ((bins >> s) & 1u) {
          cu = __shfl_sync(0xffffffffu, b.x, s) >> 3;
          cv = __shfl_sync(0xffffffffu, b.y, s);
          cw = __shfl_sync(0xffffffffu, b.z, s);
          load_window();
        }
        const int e = rest ? __ffs(rest) - 1 : ns;
        rest &= rest - 1;
        const int js = __shfl_sync(0xffffffffu, j0, s);
        if (!finite) {
          // the footprints' cells only
          for (int p = s0 + s; p < s0 + e; ++p) {
            const float *f = st + p * R::ST;
            float sx = 0.f, sy = 0.f;
            for (int k = lane; k < 4 * 256; k += 32) {
              const int j = k >> 8, r = (k >> 4) & 15, c = k & 15;
              const float wt = f[4 * warp + j] * f[R::PLANES + r] * f[R::PLANES + R::ROWS + c];
              if (wt == 0.f) continue;
              const float2 gv = __ldg(
                  grid + (int64_t(wrap3(cu * 8 - g.nsafe + warp + 4 * j, n0)) * n1 +
                          wrap3(cv * 8 - g.nsafe + r, n1)) * n2 + wrap3(cw * 8 - g.nsafe + c, n2));
              sx += wt * gv.x;
              sy += wt * gv.y;
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
              sx += __shfl_xor_sync(0xffffffffu, sx, o);
              sy += __shfl_xor_sync(0xffffffffu, sy, o);
            }
            if (lane == 0) part[warp * B + p] = make_float2(sx, sy);
          }
        } else if (js == 0) {
          win.template points<0>(st, part, s0 + s, s0 + e, warp, lane);
        } else if (js == 1) {
          win.template points<1>(st, part, s0 + s, s0 + e, warp, lane);
        } else {
          win.template points<2>(st, part, s0 + s, s0 + e, warp, lane);
        }
        s = e;
      }
    }
    __syncthreads();
    for (int q = tid; q < np; q += R::THREADS) {
      float2 v = part[q];
#pragma unroll
      for (int k = 1; k < 4; ++k) {
        const float2 a = part[k * B + q];
        v.x += a.x;
        v.y += a.y;
      }
      out[int64_t(uint32_t(info[q].w)) * os] = v;
    }
  }
}

template <typename Tc, int W>
void interp_run3f_w(const PointsDesc &pts, const Geometry &g, const KernelPoly<float> &kp,
                    const void *grid, int64_t gtrans, void *out, int64_t os, int64_t otrans,
                    int ntrans, cudaStream_t st) {
  using R = Interp3fShape<W>;
  auto kern = k_interp_run3f<Tc, W>;
  allow_smem(kern, R::SMEM);
  const uint64_t per = uint64_t(pts.npts) * uint64_t(ntrans) / (148 * 8);
  const uint32_t ppb =
      per >= R::BATCH ? R::BATCH * uint32_t(std::min<uint64_t>(8, per / R::BATCH))
                      : std::max<uint32_t>(16, uint32_t(per) & ~15u);
  dim3 grd(unsigned((uint64_t(pts.npts) + ppb - 1) / ppb), ntrans);
  kern<<<grd, R::THREADS, R::SMEM, st>>>(pts, ppb, g, kp, static_cast<const float2 *>(grid),
                                         gtrans, static_cast<float2 *>(out), os, otrans);
  DN_LAUNCHED();
}

}  // namespace dnufft

// lines64.cuh -- the FP64 pass kernels for power-of-two lengths 32 .. 1024.
//
// What bounds an FP64 pass on GB300 is FP64 issue: 1.7 operations per SM and
// cycle, shared by the SM, and at most one warp instruction per 64 cycles from
// one warp (both measured).  So the operation count decides, and a line has to
// be spread over enough warps to keep the unit fed.  The warp-level transforms
// of the FP32 passes (16 values per lane, one or two lines per warp) have the
// right count but leave a 256^2 film with 129 CTAs of two warps: 880 FP64
// instructions in a row at 64 cycles each, 44 us.  Here a thread holds R = 2 or
// 4 values: a Stockham transform through shared memory with N / R threads per
// line, the same operations spread over 4 to 8 times the warps.  The first
// stage takes its values straight from global memory and the last one leaves
// them in registers, so a pass touches shared memory between stages only.
//
// Operations per value and radix-2 level: 3 (a radix-4 butterfly with three
// twiddles: 24).  Both R make the same radix-4 butterflies, R = 2 with two
// threads each (l64_line_split), so a field has the same bits in any launch shape:
// the shape follows the number of lines, and a film alone, in a batch, and in a
// part of a batch on a stream of its own have to agree.  (Radix-2 butterflies at R =
// 2 rounded differently, with an error 5 to 9 % larger, and took twice the
// barriers: 64 x 256 32.0 us per sweep instead of 29.8, 64^2 20.0 and 19.9, 32^2 18.0
// and 18.7.)  x passes transform the z components of two rows as one complex line
// (three lines for two rows where the FP32 passes transform four).
#pragma once
#include "fft.cuh"
#include "mmc_internal.h"

namespace mmc {

__device__ __forceinline__ void pdl_wait();

// Element i of a line in shared memory: one 16-byte slot skipped every 8
// spreads the stages' strided stores over the banks.
__host__ __device__ constexpr int l64_pos(int i) { return i + (i >> 3); }
template <int N>
__host__ __device__ constexpr int l64_stride() {
  return N + N / 8;
}
template <int N>
constexpr size_t l64_smem(int lines) {
  return ((size_t)N + 2 * (size_t)lines * l64_stride<N>()) * sizeof(double2);
}

template <bool INV>
__device__ __forceinline__ double2 l64_rot(double2 a) {  // times -i (forward), +i (inverse)
  return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}
__device__ __forceinline__ double2 l64_twice_minus(double2 a, double2 b) {  // 2 a - b
  return make_double2(fma_rn(2.0, a.x, -b.x), fma_rn(2.0, a.y, -b.y));
}

// Radix-2 butterfly without a twiddle.
__device__ __forceinline__ void l64_radix2(double2& u, double2& w) {
  const double2 a = u;
  u = cadd(a, w);
  w = csub(a, w);
}

// Radix-4 butterfly on v with twiddles w[1 .. 3] (TW) or without.
template <bool INV, bool TW>
__device__ __forceinline__ void l64_radix4(double2 (&v)[4], const double2* w) {
  double2 a0, a1, a2, a3;
  if constexpr (TW) {
    a0 = INV ? cmacc(v[0], v[2], w[2]) : cmac(v[0], v[2], w[2]);
    a1 = l64_twice_minus(v[0], a0);
    const double2 p = INV ? cmulc(v[1], w[1]) : cmul(v[1], w[1]);
    a2 = INV ? cmacc(p, v[3], w[3]) : cmac(p, v[3], w[3]);
    a3 = l64_twice_minus(p, a2);
  } else {
    a0 = cadd(v[0], v[2]);
    a1 = csub(v[0], v[2]);
    a2 = cadd(v[1], v[3]);
    a3 = csub(v[1], v[3]);
  }
  const double2 r3 = l64_rot<INV>(a3);
  v[0] = cadd(a0, a2);
  v[1] = cadd(a1, r3);
  v[2] = csub(a0, a2);
  v[3] = csub(a1, r3);
}

template <int N>
__host__ __device__ constexpr int ilog2() {
  return N <= 1 ? 0 : 1 + ilog2<N / 2>();
}

// One transform of a line by its N / 4 threads, thread j holding the values j +
// t N / 4 on entry and on return (natural order both times).  a and b: the
// line's two buffers in shared memory, exchanged as the stages go.  Ends
// without a barrier: on return other threads may still read b, and a is free
// for the caller.  All threads of the CTA must call it.  A power of two that is
// no power of 4 starts with a radix-2 stage (two butterflies per thread).
template <int N, bool INV>
__device__ __forceinline__ void l64_line(double2 (&v)[4], double2*& a, double2*& b, int j, const double2* roots) {
  constexpr int Q = N / 4;
  constexpr bool odd = ilog2<N>() & 1;
  if constexpr (odd) {
    l64_radix2(v[0], v[2]);
    l64_radix2(v[1], v[3]);
    a[l64_pos(2 * j)] = v[0];
    a[l64_pos(2 * j + 1)] = v[2];
    a[l64_pos(2 * (j + Q))] = v[1];
    a[l64_pos(2 * (j + Q) + 1)] = v[3];
  } else {
    l64_radix4<INV, false>(v, nullptr);
#pragma unroll
    for (int q = 0; q < 4; ++q) a[l64_pos(4 * j + q)] = v[q];
  }
  __syncthreads();
#pragma unroll
  for (int ns = odd ? 2 : 4; ns < N; ns *= 4) {
    const int k = j & (ns - 1);
    const int st = N / (4 * ns);
    double2 w[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = a[l64_pos(j + t * Q)];
#pragma unroll
    for (int t = 1; t < 4; ++t) w[t] = roots[t * k * st];
    l64_radix4<INV, true>(v, w);
    if (4 * ns < N) {
#pragma unroll
      for (int q = 0; q < 4; ++q) b[l64_pos((j - k) * 4 + k + q * ns)] = v[q];
      __syncthreads();
    }
    double2* s = a;  // b was written and is read next; a is free (after the last stage: was read)
    a = b;
    b = s;
  }
}

// The same line by N / 2 threads: the lanes 2 jj + c of a warp share the radix-4
// butterflies of a thread jj of l64_line, lane c making the component c (0 real, 1
// imaginary) of everything, by the same operations in the same order.  u: that
// component of the values jj + t N / 4.  (A warp issues one FP64 instruction per
// 64 cycles: 12 in a row per stage instead of 24.)  Up to N = 64 a line lies
// within one warp and its stages meet without the CTA's other lines.
// Signs are turned on the high word: as FP64 negations of a lane's choice they cost
// 12 % of a 64^2 film's sweep.
__device__ __forceinline__ double l64_flip(double v, unsigned m) {
  return __hiloint2double(__double2hiint(v) ^ (int)m, __double2loint(v));
}
template <bool INV>
__device__ __forceinline__ double2 l64_pick(double2 w, int c) {
  // the factors of l64_mac: those of cmac and cmul, or of cmacc and cmulc
  if (INV) return make_double2(w.x, l64_flip(w.y, (unsigned)c << 31));
  return make_double2(c ? w.y : w.x, l64_flip(c ? w.x : w.y, (unsigned)(1 - c) << 31));
}
template <bool INV>
__device__ __forceinline__ double l64_mac(double acc, double2 a, double2 f, int c) {
  const double p = INV && c ? a.y : a.x, q = INV && c ? a.x : a.y;
  return fma_rn(q, f.y, fma_rn(p, f.x, acc));
}
template <bool INV>
__device__ __forceinline__ double l64_mul(double2 a, double2 f, int c) {
  const double p = INV && c ? a.y : a.x, q = INV && c ? a.x : a.y;
  return fma_rn(p, f.x, q * f.y);
}
__device__ __forceinline__ void l64_put(double2* line, int i, int c, double v) {
  reinterpret_cast<double*>(line + l64_pos(i))[c] = v;
}
template <int N, bool INV>
__device__ __forceinline__ void l64_line_split(double (&u)[4], double2*& a, double2*& b, int jj, int c,
                                               const double2* roots) {
  constexpr int Q = N / 4;
  constexpr bool odd = ilog2<N>() & 1;
  // a CTA of this shape has one unit: 3 lines, whole warps but for N = 32
  const unsigned mask = N >= 64 || threadIdx.x < 32 ? 0xffffffffu : 0xffffu;
  auto meet = [&] {  // the threads of a line: within a warp up to N = 64
    if constexpr (N <= 64) __syncwarp(mask);
    else __syncthreads();
  };
  // (a0, a1, a2, a3) -> the butterfly's outputs; a3's other component comes from the other lane
  auto finish = [&](double a0, double a1, double a2, double a3) {
    double r = __shfl_xor_sync(mask, a3, 1);
    r = l64_flip(r, (unsigned)(INV ? 1 - c : c) << 31);
    u[0] = a0 + a2;
    u[1] = a1 + r;
    u[2] = a0 - a2;
    u[3] = a1 - r;
  };
  if constexpr (odd) {
    l64_put(a, 2 * jj, c, u[0] + u[2]);
    l64_put(a, 2 * jj + 1, c, u[0] - u[2]);
    l64_put(a, 2 * (jj + Q), c, u[1] + u[3]);
    l64_put(a, 2 * (jj + Q) + 1, c, u[1] - u[3]);
  } else {
    finish(u[0] + u[2], u[0] - u[2], u[1] + u[3], u[1] - u[3]);
#pragma unroll
    for (int q = 0; q < 4; ++q) l64_put(a, 4 * jj + q, c, u[q]);
  }
  meet();
#pragma unroll
  for (int ns = odd ? 2 : 4; ns < N; ns *= 4) {
    const int k = jj & (ns - 1), st = N / (4 * ns);
    const double v0 = reinterpret_cast<const double*>(a + l64_pos(jj))[c];
    const double2 v1 = a[l64_pos(jj + Q)], v2 = a[l64_pos(jj + 2 * Q)], v3 = a[l64_pos(jj + 3 * Q)];
    const double a0 = l64_mac<INV>(v0, v2, l64_pick<INV>(roots[2 * k * st], c), c);
    const double p = l64_mul<INV>(v1, l64_pick<INV>(roots[k * st], c), c);
    const double a2 = l64_mac<INV>(p, v3, l64_pick<INV>(roots[3 * k * st], c), c);
    finish(a0, fma_rn(2.0, v0, -a0), a2, fma_rn(2.0, p, -a2));
    if (4 * ns < N) {
#pragma unroll
      for (int q = 0; q < 4; ++q) l64_put(b, (jj - k) * 4 + k + q * ns, c, u[q]);
      meet();
    }
    double2* s = a;
    a = b;
    b = s;
  }
}

template <int N>
__device__ __forceinline__ void l64_roots(const FftPlan& p, double2* dst) {
  const double2* src = p.tw64 + p.full_off;
  for (int i = threadIdx.x; i < N; i += blockDim.x) dst[i] = src[i];
}

// x passes: a CTA takes TP pairs of rows (2 P, 2 P + 1).  Line 0 of a pair is
// mx + i my of the first row, line 1 the same of the second, line 2 mz of the
// first + i mz of the second (0 where a last odd row has no second).
// Spectra come out doubled (the 1/2 of the split is part of the column pass's
// factor).
template <int N, int R, int TP>
__global__ void __launch_bounds__(3 * TP * N / R)
    k_x_forward64(const __grid_constant__ FftPlan p, int xdata, FastDiv dyd, int nrows, const double* __restrict__ in,
                  long long in_cstride, double2* __restrict__ S, long long nspec, int nyp, int pitch,
                  long long in_rstride, long long s_rstride) {
  constexpr int Q = N / R, LS = l64_stride<N>(), HX = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* roots = reinterpret_cast<double2*>(smem_raw);
  double2* buf = roots + N;
  in += blockIdx.z * in_rstride;
  S += blockIdx.z * s_rstride;
  const int line = threadIdx.x / Q, j = threadIdx.x - line * Q;
  const int pair = line / 3, w = line - 3 * pair;
  const int row0 = 2 * (blockIdx.x * TP + pair);
  l64_roots<N>(p, roots);
  pdl_wait();
  double2* a = buf + line * LS;
  double2* b = a + 3 * TP * LS;
  if constexpr (R == 2) {
    const int jj = j >> 1, c = j & 1, row = w == 2 ? row0 + c : row0 + w;
    const double* src = in + (w == 2 ? 2 : c) * in_cstride + (long long)row * xdata;
    double u[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int x = jj + t * (N / 4);
      u[t] = x < xdata && row < nrows ? src[x] : 0.0;
    }
    __syncthreads();  // roots
    l64_line_split<N, false>(u, a, b, jj, c, roots);
#pragma unroll
    for (int q = 0; q < 4; ++q) l64_put(a, jj + q * (N / 4), c, u[q]);
  } else {
    double2 v[4];
    const int ra = w == 1 ? row0 + 1 : row0, rb = w == 0 ? row0 : row0 + 1;
    const double* re = in + (w == 2 ? 2 * in_cstride : 0) + (long long)ra * xdata;
    const double* im = in + (w == 2 ? 2 * in_cstride : in_cstride) + (long long)rb * xdata;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int x = j + t * Q;
      v[t] = make_double2(x < xdata && ra < nrows ? re[x] : 0.0, x < xdata && rb < nrows ? im[x] : 0.0);
    }
    __syncthreads();  // roots
    l64_line<N, false>(v, a, b, j, roots);
#pragma unroll
    for (int q = 0; q < 4; ++q) a[l64_pos(j + q * Q)] = v[q];
  }
  const double2* res = a - line * LS;  // every line ends in the same buffer
  __syncthreads();
  for (int idx = threadIdx.x; idx < 3 * TP * HX; idx += 3 * TP * Q) {
    const int l = idx / HX, k = idx - l * HX;
    const int pr = l / 3, ww = l - 3 * pr;
    const int r0 = 2 * (blockIdx.x * TP + pr), ra = ww == 1 ? r0 + 1 : r0, rb = ww == 0 ? r0 : r0 + 1;
    const double2 A = res[l * LS + l64_pos(k)];
    const double2 B = res[l * LS + l64_pos(k == 0 ? 0 : N - k)];
    const int za = dyd.div(ra), zb = dyd.div(rb), ny = (int)dyd.d;
    double2* sa = S + (ww == 2 ? 2 * nspec : 0) + ((long long)za * nyp + (ra - za * ny)) * pitch + k;
    double2* sb = S + (ww == 2 ? 2 * nspec : nspec) + ((long long)zb * nyp + (rb - zb * ny)) * pitch + k;
    if (ra < nrows) *sa = make_double2(A.x + B.x, A.y - B.y);
    if (rb < nrows) *sb = make_double2(A.y + B.y, B.x - A.x);
  }
}

template <int N, int R, int TP>
__global__ void __launch_bounds__(3 * TP * N / R)
    k_x_inverse64(const __grid_constant__ FftPlan p, const double2* __restrict__ S, long long nspec, int nyp, int pitch,
                  int xout, FastDiv dyo, int nrows, double* __restrict__ out, long long out_cstride,
                  long long s_rstride, long long out_rstride) {
  constexpr int Q = N / R, LS = l64_stride<N>(), HX = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* roots = reinterpret_cast<double2*>(smem_raw);
  double2* buf = roots + N;
  S += blockIdx.z * s_rstride;
  out += blockIdx.z * out_rstride;
  const int line = threadIdx.x / Q, j = threadIdx.x - line * Q;
  const int pair = line / 3, w = line - 3 * pair;
  const int row0 = 2 * (blockIdx.x * TP + pair);
  const int ra = w == 1 ? row0 + 1 : row0, rb = w == 0 ? row0 : row0 + 1;
  l64_roots<N>(p, roots);
  pdl_wait();
  double2* a = buf + line * LS;
  double2* b = a + 3 * TP * LS;
  const int za = dyo.div(ra), zb = dyo.div(rb), ny = (int)dyo.d;
  const double2* sa = S + (w == 2 ? 2 * nspec : 0) + ((long long)za * nyp + (ra - za * ny)) * pitch;
  const double2* sb = S + (w == 2 ? 2 * nspec : nspec) + ((long long)zb * nyp + (rb - zb * ny)) * pitch;
  double* oa = out + (w == 2 ? 2 * out_cstride : 0) + (long long)ra * xout;
  double* ob = out + (w == 2 ? 2 * out_cstride : out_cstride) + (long long)rb * xout;
  if constexpr (R == 2) {
    // component c of u0 + i u1: u0.x - u1.y, or u0.y + u1.x
    const int jj = j >> 1, c = j & 1;
    double u[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int k = jj + t * (N / 4), kk = k < HX ? k : N - k;
      const double f0 = ra < nrows ? reinterpret_cast<const double*>(sa + kk)[c] : 0.0;
      const double f1 = rb < nrows ? reinterpret_cast<const double*>(sb + kk)[1 - c] : 0.0;
      const double re = c ? f1 : f0;
      double im = c ? f0 : f1;
      im = l64_flip(im, ((k >= HX) != (c == 0)) ? 0x80000000u : 0u);
      if (k == 0 || 2 * k == N) im = 0;  // bins that are real for a real output
      u[t] = re + im;
    }
    __syncthreads();  // roots
    l64_line_split<N, true>(u, a, b, jj, c, roots);
    double* o = c ? ob : oa;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = jj + q * (N / 4);
      if (x < xout && (c ? rb : ra) < nrows) o[x] = u[q];
    }
  } else {
    double2 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int k = j + t * Q, kk = k < HX ? k : N - k;
      double2 u0 = ra < nrows ? sa[kk] : make_double2(0, 0), u1 = rb < nrows ? sb[kk] : make_double2(0, 0);
      if (k >= HX) u0.y = -u0.y, u1.y = -u1.y;
      if (k == 0 || 2 * k == N) u0.y = u1.y = 0;  // bins that are real for a real output
      v[t] = make_double2(u0.x - u1.y, u0.y + u1.x);
    }
    __syncthreads();  // roots
    l64_line<N, true>(v, a, b, j, roots);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int x = j + q * Q;
      if (x < xout && ra < nrows) oa[x] = v[q].x;
      if (x < xout && rb < nrows) ob[x] = v[q].y;
    }
  }
}

// Column pass along y or z over TX kx columns (see k_col_pass for the layout
// and the limits): MODE 0 forward only, 1 inverse only, 2 forward, the tensor
// product, inverse.  Thread (c, j, t) holds component c of column t; the product
// reads the other two components from shared memory and leaves component c in
// the registers the inverse starts from.
template <int N, int R, int TX, int MODE>
__global__ void __launch_bounds__(3 * TX * N / R)
    k_col64(const __grid_constant__ FftPlan p, double2* __restrict__ S, long long nspec,
            const double2* __restrict__ khat, int hx, long long plane_stride, long long pos_stride, int load_lim,
            int store_lim, int sym, double factor, long long s_rstride) {
  constexpr int Q = N / R, LS = l64_stride<N>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* roots = reinterpret_cast<double2*>(smem_raw);
  double2* buf = roots + N;
  S += blockIdx.z * s_rstride;
  const int t = threadIdx.x % TX, rest = threadIdx.x / TX, c = rest / Q, j = rest - c * Q;
  const int kx = blockIdx.x * TX + t;
  const bool ok = kx < hx;
  const long long base = (long long)blockIdx.y * plane_stride + (ok ? kx : 0);
  l64_roots<N>(p, roots);
  pdl_wait();
  double2* Sc = S + c * nspec + base;
  const int line = c * TX + t;
  double2* a = buf + line * LS;
  double2* b = a + 3 * TX * LS;
  // row c of K^: (xx, xy, xz), (xy, yy, yz) or (xz, yz, zz) in the six blocks xx, xy, xz, yy, yz, zz
  const int o0 = c, o1 = c == 0 ? 1 : c == 1 ? 3 : 4, o2 = c == 0 ? 2 : c == 1 ? 4 : 5;
  const double2* kk = khat + base;
  if constexpr (R == 2) {
    static_assert(TX == 1, "the two lanes of a butterfly are neighbours");
    const int jj = j >> 1, e = j & 1;
    double u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int pos = jj + q * (N / 4);
      u[q] = ok && pos < load_lim ? reinterpret_cast<const double*>(Sc + pos * pos_stride)[e] : 0.0;
    }
    __syncthreads();  // roots
    if constexpr (MODE != 1) l64_line_split<N, false>(u, a, b, jj, e, roots);
    if constexpr (MODE == 2) {
#pragma unroll
      for (int q = 0; q < 4; ++q) l64_put(a, jj + q * (N / 4), e, u[q]);
      const double2* mx = a - line * LS;
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int pos = jj + q * (N / 4), i = l64_pos(pos);
        const long long kp = pos * pos_stride;
        double2 k0 = kk[o0 * nspec + kp], k1 = kk[o1 * nspec + kp], k2 = kk[o2 * nspec + kp];
        if (sym) k0.y = k1.y = k2.y = 0.0;
        // tensor_row's component e
        double h = l64_mul<false>(mx[i], l64_pick<false>(k0, e), e);
        h = l64_mac<false>(h, mx[LS + i], l64_pick<false>(k1, e), e);
        h = l64_mac<false>(h, mx[2 * LS + i], l64_pick<false>(k2, e), e);
        u[q] = h * factor;
      }
      // the inverse's second stage writes the lines that the product reads; its
      // own barriers are those of one warp here
      if constexpr (N <= 64) __syncthreads();
      double2* s = a;  // as below
      a = b;
      b = s;
    }
    if constexpr (MODE != 0) l64_line_split<N, true>(u, a, b, jj, e, roots);
    if (!ok) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int pos = jj + q * (N / 4);
      if (pos < store_lim) reinterpret_cast<double*>(Sc + pos * pos_stride)[e] = u[q];
    }
  } else {
    double2 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int pos = j + q * Q;
      v[q] = (ok && pos < load_lim) ? Sc[pos * pos_stride] : make_double2(0, 0);
    }
    __syncthreads();  // roots
    if constexpr (MODE != 1) l64_line<N, false>(v, a, b, j, roots);
    if constexpr (MODE == 2) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[l64_pos(j + q * Q)] = v[q];
      const double2* mx = a - line * LS + t * LS;
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int pos = j + q * Q, e = l64_pos(pos);
        const long long kp = pos * pos_stride;
        double2 k0 = kk[o0 * nspec + kp], k1 = kk[o1 * nspec + kp], k2 = kk[o2 * nspec + kp];
        if (sym) k0.y = k1.y = k2.y = 0.0;
        const double2 h = tensor_row(mx[e], mx[TX * LS + e], mx[2 * TX * LS + e], k0, k1, k2);
        v[q] = make_double2(h.x * factor, h.y * factor);
      }
      // the inverse's first stage writes b, which the forward transform's last
      // stage has read before the barrier above
      double2* s = a;
      a = b;
      b = s;
    }
    if constexpr (MODE != 0) l64_line<N, true>(v, a, b, j, roots);
    if (!ok) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int pos = j + q * Q;
      if (pos < store_lim) Sc[pos * pos_stride] = v[q];
    }
  }
}

// Launch shapes (R, columns or row pairs per CTA).  `units` columns x planes x
// replicas (row pairs x replicas): with less than four warps per SM at R = 4
// the pass is a chain of FP64 instructions at 64 cycles each, and R = 2 halves
// it; with more, R = 4 has half the barriers.  Wider tiles (whole 32-byte
// sectors, shared roots) once the CTAs cover the SMs twice.
struct L64Fns {
  void (*xf)(FftPlan, int, FastDiv, int, const double*, long long, double2*, long long, int, int, long long, long long);
  void (*xi)(FftPlan, const double2*, long long, int, int, int, FastDiv, int, double*, long long, long long, long long);
  void (*col[3])(FftPlan, double2*, long long, const double2*, int, long long, long long, int, int, int, double,
                 long long);
  int tile, threads;
  size_t smem;
};
template <int N, int R, int TX>
L64Fns l64_fns() {
  return {k_x_forward64<N, R, TX>, k_x_inverse64<N, R, TX>,
          {k_col64<N, R, TX, 0>, k_col64<N, R, TX, 1>, k_col64<N, R, TX, 2>},
          TX, 3 * TX * N / R, l64_smem<N>(3 * TX)};
}
inline bool l64_lookup(int n, int shape, L64Fns& f) {  // shape 0: few lines, 1: one unit per CTA, 2: wide tiles
#define MMC_L64(N_, R0_, TX0_, TX1_, TX2_)                                     \
  case N_:                                                                     \
    f = shape == 0   ? l64_fns<N_, R0_, TX0_>()                                \
        : shape == 1 ? l64_fns<N_, 4, TX1_>()                                  \
                     : l64_fns<N_, 4, TX2_>();                                 \
    return true;
  switch (n) {
    MMC_L64(32, 2, 1, 2, 8)
    MMC_L64(64, 2, 1, 1, 4)
    MMC_L64(128, 2, 1, 1, 2)
    MMC_L64(256, 2, 1, 1, 2)
    MMC_L64(512, 4, 1, 1, 1)
    MMC_L64(1024, 4, 1, 1, 1)
    default:
      return false;
  }
#undef MMC_L64
}
inline bool l64_pick(const FftPlan& p, long long units, L64Fns& f) {
  if (!p.warp_a) return false;
  const long long sms = 152;
  if (units * 3 * p.n / 4 < 4 * 32 * sms) return l64_lookup(p.n, 0, f);
  if (!l64_lookup(p.n, 2, f)) return false;
  return units >= 2 * sms * f.tile || l64_lookup(p.n, 1, f);
}
inline cudaError_t l64_prepare(int max_dyn_smem) {
  for (int n = 32; n <= 1024; n *= 2)
    for (int s = 0; s < 3; ++s) {
      L64Fns f;
      l64_lookup(n, s, f);
      const void* fns[] = {(const void*)f.xf, (const void*)f.xi, (const void*)f.col[0], (const void*)f.col[1],
                           (const void*)f.col[2]};
      for (const void* q : fns) {
        const cudaError_t e = cudaFuncSetAttribute(q, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem);
        if (e != cudaSuccess) return e;
      }
    }
  return cudaSuccess;
}

}  // namespace mmc

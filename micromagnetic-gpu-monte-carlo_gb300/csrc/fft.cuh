// fft.cuh -- batched mixed-radix Stockham FFT on lines held in shared memory.
//
// The reference ran cuFFT (src/main.cu:593-675, 868-877).  Here every
// transform is a hand-written autosort (Stockham) FFT over a batch of lines in
// shared memory, so that a pass kernel can load a tile, transform it, apply
// the tensor product and transform back without leaving the SM.  Stage s of a
// length-n transform with radix R and span Ns reads element j + t*(n/R) of the
// source, multiplies by exp(-+2 pi i t k/(Ns R)), k = j mod Ns, does an R-point
// DFT and writes element (j-k)*R + k + q*Ns of the destination.
#pragma once
#include "mmc_internal.h"

namespace mmc {

template <typename T>
struct Cplx;
template <>
struct Cplx<float> {
  using type = float2;
};
template <>
struct Cplx<double> {
  using type = double2;
};
// FP64 whose products are never contracted into multiply-adds: the transforms
// of the relaxation (see launch_demag_sym) use it in place of double.
struct f64s {
  double v;
  f64s() = default;
  __host__ __device__ __forceinline__ f64s(double d) : v(d) {}
};
#if defined(__CUDACC__)
__device__ __forceinline__ f64s operator+(f64s a, f64s b) { return __dadd_rn(a.v, b.v); }
__device__ __forceinline__ f64s operator-(f64s a, f64s b) { return __dadd_rn(a.v, -b.v); }
__device__ __forceinline__ f64s operator*(f64s a, f64s b) { return __dmul_rn(a.v, b.v); }
__device__ __forceinline__ f64s operator-(f64s a) { return -a.v; }
#endif
struct alignas(16) f64s2 {
  f64s x, y;
};
template <>
struct Cplx<f64s> {
  using type = f64s2;
};
template <typename T>
using C = typename Cplx<T>::type;
// double proper: products written with explicit multiply-adds
template <typename V>
constexpr bool fused_mul = sizeof(V) == sizeof(double2) && !__is_same(V, f64s2);

template <typename V>
__device__ __forceinline__ V cmk(decltype(V::x) a, decltype(V::x) b) {
  V r;
  r.x = a;
  r.y = b;
  return r;
}
template <typename V>
__device__ __forceinline__ V cadd(V a, V b) {
  return cmk<V>(a.x + b.x, a.y + b.y);
}
template <typename V>
__device__ __forceinline__ V csub(V a, V b) {
  return cmk<V>(a.x - b.x, a.y - b.y);
}
// The same as padd and psub where neither operand is a product the compiler
// contracts with the sum: in FP32 one packed instruction for the real and the
// imaginary part, the same two sums in one issue slot.
template <typename V>
__device__ __forceinline__ V padd(V a, V b) {
  return cadd(a, b);
}
template <typename V>
__device__ __forceinline__ V psub(V a, V b) {
  return csub(a, b);
}
__device__ __forceinline__ unsigned long long f2_bits(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 f2_of(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
__device__ __forceinline__ float2 padd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
}
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
}
// FP64 products are written with explicit multiply-adds.  The FP64 kernels are
// built without contraction (the sweep's decisions round like the oracle's),
// but the transforms only have to be accurate, and GB300 issues 1.7 FP64
// operations per SM and cycle (measured; FP32: 118), so an FP64 pass takes as
// long as its operation count: 4 instead of 6 per complex product, 6 instead
// of 10 per butterfly with a twiddle (Goedecker, SIAM J. Sci. Comput. 18,
// 1997), each rounding once less.
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
template <typename V>
__device__ __forceinline__ V cmul(V a, V b) {
  if constexpr (fused_mul<V>) return cmk<V>(fma_rn(a.x, b.x, -(a.y * b.y)), fma_rn(a.x, b.y, a.y * b.x));
  return cmk<V>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
template <typename V>
__device__ __forceinline__ V cmulc(V a, V b) {
  if constexpr (fused_mul<V>) return cmk<V>(fma_rn(a.x, b.x, a.y * b.y), fma_rn(a.y, b.x, -(a.x * b.y)));
  return cmk<V>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// acc + a * b, acc + a * conj(b)
template <typename V>
__device__ __forceinline__ V cmac(V acc, V a, V b) {
  if constexpr (fused_mul<V>)
    return cmk<V>(fma_rn(-a.y, b.y, fma_rn(a.x, b.x, acc.x)), fma_rn(a.y, b.x, fma_rn(a.x, b.y, acc.y)));
  return cadd(acc, cmul(a, b));
}
template <typename V>
__device__ __forceinline__ V cmacc(V acc, V a, V b) {
  if constexpr (fused_mul<V>)
    return cmk<V>(fma_rn(a.y, b.y, fma_rn(a.x, b.x, acc.x)), fma_rn(-a.x, b.y, fma_rn(a.y, b.x, acc.y)));
  return cadd(acc, cmulc(a, b));
}

// The products of the power-of-two transforms and of the tensor with the
// contraction written out in FP32, the one the compiler chose for cmul and
// cmulc in the first passes: which product of a sum it fuses depends on the code
// around, and every pass has to round alike.
template <typename V>
__device__ __forceinline__ V tmul(V a, V b) {
  return cmul(a, b);
}
template <typename V>
__device__ __forceinline__ V tmulc(V a, V b) {
  return cmulc(a, b);
}
__device__ __forceinline__ float2 tmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 tmulc(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, -__fmul_rn(a.x, b.y)));
}

// K^ . M^ at one frequency (src/demag_cu.cu:98-111): the real and imaginary
// parts of sum_b K_ab M_b for a = x, y, z, from the six tensor blocks.
template <typename V>
__device__ __forceinline__ V tensor_row(V mx, V my, V mz, V k0, V k1, V k2) {
  if constexpr (fused_mul<V>) return cmac(cmac(cmul(mx, k0), my, k1), mz, k2);
  const V p0 = tmul(mx, k0), p1 = tmul(my, k1), p2 = tmul(mz, k2);
  return padd(padd(p0, p1), p2);
}

template <typename T>
__device__ __forceinline__ const C<T>* plan_tw(const FftPlan& p);
template <>
__device__ __forceinline__ const float2* plan_tw<float>(const FftPlan& p) {
  return p.tw32;
}
template <>
__device__ __forceinline__ const double2* plan_tw<double>(const FftPlan& p) {
  return p.tw64;
}
template <>
__device__ __forceinline__ const f64s2* plan_tw<f64s>(const FftPlan& p) {
  return reinterpret_cast<const f64s2*>(p.tw64);
}

// Copies the plan's twiddle table into shared memory (call before the FFT,
// followed by __syncthreads()).
template <typename T>
__device__ __forceinline__ void load_twiddles(const FftPlan& p, C<T>* dst) {
  const C<T>* src = plan_tw<T>(p);
  for (int i = threadIdx.x; i < p.tw_total; i += blockDim.x) dst[i] = src[i];
}

// One stage of an odd radix R >= 7: the direct R-point DFT with R known at
// compile time, so that the R values stay in registers and the matrix of roots
// [q][t] is read from global memory, the same word for a whole warp.  (One loop
// over a run-time R held them in local memory: the demag convolution of an open
// 512^2 film, lines of 1023 = 3 11 31, took 423 us in FP32 and 5601 us in FP64;
// now 199 and 1506 us.)  Bound by the R^2 multiply-adds per butterfly.  FP32
// products are contracted as they were in that loop, written out.
__device__ __forceinline__ float2 odd_mul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}
template <bool INV, typename V>
__device__ __forceinline__ V odd_twiddle(V a, V b) {
  if constexpr (sizeof(V) == sizeof(float2)) return INV ? tmulc(a, b) : odd_mul(a, b);
  return INV ? cmulc(a, b) : cmul(a, b);
}
template <bool INV, typename V>
__device__ __forceinline__ V odd_mac(V acc, V a, V b) {
  if constexpr (sizeof(V) == sizeof(float2)) return padd(acc, INV ? tmulc(a, b) : odd_mul(a, b));
  return INV ? cmacc(acc, a, b) : cmac(acc, a, b);
}
template <typename T, bool INV, int R>
__device__ __noinline__ void odd_stage(const C<T>* src, C<T>* dst, int total, int stride, int nb, int Ns, FastDiv dnb,
                                       FastDiv dns, const C<T>* W, const C<T>* __restrict__ mat) {
  using V = C<T>;
  // long radices leave few butterflies (99 for three lines of 1023 in radix 31):
  // `parts` threads share one, each taking a range of its outputs
  const int parts = min(8, max(1, (2 * (int)blockDim.x + total - 1) / total)), per = (R + parts - 1) / parts;
  for (int idx0 = threadIdx.x; idx0 < total * parts; idx0 += blockDim.x) {
    const int part = idx0 / total, idx = idx0 - part * total;
    const int line = dnb.div(idx), j = idx - line * nb, k = j - dns.div(j) * Ns;
    const V* in = src + (long long)line * stride + j;
    V* out = dst + (long long)line * stride + (j - k) * R + k;
    V v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = in[t * nb];
    if (k) {
#pragma unroll
      for (int t = 1; t < R; ++t) v[t] = odd_twiddle<INV>(v[t], W[(t - 1) * Ns + k]);
    }
    if constexpr (fused_mul<V>) {
      // FP64: the values t and R - t in their sum a and difference b, which give
      // the outputs q and R - q together, X = (v0 + sum a cos) -+ i sum b sin:
      // (R - 1)^2 operations instead of 4 R (R - 1)
      constexpr int H = (R - 1) / 2;
      V s0 = v[0];
#pragma unroll
      for (int t = 1; t <= H; ++t) {
        const V a = cadd(v[t], v[R - t]), b = csub(v[t], v[R - t]);
        v[t] = a;
        v[R - t] = b;
        s0 = cadd(s0, a);
      }
      const int perh = (H + parts - 1) / parts, p1 = min(H, (part + 1) * perh);
      if (part == 0) out[0] = s0;
#pragma unroll 1
      for (int q = 1 + part * perh; q <= p1; ++q) {
        const V* row = mat + q * R;
        V P = v[0], S = cmk<V>(0, 0);
#pragma unroll
        for (int t = 1; t <= H; ++t) {
          const V w = row[t];
          P = cmk<V>(fma_rn(v[t].x, w.x, P.x), fma_rn(v[t].y, w.x, P.y));
          S = cmk<V>(fma_rn(v[R - t].x, w.y, S.x), fma_rn(v[R - t].y, w.y, S.y));
        }
        const V u = cmk<V>(P.x - S.y, P.y + S.x), d = cmk<V>(P.x + S.y, P.y - S.x);  // P + i S, P - i S
        out[q * Ns] = INV ? d : u;
        out[(R - q) * Ns] = INV ? u : d;
      }
      continue;
    }
    const int q1 = min(R, (part + 1) * per);
#pragma unroll 1
    for (int q = part * per; q < q1; ++q) {
      const V* row = mat + q * R;
      V acc = v[0];
#pragma unroll
      for (int t = 1; t < R; ++t) acc = odd_mac<INV>(acc, v[t], row[t]);
      out[q * Ns] = acc;
    }
  }
}
template <typename T, bool INV>
__device__ __forceinline__ void odd_stages(const C<T>* src, C<T>* dst, int total, int stride, int R, int nb, int Ns,
                                           FastDiv dnb, FastDiv dns, const C<T>* W, const C<T>* mat) {
  switch (R) {
#define MMC_ODD(R_) \
  case R_: odd_stage<T, INV, R_>(src, dst, total, stride, nb, Ns, dnb, dns, W, mat); break;
    MMC_ODD(7) MMC_ODD(11) MMC_ODD(13) MMC_ODD(17) MMC_ODD(19) MMC_ODD(23) MMC_ODD(29) MMC_ODD(31)
#undef MMC_ODD
  }
}

// Whether a plan has a stage for odd_stage.
inline bool plan_odd(const FftPlan& p) {
  for (int s = 0; s < p.nstages; ++s)
    if (p.radix[s] >= 7) return true;
  return false;
}

// Transforms `nlines` lines of length p.n; line l starts at buf + l*stride.
// `a` holds the input, `b` is scratch of the same shape.  Returns the buffer
// holding the result (a or b).  All threads of the block must call it.
// ODD: the length may have radices of 7 and above (plan_odd).  Their stages keep
// up to 31 values in registers and a kernel's register allocation covers
// everything it calls, so only kernels instantiated with ODD contain them and
// only plans that need them reach those: with them in every kernel, k_rows<float>
// took 203 registers instead of 128 and k_col_pass<float> 127 instead of 70; us
// per sweep with / without them: 8 x 96^2 films 32.2 / 25.1 in FP32, 93.0 / 76.8 in
// FP64, 16 x 128^2 by the row kernel in bands of 2 57.3 / 37.5.
template <typename T, bool INV, bool ODD>
__device__ __noinline__ C<T>* fft_lines(C<T>* a, C<T>* b, int nlines, int stride, const FftPlan& p,
                                        const C<T>* tw) {
  using V = C<T>;
  V* src = a;
  V* dst = b;
  const int n = p.n;
  for (int s = 0; s < p.nstages; ++s) {
    const int R = p.radix[s], Ns = p.ns[s], nb = n / R;
    const FastDiv dnb = p.dnb[s], dns = p.dns[s];
    const V* W = tw + p.tw_off[s];
    const int total = nlines * nb;
    if constexpr (ODD) {
      if (R >= 7) odd_stages<T, INV>(src, dst, total, stride, R, nb, Ns, dnb, dns, W, plan_tw<T>(p) + p.odd_off[s]);
    }
    for (int idx = threadIdx.x; (!ODD || R < 7) && idx < total; idx += blockDim.x) {
      const int line = dnb.div(idx);
      const int j = idx - line * nb;
      const int k = j - dns.div(j) * Ns;
      const V* in = src + (long long)line * stride + j;
      V* out = dst + (long long)line * stride + (j - k) * R + k;
      if (R == 4) {
        V v0 = in[0], v1 = in[nb], v2 = in[2 * nb], v3 = in[3 * nb];
        if (k) {
          V w1 = W[k], w2 = W[Ns + k], w3 = W[2 * Ns + k];
          if (INV) {
            v1 = cmulc(v1, w1);
            v2 = cmulc(v2, w2);
            v3 = cmulc(v3, w3);
          } else {
            v1 = cmul(v1, w1);
            v2 = cmul(v2, w2);
            v3 = cmul(v3, w3);
          }
        }
        V a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = csub(v1, v3);
        V r3 = INV ? cmk<V>(-a3.y, a3.x) : cmk<V>(a3.y, -a3.x);
        out[0] = cadd(a0, a2);
        out[Ns] = cadd(a1, r3);
        out[2 * Ns] = csub(a0, a2);
        out[3 * Ns] = csub(a1, r3);
      } else if (R == 2) {
        V v0 = in[0], v1 = in[nb];
        if (k) v1 = INV ? cmulc(v1, W[k]) : cmul(v1, W[k]);
        out[0] = cadd(v0, v1);
        out[Ns] = csub(v0, v1);
      } else if (R == 3) {
        V v0 = in[0], v1 = in[nb], v2 = in[2 * nb];
        if (k) {
          V w1 = W[k], w2 = W[Ns + k];
          if (INV) {
            v1 = cmulc(v1, w1);
            v2 = cmulc(v2, w2);
          } else {
            v1 = cmul(v1, w1);
            v2 = cmul(v2, w2);
          }
        }
        const T s3 = (T)0.86602540378443864676;  // sin(2 pi / 3)
        V t1 = cadd(v1, v2);
        V t2 = cmk<V>(v0.x - (T)0.5 * t1.x, v0.y - (T)0.5 * t1.y);
        V t3 = csub(v1, v2);
        V r = INV ? cmk<V>(-s3 * t3.y, s3 * t3.x) : cmk<V>(s3 * t3.y, -s3 * t3.x);
        out[0] = cadd(v0, t1);
        out[Ns] = cadd(t2, r);
        out[2 * Ns] = csub(t2, r);
      } else if (R == 5) {
        V v0 = in[0], v1 = in[nb], v2 = in[2 * nb], v3 = in[3 * nb], v4 = in[4 * nb];
        if (k) {
          const V w1 = W[k], w2 = W[Ns + k], w3 = W[2 * Ns + k], w4 = W[3 * Ns + k];
          if (INV) {
            v1 = cmulc(v1, w1);
            v2 = cmulc(v2, w2);
            v3 = cmulc(v3, w3);
            v4 = cmulc(v4, w4);
          } else {
            v1 = cmul(v1, w1);
            v2 = cmul(v2, w2);
            v3 = cmul(v3, w3);
            v4 = cmul(v4, w4);
          }
        }
        // 5-point DFT from the symmetric and antisymmetric pairs:
        // cos(2 pi / 5), cos(4 pi / 5), sin(2 pi / 5), sin(4 pi / 5)
        const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
        const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
        const V t1 = cadd(v1, v4), t2 = cadd(v2, v3), t3 = csub(v1, v4), t4 = csub(v2, v3);
        const V a1 = cmk<V>(v0.x + c1 * t1.x + c2 * t2.x, v0.y + c1 * t1.y + c2 * t2.y);
        const V a2 = cmk<V>(v0.x + c2 * t1.x + c1 * t2.x, v0.y + c2 * t1.y + c1 * t2.y);
        const V b1 = cmk<V>(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y);
        const V b2 = cmk<V>(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y);
        // forward: X1 = a1 - i b1, X4 = a1 + i b1, X2 = a2 - i b2, X3 = a2 + i b2
        const V mb1 = INV ? cmk<V>(-b1.y, b1.x) : cmk<V>(b1.y, -b1.x);  // -+ i b1
        const V mb2 = INV ? cmk<V>(-b2.y, b2.x) : cmk<V>(b2.y, -b2.x);
        out[0] = cadd(v0, cadd(t1, t2));
        out[Ns] = cadd(a1, mb1);
        out[2 * Ns] = cadd(a2, mb2);
        out[3 * Ns] = csub(a2, mb2);
        out[4 * Ns] = csub(a1, mb1);
      }
    }
    __syncthreads();
    V* t = src;
    src = dst;
    dst = t;
  }
  return src;
}

// ------------------------------------------------------------ warp-level FFT
// 32nd roots of unity exp(-2 pi i k / 32), k = 0..15 (cos, -sin): cos(pi k / 16)
// and -sin(pi k / 16) to 20 digits.
__device__ __forceinline__ double w32_re(int k) {
  const double c[16] = {1.0,
                        0.98078528040323044913,
                        0.92387953251128675613,
                        0.83146961230254523708,
                        0.70710678118654752440,
                        0.55557023301960222474,
                        0.38268343236508977173,
                        0.19509032201612826785,
                        0.0,
                        -0.19509032201612826785,
                        -0.38268343236508977173,
                        -0.55557023301960222474,
                        -0.70710678118654752440,
                        -0.83146961230254523708,
                        -0.92387953251128675613,
                        -0.98078528040323044913};
  return c[k];
}
__device__ __forceinline__ double w32_im(int k) {
  const double s[16] = {0.0,
                        -0.19509032201612826785,
                        -0.38268343236508977173,
                        -0.55557023301960222474,
                        -0.70710678118654752440,
                        -0.83146961230254523708,
                        -0.92387953251128675613,
                        -0.98078528040323044913,
                        -1.0,
                        -0.98078528040323044913,
                        -0.92387953251128675613,
                        -0.83146961230254523708,
                        -0.70710678118654752440,
                        -0.55557023301960222474,
                        -0.38268343236508977173,
                        -0.19509032201612826785};
  return s[k];
}

// In-register DFT of N in {1, 2, 4, 8, 16, 32} values, natural order in and out,
// by radix-2 decimation in time.  INV uses the conjugate roots.
template <typename T, bool INV, int N>
struct RegDft {
  __device__ __forceinline__ static void run(C<T>* v) {
    using V = C<T>;
    V e[N / 2], o[N / 2];
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      e[i] = v[2 * i];
      o[i] = v[2 * i + 1];
    }
    RegDft<T, INV, N / 2>::run(e);
    RegDft<T, INV, N / 2>::run(o);
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
      V t;
      if (k == 0) {
        t = o[k];
      } else if (4 * k == N) {  // multiply by -i (forward) or +i (inverse)
        t = INV ? cmk<V>(-o[k].y, o[k].x) : cmk<V>(o[k].y, -o[k].x);
      } else {
        const T wr = (T)w32_re(k * (32 / N));
        const T wi = INV ? (T)-w32_im(k * (32 / N)) : (T)w32_im(k * (32 / N));
        if constexpr (fused_mul<V>) {  // e + w o, and e - w o as 2 e - (e + w o)
          v[k] = cmac(e[k], o[k], cmk<V>(wr, wi));
          v[k + N / 2] = cmk<V>(fma_rn((T)2, e[k].x, -v[k].x), fma_rn((T)2, e[k].y, -v[k].y));
          continue;
        }
        t = cmk<V>(o[k].x * wr - o[k].y * wi, o[k].x * wi + o[k].y * wr);
      }
      v[k] = padd(e[k], t);
      v[k + N / 2] = psub(e[k], t);
    }
  }
};
template <typename T, bool INV>
struct RegDft<T, INV, 1> {
  __device__ __forceinline__ static void run(C<T>*) {}
};

// One line of length N = A * B owned by B lanes of one warp (lane b of the
// group), with the input already in registers: v[a] = x[b + B a].
//   x[b + B a] --(A-point DFT over a)--> Y[b][ka] --(* W_N^(b ka))-->
//   transpose in the line --(B-point DFT over b)--> X[ka + A kb].
// On return lane b holds the columns ka = b Q + t, t < Q = A / B: v[t B + kb] =
// X[ka + A kb].  Lp is the line's room in shared memory for the transpose.  All
// lanes of the warp must call it (inactive groups with active = false).
// roots: exp(-2 pi i j / N), j < N, or (LANES) the same roots as [ka][b].
// The transpose goes through rows of B + 1 elements when PAD (row ka at
// ka (B + 1): every address is the lane's base plus a compile-time offset,
// and the line then needs N + A - 1 elements of room), else through rows of
// B with the columns rotated by ka (N elements of room).
template <typename T, bool INV, int A, int B, bool PAD = false, bool LANES = false>
__device__ __forceinline__ void fft_line_cols(C<T> (&v)[A], C<T>* Lp, int b, bool active, const C<T>* roots) {
  using V = C<T>;
  constexpr int Q = A / B;
  RegDft<T, INV, A>::run(v);
#pragma unroll
  for (int ka = 1; ka < A; ++ka) {
    const V w = LANES ? roots[ka * B + b] : roots[b * ka];
    v[ka] = INV ? tmulc(v[ka], w) : tmul(v[ka], w);
  }
  __syncwarp();
  if (active) {
    if constexpr (PAD) {
      C<T>* row = Lp + b;
#pragma unroll
      for (int ka = 0; ka < A; ++ka) row[ka * (B + 1)] = v[ka];
    } else {
#pragma unroll
      for (int ka = 0; ka < A; ++ka) Lp[ka * B + ((b + ka) & (B - 1))] = v[ka];
    }
  }
  __syncwarp();
  // v is dead after the transpose: reuse it for the columns
  if (active) {
    if constexpr (PAD) {
      const C<T>* col = Lp + b * Q * (B + 1);
#pragma unroll
      for (int t = 0; t < Q; ++t)
#pragma unroll
        for (int bb = 0; bb < B; ++bb) v[t * B + bb] = col[t * (B + 1) + bb];
    } else {
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const int ka = b * Q + t;
#pragma unroll
        for (int bb = 0; bb < B; ++bb) v[t * B + bb] = Lp[ka * B + ((bb + ka) & (B - 1))];
      }
    }
  }
#pragma unroll
  for (int t = 0; t < Q; ++t) RegDft<T, INV, B>::run(v + t * B);
}

// The same with X left in Lp in natural order.
template <typename T, bool INV, int A, int B, bool PAD = false>
__device__ __forceinline__ void fft_line_regs(C<T> (&v)[A], C<T>* Lp, int b, bool active, const C<T>* roots) {
  constexpr int Q = A / B;
  fft_line_cols<T, INV, A, B, PAD>(v, Lp, b, active, roots);
  __syncwarp();
  if (active) {
#pragma unroll
    for (int t = 0; t < Q; ++t)
#pragma unroll
      for (int kb = 0; kb < B; ++kb) Lp[(b * Q + t) + A * kb] = v[t * B + kb];
  }
  __syncwarp();
}

// Transforms `nlines` lines of length N = A * B in place (line l at
// buf + l * stride, stride >= N + A - 1 when PAD), 32 / B lines per warp at
// a time; only __syncwarp is needed inside.
template <typename T, bool INV, int A, int B, bool PAD = false>
__device__ __forceinline__ void fft_lines_warp_body(C<T>* buf, int nlines, int stride, const C<T>* roots) {
  using V = C<T>;
  constexpr int GPW = 32 / B;  // lines per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int grp = lane / B, b = lane - grp * B;
  for (int line0 = warp * GPW; line0 < nlines; line0 += nwarps * GPW) {
    const int line = line0 + grp;
    const bool active = line < nlines;
    V* Lp = buf + (long long)(active ? line : 0) * stride;
    V v[A];
    if (active) {
#pragma unroll
      for (int a = 0; a < A; ++a) v[a] = Lp[b + B * a];
    }
    fft_line_regs<T, INV, A, B, PAD>(v, Lp, b, active, roots);
  }
}

// Out-of-line copy (kernels that hold much state around the transform call it
// so that the transform's registers are not added to theirs).
template <typename T, bool INV, int A, int B, bool PAD = false>
__device__ __noinline__ void fft_lines_warp(C<T>* buf, int nlines, int stride, const C<T>* roots) {
  fft_lines_warp_body<T, INV, A, B, PAD>(buf, nlines, stride, roots);
}

// ------------------------------------------------------ per-thread DFT
// A whole short line (N <= 16) in one thread's registers, by mixed-radix
// decimation in time with every index known at compile time: N = F M with F
// the smallest prime factor, X[k1 + M k2] = DFT_F over f of
// W_N^(f k1) Y_f[k1], Y_f = DFT_M(x[F m + f]).  Radix 2, 3, 4 and 5
// butterflies are written out; other primes are direct DFTs.  Roots:
// rt[j * RS] = exp(-2 pi i j / N) (a table of N * RS roots in shared memory).
template <int N>
struct SmallFactor {
  static constexpr int value = N % 4 == 0 ? 4 : N % 2 == 0 ? 2 : N % 3 == 0 ? 3 : N % 5 == 0 ? 5 : N % 7 == 0 ? 7 : N;
};

template <typename T, bool INV, int N, int RS>
struct ThreadDft {
  __device__ __forceinline__ static void run(C<T>* v, const C<T>* rt) {
    using V = C<T>;
    constexpr int F = SmallFactor<N>::value, M = N / F;
    if constexpr (M == 1) {
      butterfly(v, rt);
    } else {
      V sub[F][M];
#pragma unroll
      for (int f = 0; f < F; ++f)
#pragma unroll
        for (int m = 0; m < M; ++m) sub[f][m] = v[F * m + f];
#pragma unroll
      for (int f = 0; f < F; ++f) ThreadDft<T, INV, M, RS * F>::run(sub[f], rt);
#pragma unroll
      for (int k1 = 0; k1 < M; ++k1) {
        V z[F];
#pragma unroll
        for (int f = 0; f < F; ++f) {
          const int e = (f * k1) % N;
          if (e == 0) {
            z[f] = sub[f][k1];
          } else {
            const V w = rt[e * RS];
            z[f] = INV ? cmulc(sub[f][k1], w) : cmul(sub[f][k1], w);
          }
        }
        ThreadDft<T, INV, F, RS * M>::run(z, rt);
#pragma unroll
        for (int k2 = 0; k2 < F; ++k2) v[k1 + M * k2] = z[k2];
      }
    }
  }
  // N prime or 4: the butterfly on v[0..N)
  __device__ __forceinline__ static void butterfly(C<T>* v, const C<T>* rt) {
    using V = C<T>;
    if constexpr (N == 2) {
      const V a = v[0], b = v[1];
      v[0] = cadd(a, b);
      v[1] = csub(a, b);
    } else if constexpr (N == 4) {
      const V a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]), a2 = cadd(v[1], v[3]), a3 = csub(v[1], v[3]);
      const V r3 = INV ? cmk<V>(-a3.y, a3.x) : cmk<V>(a3.y, -a3.x);
      v[0] = cadd(a0, a2);
      v[1] = cadd(a1, r3);
      v[2] = csub(a0, a2);
      v[3] = csub(a1, r3);
    } else if constexpr (N == 3) {
      const T s3 = (T)0.86602540378443864676;  // sin(2 pi / 3)
      const V v0 = v[0], t1 = cadd(v[1], v[2]), t3 = csub(v[1], v[2]);
      const V t2 = cmk<V>(v0.x - (T)0.5 * t1.x, v0.y - (T)0.5 * t1.y);
      const V r = INV ? cmk<V>(-s3 * t3.y, s3 * t3.x) : cmk<V>(s3 * t3.y, -s3 * t3.x);
      v[0] = cadd(v0, t1);
      v[1] = cadd(t2, r);
      v[2] = csub(t2, r);
    } else if constexpr (N == 5) {
      const T c1 = (T)0.30901699437494742410, c2 = (T)-0.80901699437494742410;
      const T s1 = (T)0.95105651629515357212, s2 = (T)0.58778525229247312917;
      const V v0 = v[0];
      const V t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
      const V a1 = cmk<V>(v0.x + c1 * t1.x + c2 * t2.x, v0.y + c1 * t1.y + c2 * t2.y);
      const V a2 = cmk<V>(v0.x + c2 * t1.x + c1 * t2.x, v0.y + c2 * t1.y + c1 * t2.y);
      const V b1 = cmk<V>(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y);
      const V b2 = cmk<V>(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y);
      const V mb1 = INV ? cmk<V>(-b1.y, b1.x) : cmk<V>(b1.y, -b1.x);
      const V mb2 = INV ? cmk<V>(-b2.y, b2.x) : cmk<V>(b2.y, -b2.x);
      v[0] = cadd(v0, cadd(t1, t2));
      v[1] = cadd(a1, mb1);
      v[2] = cadd(a2, mb2);
      v[3] = csub(a2, mb2);
      v[4] = csub(a1, mb1);
    } else {  // other primes: direct DFT
      V x[N];
#pragma unroll
      for (int j = 0; j < N; ++j) x[j] = v[j];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        V acc = x[0];
#pragma unroll
        for (int j = 1; j < N; ++j) {
          const int e = (j * k) % N;
          if (e == 0) {
            acc = cadd(acc, x[j]);
          } else {
            const V w = rt[e * RS];
            acc = INV ? cmacc(acc, x[j], w) : cmac(acc, x[j], w);
          }
        }
        v[k] = acc;
      }
    }
  }
};
template <typename T, bool INV, int RS>
struct ThreadDft<T, INV, 1, RS> {
  __device__ __forceinline__ static void run(C<T>*, const C<T>*) {}
};

// Transform dispatcher: the warp-level path for the lengths the plan marks,
// the Stockham stages otherwise.  Returns the buffer holding the result; all
// threads of the block must call it after the input is complete
// (__syncthreads()), and the result is complete for all threads on return.
template <typename T, bool INV, int A, int B, bool INL, bool PAD = false>
__device__ __forceinline__ void fft_warp_call(C<T>* buf, int nlines, int stride, const C<T>* roots) {
  if constexpr (INL)
    fft_lines_warp_body<T, INV, A, B, PAD>(buf, nlines, stride, roots);
  else
    fft_lines_warp<T, INV, A, B, PAD>(buf, nlines, stride, roots);
}

// INL: expand the warp-level transforms into the calling kernel.
// WIDE: also the 32-value shapes (lengths 512 and 1024).  They need about
// twice the registers, and a kernel's register allocation covers everything
// it calls, so only kernels instantiated with WIDE = true contain them; a
// plan with warp_a == 32 must only reach those (the host checks).
// PAD: the warp-level transforms use padded transpose rows (stride >=
// n + warp_a - 1).
// The wide shapes alone (kernels that only plans with warp_a == 32 reach).
template <typename T, bool INV, bool INL, bool PAD>
__device__ __forceinline__ void fft_wide(C<T>* a, int nlines, int stride, const FftPlan& p, const C<T>* tw) {
  if (p.warp_b == 32)
    fft_warp_call<T, INV, 32, 32, INL, PAD>(a, nlines, stride, tw + p.full_off);
  else
    fft_warp_call<T, INV, 32, 16, INL, PAD>(a, nlines, stride, tw + p.full_off);
  __syncthreads();
}

// (ODD: see fft_lines.)
template <typename T, bool INV, bool ODD, bool INL = false, bool WIDE = false, bool PAD = false>
__device__ C<T>* fft_run(C<T>* a, C<T>* b, int nlines, int stride, const FftPlan& p, const C<T>* tw) {
  if constexpr (WIDE) {
    if (p.warp_a == 32) {
      if (p.warp_b == 32)
        fft_warp_call<T, INV, 32, 32, INL, PAD>(a, nlines, stride, tw + p.full_off);
      else
        fft_warp_call<T, INV, 32, 16, INL, PAD>(a, nlines, stride, tw + p.full_off);
      __syncthreads();
      return a;
    }
  }
  if (p.warp_a == 16 && p.warp_b == 16) {
    fft_warp_call<T, INV, 16, 16, INL, PAD>(a, nlines, stride, tw + p.full_off);
  } else if (p.warp_a == 16 && p.warp_b == 8) {
    fft_warp_call<T, INV, 16, 8, INL, PAD>(a, nlines, stride, tw + p.full_off);
  } else if (p.warp_a == 8 && p.warp_b == 8) {
    fft_warp_call<T, INV, 8, 8, INL, PAD>(a, nlines, stride, tw + p.full_off);
  } else if (p.warp_a == 16 && p.warp_b == 2) {
    fft_warp_call<T, INV, 16, 2, INL, PAD>(a, nlines, stride, tw + p.full_off);
  } else if (p.warp_a == 8 && p.warp_b == 4) {
    fft_warp_call<T, INV, 8, 4, INL, PAD>(a, nlines, stride, tw + p.full_off);
  } else {
    return fft_lines<T, INV, ODD>(a, b, nlines, stride, p, tw);
  }
  __syncthreads();
  return a;
}

}  // namespace mmc

// kernels.cuh -- demag convolution passes, Metropolis sweep, energy and field
// kernels, templated on the working precision T (float or double).
//
// Included by kernels_f32.cu (built with multiply-add contraction) and
// kernels_f64.cu (built with -fmad=false so that FP64 results match the CPU
// oracle bit for bit where the operation order is the same).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "fft.cuh"
#include "lines64.cuh"
#include "mmc_internal.h"
#include "mmc_math.h"

namespace mmc {

// =========================================================== launch helpers
// Programmatic dependent launch: a kernel launched by launch_pdl may be
// scheduled before the previous kernel of its stream (or graph branch) has
// retired, and calls pdl_wait() before it reads anything a previous kernel
// writes or writes anything one reads; before the wait it touches only
// constant tables (transform roots and twiddles).  The previous kernels
// trigger implicitly when their CTAs exit: an explicit early trigger let the
// next grid's waiting CTAs take SM slots during the tail and cost 4 us per
// batched sweep.  The wait returns at once for a kernel launched without the
// attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// 16-byte asynchronous copy from global to shared memory.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// =========================================================== demag passes
//
// The reference computes H^ = K^ . M^ / N with three cuFFT R2C transforms and
// calHexchangeKernel (src/main.cu:868-884, src/demag_cu.cu:68-116) and never
// runs the inverse.  Here the convolution is complete and split into
//   x_forward : real rows -> half spectrum along x (two real rows per complex FFT)
//   col_pass  : complex FFT along y or z over tiles of kx columns, optionally
//               fused with the 3x3 tensor product and the inverse FFT
//   x_inverse : half spectrum -> real rows, cropped to the lattice
// Rows that are pure zero padding are never loaded (pruned transform).

// Real rows in[c][row][x] (x < xdata, zero up to p.n) -> S[c][z][y][kx], kx < hx.
// NC: components (3 for m, 6 for the tensor), fixed at compile time so the
// per-element work covers only the components that exist.  Three components
// come in lengths without a warp-level plan only (k_x_forward_w and its like take
// those).  ODD: see fft_lines.
// (Register budget in FP32: 64 per thread, 128 with the odd stages, whose 130
// left three CTAs of 128 threads per SM instead of four: 211 us for the demag
// field of an open 512^2 film instead of 199.)
template <typename T, bool ODD>
constexpr int x_min_blocks() {
  return sizeof(T) == 8 ? 1 : ODD ? 2 : 4;
}
template <typename T, int NC, bool ODD>
__global__ void __launch_bounds__(256, x_min_blocks<T, ODD>()) k_x_forward(FftPlan p, int xdata, FastDiv dyd, int nrows, const T* __restrict__ in,
                            long long in_cstride, C<T>* __restrict__ S, long long nspec, int nyp, FastDiv dhx,
                            int pitch, int rows_per_cta, long long in_rstride, long long s_rstride) {
  constexpr int ncomp = NC;
  const int hx = (int)dhx.d, ydata = (int)dyd.d;
  using V = C<T>;
  in += blockIdx.z * in_rstride;  // replica of a batch
  S += blockIdx.z * s_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* tw = reinterpret_cast<V*>(smem_raw);
  const int L = p.n;
  constexpr int npairs = (ncomp + 1) / 2;
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  V* bufA = tw + ((p.tw_total + 1) & ~1);
  V* bufB = bufA + (long long)rows_per_cta * npairs * L;
  load_twiddles<T>(p, tw);
  // loads are issued four elements per thread at a time, before any store, so
  // their latencies overlap
  const int total = nr * L;
  for (int base = threadIdx.x; base < total; base += 4 * blockDim.x) {
    T v[4][2 * npairs];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base + u * blockDim.x;
      const int rr = p.dn.div(idx), x = idx - rr * L;
      const bool ok = idx < total && x < xdata;
      const long long rbase = (long long)(row0 + rr) * xdata + x;
#pragma unroll
      for (int c = 0; c < 2 * npairs; ++c) v[u][c] = (ok && c < ncomp) ? in[c * in_cstride + rbase] : (T)0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base + u * blockDim.x;
      if (idx < total) {
        const int rr = p.dn.div(idx), x = idx - rr * L;
#pragma unroll
        for (int pr = 0; pr < npairs; ++pr)
          bufA[(long long)(rr * npairs + pr) * L + x] = cmk<V>(v[u][2 * pr], v[u][2 * pr + 1]);
      }
    }
  }
  __syncthreads();
  V* res;
  if constexpr (NC == 6)
    res = fft_run<T, false, ODD, false, true>(bufA, bufB, nr * npairs, L, p, tw);
  else
    res = fft_lines<T, false, ODD>(bufA, bufB, nr * npairs, L, p, tw);
  for (int idx = threadIdx.x; idx < nr * npairs * hx; idx += blockDim.x) {
    const int rest = dhx.div(idx);
    const int k = idx - rest * hx;
    const int rr = rest / npairs, pr = rest - rr * npairs;  // npairs is a compile-time 2 or 3
    const V* line = res + (long long)(rr * npairs + pr) * L;
    const V A = line[k];
    const V B = line[k == 0 ? 0 : L - k];
    const int row = row0 + rr;
    const int z = dyd.div(row), y = row - z * ydata;
    const long long off = ((long long)z * nyp + y) * pitch + k;
    const int ca = 2 * pr, cb = 2 * pr + 1;
    S[ca * nspec + off] = cmk<V>((T)0.5 * (A.x + B.x), (T)0.5 * (A.y - B.y));
    if (cb < ncomp) S[cb * nspec + off] = cmk<V>((T)0.5 * (A.y + B.y), (T)-0.5 * (A.x - B.x));
  }
}

// Half spectra S[0..2][z][y][kx] -> real rows out[c][row][x], x < xout.
template <typename T, bool ODD>
__global__ void __launch_bounds__(256, x_min_blocks<T, ODD>()) k_x_inverse(FftPlan p, const C<T>* __restrict__ S, long long nspec, int nyp, int hx, int pitch,
                            FastDiv dxo, FastDiv dyo, int nrows, T* __restrict__ out, long long out_cstride,
                            int rows_per_cta, long long s_rstride, long long out_rstride) {
  const int xout = (int)dxo.d, yout = (int)dyo.d;
  using V = C<T>;
  S += blockIdx.z * s_rstride;
  out += blockIdx.z * out_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* tw = reinterpret_cast<V*>(smem_raw);
  const int L = p.n;
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  V* bufA = tw + ((p.tw_total + 1) & ~1);
  V* bufB = bufA + (long long)rows_per_cta * 2 * L;
  load_twiddles<T>(p, tw);
  const int total = nr * L;
  for (int base0 = threadIdx.x; base0 < total; base0 += 4 * blockDim.x) {
    V v[4][3];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base0 + u * blockDim.x;
      const int rr = p.dn.div(idx), k = idx - rr * L;
      const int row = row0 + rr;
      const int z = dyo.div(row), y = row - z * yout;
      const long long base = ((long long)z * nyp + y) * pitch;
      const long long kk = k < hx ? k : L - k;
#pragma unroll
      for (int c = 0; c < 3; ++c) v[u][c] = idx < total ? S[c * nspec + base + kk] : cmk<V>(0, 0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int idx = base0 + u * blockDim.x;
      if (idx < total) {
        const int rr = p.dn.div(idx), k = idx - rr * L;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (k >= hx) v[u][c].y = -v[u][c].y;
          if (k == 0 || 2 * k == L) v[u][c].y = 0;  // bins that are real for a real output
        }
        bufA[(long long)(rr * 2) * L + k] = cmk<V>(v[u][0].x - v[u][1].y, v[u][0].y + v[u][1].x);
        bufA[(long long)(rr * 2 + 1) * L + k] = v[u][2];
      }
    }
  }
  __syncthreads();
  V* res = fft_lines<T, true, ODD>(bufA, bufB, nr * 2, L, p, tw);
  for (int idx = threadIdx.x; idx < nr * xout; idx += blockDim.x) {
    const int rr = dxo.div(idx), x = idx - rr * xout;
    const long long o = (long long)(row0 + rr) * xout + x;
    const V a = res[(long long)(rr * 2) * L + x];
    const V b = res[(long long)(rr * 2 + 1) * L + x];
    out[o] = a.x;
    out[out_cstride + o] = a.y;
    out[2 * out_cstride + o] = b.x;
  }
}

// ----------------------------------------------------- warp-shaped x passes
// The same two transforms for lengths with a warp-level plan (L = A * B):
// each line (a pair of components of one row) goes straight from global
// memory into the registers of its B lanes in the order the transform takes
// it (element b + B a in lane b of the group), so the input is never staged
// in shared memory, and the loops over rows and columns need no division.
// Same arithmetic as k_x_forward / k_x_inverse, so the results are the same
// bit for bit.  Shared memory: the L roots and one L-element line per
// (row, pair).
template <typename T>
__device__ __forceinline__ void load_roots(const FftPlan& p, C<T>* dst) {
  const C<T>* src = plan_tw<T>(p) + p.full_off;
  for (int i = threadIdx.x; i < p.n; i += blockDim.x) dst[i] = src[i];
}

// They serve the relaxation (f64s): FP32 lines have k_x_forward_r / k_x_inverse_r,
// FP64 ones the passes of lines64.cuh.  (Register budget: 128 per thread with 16
// values per lane, 255 with 32.)
template <int A>
constexpr int x_w_min_blocks() {
  return A >= 32 ? 1 : 2;
}
template <typename T, int A, int B>
__global__ void __launch_bounds__(256, x_w_min_blocks<A>()) k_x_forward_w(FftPlan p, int xdata, FastDiv dyd, int nrows, const T* __restrict__ in,
                              long long in_cstride, C<T>* __restrict__ S, long long nspec, int nyp, int hx,
                              int pitch, int rows_per_cta, long long in_rstride, long long s_rstride) {
  constexpr int L = A * B, GPW = 32 / B;
  using V = C<T>;
  const int ydata = (int)dyd.d;
  in += blockIdx.z * in_rstride;
  S += blockIdx.z * s_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LS = L + A;  // line stride: room for the padded transpose
  V* roots = reinterpret_cast<V*>(smem_raw);
  V* buf = roots + L;  // line pr * nr + rr: row rr, pair pr (mx + i my, mz + 0 i)
  load_roots<T>(p, roots);
  pdl_wait();
  __syncthreads();
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  const int nlines = 2 * nr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int grp = lane / B, b = lane - grp * B;
  // pair-major line order: the groups of a warp mostly load the same pair
  for (int line0 = warp * GPW; line0 < nlines; line0 += nwarps * GPW) {
    const int line = line0 + grp;
    const bool active = line < nlines;
    const int pr = line >= nr ? 1 : 0, rr = line - pr * nr;
    V v[A];
    if (active) {
      const T* re = in + (long long)(2 * pr) * in_cstride + (long long)(row0 + rr) * xdata;
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const int x = b + B * a;
        const bool ok = x < xdata;
        v[a] = cmk<V>(ok ? re[x] : (T)0, (ok && pr == 0) ? re[in_cstride + x] : (T)0);
      }
    }
    fft_line_regs<T, false, A, B, true>(v, buf + (active ? line : 0) * LS, b, active, roots);
  }
  __syncthreads();
  // split each pair into the half spectra of its two real rows
  for (int line = warp; line < nlines; line += nwarps) {
    const int pr = line >= nr ? 1 : 0, rr = line - pr * nr;
    const V* ln = buf + line * LS;
    const int row = row0 + rr;
    const int z = dyd.div(row), y = row - z * ydata;
    V* so = S + (long long)(2 * pr) * nspec + ((long long)z * nyp + y) * pitch;
    for (int k = lane; k < hx; k += 32) {
      const V Av = ln[k];
      const V Bv = ln[k == 0 ? 0 : L - k];
      so[k] = cmk<V>((T)0.5 * (Av.x + Bv.x), (T)0.5 * (Av.y - Bv.y));
      if (pr == 0) so[nspec + k] = cmk<V>((T)0.5 * (Av.y + Bv.y), (T)-0.5 * (Av.x - Bv.x));
    }
  }
}

template <typename T, int A, int B>
__global__ void __launch_bounds__(256, x_w_min_blocks<A>()) k_x_inverse_w(FftPlan p, const C<T>* __restrict__ S, long long nspec, int nyp, int hx, int pitch,
                              FastDiv dxo, FastDiv dyo, int nrows, T* __restrict__ out, long long out_cstride,
                              int rows_per_cta, long long s_rstride, long long out_rstride) {
  constexpr int L = A * B, GPW = 32 / B;
  using V = C<T>;
  const int xout = (int)dxo.d, yout = (int)dyo.d;
  S += blockIdx.z * s_rstride;
  out += blockIdx.z * out_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LS = L + A;  // line stride: room for the padded transpose
  V* roots = reinterpret_cast<V*>(smem_raw);
  V* buf = roots + L;  // line rr: hx + i hy of row rr; line nr + rr: hz
  load_roots<T>(p, roots);
  pdl_wait();
  __syncthreads();
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  const int nlines = 2 * nr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int grp = lane / B, b = lane - grp * B;
  for (int line0 = warp * GPW; line0 < nlines; line0 += nwarps * GPW) {
    const int line = line0 + grp;
    const bool active = line < nlines;
    const int pr = line >= nr ? 1 : 0, rr = line - pr * nr;
    V v[A];
    if (active) {
      const int row = row0 + rr;
      const int z = dyo.div(row), y = row - z * yout;
      const V* si = S + (long long)(2 * pr) * nspec + ((long long)z * nyp + y) * pitch;
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const int k = b + B * a;
        const int kk = k < hx ? k : L - k;
        V u0 = si[kk];
        if (k >= hx) u0.y = -u0.y;
        if (k == 0 || 2 * k == L) u0.y = 0;  // bins that are real for a real output
        if (pr == 0) {
          V u1 = si[nspec + kk];
          if (k >= hx) u1.y = -u1.y;
          if (k == 0 || 2 * k == L) u1.y = 0;
          v[a] = cmk<V>(u0.x - u1.y, u0.y + u1.x);
        } else {
          v[a] = u0;
        }
      }
    }
    fft_line_regs<T, true, A, B, true>(v, buf + (active ? line : 0) * LS, b, active, roots);
  }
  __syncthreads();
  for (int rr = warp; rr < nr; rr += nwarps) {
    const V* l0 = buf + rr * LS;
    const V* l1 = buf + (nr + rr) * LS;
    T* o = out + (long long)(row0 + rr) * xout;
    for (int x = lane; x < xout; x += 32) {
      const V a = l0[x];
      o[x] = a.x;
      o[out_cstride + x] = a.y;
      o[2 * out_cstride + x] = l1[x].x;
    }
  }
}

// The FP32 x passes.  The same lines, transforms and splits as k_x_forward_w /
// k_x_inverse_w, bit for bit, with each line finished by the warp that holds
// it: the split needs X[L - k] beside X[k], which sits in the mirrored lane's
// registers (two shuffles per value instead of a line written to shared memory
// and read back twice), and the inverse's rows go straight to global memory.
// Shared memory carries the transposes only, so the kernel has no barrier after
// its table of roots, which it holds in the lanes' order (the products b ka of
// the plain order meet in the same banks).  64 x 256^2: 26.9 -> 23.7 us forward
// and 28.5 -> 26.8 back; bound by the latency of its loads with the L1 path 70 to
// 74 % busy (56 and 51 % issue).
// SPLIT: m and h rows in the colour-split order (see k_mc_split): cell x of row
// (y, z) at split_pos(x, y + z, nx); a lane's values have one parity (B and A
// are even), so its addresses stay a base plus a compile-time step.
__host__ __device__ __forceinline__ int split_pos(int x, int yz, int nx) {
  return ((x + yz) & 1) * (nx >> 1) + (x >> 1);
}
template <int A>
constexpr int x_r_min_blocks() {
  return A >= 32 ? 2 : 4;
}
template <int A, int B>
__device__ __forceinline__ void load_lane_roots(const FftPlan& p, float2* dst) {
  const float2* src = p.tw32 + p.lane_off;
  for (int i = threadIdx.x; i < A * B; i += blockDim.x) dst[i] = src[i];
}
template <int A, int B, bool SPLIT>
__global__ void __launch_bounds__(256, x_r_min_blocks<A>())
    k_x_forward_r(FftPlan p, int xdata, FastDiv dyd, int nrows, const float* __restrict__ in, long long in_cstride,
                  float2* __restrict__ S, long long nspec, int nyp, int hx, int pitch, int rows_per_cta,
                  long long in_rstride, long long s_rstride) {
  using V = float2;
  constexpr int L = A * B, GPW = 32 / B, Q = A / B, LS = L + A;
  const int ydata = (int)dyd.d;
  in += blockIdx.z * in_rstride;
  S += blockIdx.z * s_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* roots = reinterpret_cast<V*>(smem_raw);
  load_lane_roots<A, B>(p, roots);
  pdl_wait();
  __syncthreads();
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  const int nlines = 2 * nr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int grp = lane / B, b = lane - grp * B;
  V* Lp = roots + L + (warp * GPW + grp) * LS;
  for (int line0 = warp * GPW; line0 < nlines; line0 += nwarps * GPW) {
    const int line = line0 + grp;
    const bool active = line < nlines;
    const int pr = line >= nr ? 1 : 0, row = row0 + (active ? line - pr * nr : 0);
    const int z = dyd.div(row), y = row - z * ydata;
    V v[A];
    if (active) {
      const float* re = in + (long long)(2 * pr) * in_cstride + (long long)row * xdata +
                        (SPLIT ? split_pos(b, y + z, xdata) : b);
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const int o = SPLIT ? B / 2 * a : B * a;
        const bool ok = b + B * a < xdata;
        v[a] = make_float2(ok ? re[o] : 0.0f, (ok && pr == 0) ? re[in_cstride + o] : 0.0f);
      }
    }
    fft_line_cols<float, false, A, B, true, true>(v, Lp, b, active, roots);
    V* so = S + (long long)(2 * pr) * nspec + ((long long)z * nyp + y) * pitch;
    // this lane's columns ka = b Q + t, the half kb < B / 2 (k < L / 2): the mirror
    // of X[ka + A kb] is X[A - ka + A (B - 1 - kb)] in lane B - b (t = 0) or
    // B - 1 - b (column Q - t there); lane 0's column 0 mirrors onto itself, kb to B - kb
#pragma unroll
    for (int kb = 0; kb < B / 2; ++kb) {
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const V a = v[t * B + kb];
        V m;
        if (t == 0) {
          const V s0 = v[(B - kb) & (B - 1)], s1 = v[B - 1 - kb];
          m.x = __shfl_sync(0xffffffffu, b == 0 ? s0.x : s1.x, (B - b) & (B - 1), B);
          m.y = __shfl_sync(0xffffffffu, b == 0 ? s0.y : s1.y, (B - b) & (B - 1), B);
        } else {
          const V s1 = v[(Q - t) * B + B - 1 - kb];
          m.x = __shfl_sync(0xffffffffu, s1.x, B - 1 - b, B);
          m.y = __shfl_sync(0xffffffffu, s1.y, B - 1 - b, B);
        }
        const int k = b * Q + t + A * kb;
        if (active) {
          so[k] = make_float2(0.5f * (a.x + m.x), 0.5f * (a.y - m.y));
          if (pr == 0) so[nspec + k] = make_float2(0.5f * (a.y + m.y), -0.5f * (a.x - m.x));
        }
      }
    }
    if (active && b == 0) {  // k = L / 2 mirrors onto itself
      const V a = v[B / 2];
      so[L / 2] = make_float2(0.5f * (a.x + a.x), 0.5f * (a.y - a.y));
      if (pr == 0) so[nspec + L / 2] = make_float2(0.5f * (a.y + a.y), -0.5f * (a.x - a.x));
    }
  }
}

template <int A, int B, bool SPLIT>
__global__ void __launch_bounds__(256, x_r_min_blocks<A>())
    k_x_inverse_r(FftPlan p, const float2* __restrict__ S, long long nspec, int nyp, int hx, int pitch, FastDiv dxo,
                  FastDiv dyo, int nrows, float* __restrict__ out, long long out_cstride, int rows_per_cta,
                  long long s_rstride, long long out_rstride) {
  using V = float2;
  constexpr int L = A * B, GPW = 32 / B, Q = A / B, LS = L + A;
  const int xout = (int)dxo.d, yout = (int)dyo.d;
  S += blockIdx.z * s_rstride;
  out += blockIdx.z * out_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* roots = reinterpret_cast<V*>(smem_raw);
  load_lane_roots<A, B>(p, roots);
  pdl_wait();
  __syncthreads();
  const int row0 = blockIdx.x * rows_per_cta;
  const int nr = min(rows_per_cta, nrows - row0);
  const int nlines = 2 * nr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int grp = lane / B, b = lane - grp * B;
  V* Lp = roots + L + (warp * GPW + grp) * LS;
  for (int line0 = warp * GPW; line0 < nlines; line0 += nwarps * GPW) {
    const int line = line0 + grp;
    const bool active = line < nlines;
    const int pr = line >= nr ? 1 : 0, row = row0 + (active ? line - pr * nr : 0);
    const int z = dyo.div(row), y = row - z * yout;
    V v[A];
    if (active) {
      const V* si = S + (long long)(2 * pr) * nspec + ((long long)z * nyp + y) * pitch;
#pragma unroll
      for (int a = 0; a < A; ++a) {
        const int k = b + B * a;
        const int kk = k < hx ? k : L - k;
        V u0 = si[kk];
        if (k >= hx) u0.y = -u0.y;
        if (k == 0 || 2 * k == L) u0.y = 0;  // bins that are real for a real output
        if (pr == 0) {
          V u1 = si[nspec + kk];
          if (k >= hx) u1.y = -u1.y;
          if (k == 0 || 2 * k == L) u1.y = 0;
          v[a] = make_float2(u0.x - u1.y, u0.y + u1.x);
        } else {
          v[a] = u0;
        }
      }
    }
    fft_line_cols<float, true, A, B, true, true>(v, Lp, b, active, roots);
    if (active) {
      float* o = out + (long long)(2 * pr) * out_cstride + (long long)row * xout;
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const int x0 = b * Q + t;
        float* ot = o + (SPLIT ? split_pos(x0, y + z, xout) : x0);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) {
          if (x0 + A * kb >= xout) continue;
          const int d = SPLIT ? A / 2 * kb : A * kb;
          ot[d] = v[t * B + kb].x;
          if (pr == 0) ot[out_cstride + d] = v[t * B + kb].y;
        }
      }
    }
  }
}

// PASS_SYM (with PASS_MUL): multiply by the real part of K^ only, i.e. by the
// spectrum of (K(r) + K(-r)) / 2 -- the symmetrised tensor of the energy's
// adjoint.
enum : int { PASS_FWD = 1, PASS_MUL = 2, PASS_INV = 4, PASS_SYM = 8 };

// Complex FFT along a strided axis (y or z) of tiles of `tx` consecutive kx
// columns.  Element (c, pos, col) lives at S[c*nspec + plane*plane_stride +
// pos*pos_stride + kx0 + col].  Loads pos < load_lim (zero above), stores
// pos < store_lim.  With PASS_MUL the tile is multiplied by the symmetric
// tensor spectrum (K^ . M^ / N, calHexchangeKernel) between the transforms.
template <typename T, bool INL, bool WIDE, bool ODD>
__device__ __forceinline__ void col_pass_body(const FftPlan& p, int ncomp, C<T>* __restrict__ S, long long nspec,
                                              const C<T>* __restrict__ khat, int hx, long long plane_stride,
                                              long long pos_stride, int load_lim, int store_lim, int flags, T inv_n,
                                              int tx, long long s_rstride, int lean) {
  using V = C<T>;
  S += blockIdx.z * s_rstride;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* tw = reinterpret_cast<V*>(smem_raw);
  const int L = p.n;
  const int stride = col_line_stride(p, sizeof(V));
  const int kx0 = blockIdx.x * tx;
  const int ntx = min(tx, hx - kx0);
  const long long pbase = (long long)blockIdx.y * plane_stride + kx0;
  const int nlines = ncomp * ntx;
  // lean 1 (warp-level transforms only): one buffer, transformed in place,
  // and the tensor read from global memory in the product -- a third of the
  // shared memory, so more CTAs fit on an SM.  lean 2: two buffers, the tensor
  // read from global memory (lines too long for the staged tensor tile).
  V* bufA = tw + ((p.tw_total + 1) & ~1);
  V* bufB = lean == 1 ? bufA : bufA + (long long)ncomp * tx * stride;
  V* ktile = bufB + (long long)ncomp * tx * stride;  // [comp][pos][t] when PASS_MUL and not lean
  load_twiddles<T>(p, tw);
  // the tensor tile goes to shared memory asynchronously while the forward
  // transform runs (16-byte copies when the tile rows are 16-byte aligned)
  const bool kasync = !lean && (flags & PASS_MUL) && (((long long)ntx * sizeof(V)) % 16 == 0) && ((kx0 * sizeof(V)) % 16 == 0) &&
                      ((plane_stride * sizeof(V)) % 16 == 0) && ((pos_stride * sizeof(V)) % 16 == 0);
  const FastDiv dt((uint32_t)ntx);  // index arithmetic without run-time division
  if ((flags & PASS_MUL) && !lean) {
    const int per = (int)(ntx * sizeof(V) / 16);
    if (kasync) {
      const FastDiv dper((uint32_t)per);
      for (int idx = threadIdx.x; idx < 6 * L * per; idx += blockDim.x) {
        const int rest = dper.div(idx), q = idx - rest * per;
        const int c = p.dn.div(rest), pos = rest - c * L;
        const int e = 16 / (int)sizeof(V);
        const unsigned sd = (unsigned)__cvta_generic_to_shared(ktile + ((long long)c * L + pos) * ntx + q * e);
        const V* src = khat + c * nspec + pbase + pos * pos_stride + q * e;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sd), "l"(src) : "memory");
      }
    } else {
      for (int idx = threadIdx.x; idx < 6 * L * ntx; idx += blockDim.x) {
        const int rest = dt.div(idx), t = idx - rest * ntx;
        const int c = p.dn.div(rest), pos = rest - c * L;
        ktile[((long long)c * L + pos) * ntx + t] = khat[c * nspec + pbase + pos * pos_stride + t];
      }
    }
  }
  pdl_wait();  // the spectrum is the previous pass's output
  // thread -> (column t, first position pos0); positions advance by pstep, so
  // the loops below need no division (tx is a power of two)
  const int lg = __ffs(tx) - 1;
  const int t = threadIdx.x & (tx - 1), pos0 = threadIdx.x >> lg, pstep = blockDim.x >> lg;
  const bool tok = t < ntx;
  constexpr int LB = 8;  // loads in flight per thread
  for (int c = 0; c < ncomp; ++c) {
    const V* src = S + c * nspec + pbase + t;
    V* dst = bufA + (long long)(c * ntx + t) * stride;
    for (int pos = pos0; pos < L; pos += LB * pstep) {
      V v[LB];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int q = pos + u * pstep;
        v[u] = (tok && q < load_lim) ? src[(long long)q * pos_stride] : cmk<V>(0, 0);
      }
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        const int q = pos + u * pstep;
        if (tok && q < L) dst[q] = v[u];
      }
    }
  }
  __syncthreads();
  V* cur = bufA;
  V* oth = bufB;
  if (flags & PASS_FWD) {
    V* r = cur;
    if constexpr (WIDE) fft_wide<T, false, INL, true>(cur, nlines, stride, p, tw);
    else r = fft_run<T, false, ODD, INL, false, true>(cur, oth, nlines, stride, p, tw);
    if (r != cur) {
      oth = cur;
      cur = r;
    }
  }
  if (flags & PASS_MUL) {
    if (kasync) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int pos = pos0; tok && pos < L; pos += pstep) {
      const V* kk = lean ? khat + pbase + pos * pos_stride + t : ktile + (long long)pos * ntx + t;
      const long long ks = lean ? nspec : (long long)L * ntx;
      V kxx = kk[0], kxy = kk[ks], kxz = kk[2 * ks];
      V kyy = kk[3 * ks], kyz = kk[4 * ks], kzz = kk[5 * ks];
      if (flags & PASS_SYM) kxx.y = kxy.y = kxz.y = kyy.y = kyz.y = kzz.y = (T)0;
      V* px = cur + (long long)(0 * ntx + t) * stride + pos;
      V* py = cur + (long long)(1 * ntx + t) * stride + pos;
      V* pz = cur + (long long)(2 * ntx + t) * stride + pos;
      const V mx = *px, my = *py, mz = *pz;
      const V hx_ = tensor_row(mx, my, mz, kxx, kxy, kxz);
      const V hy_ = tensor_row(mx, my, mz, kxy, kyy, kyz);
      const V hz_ = tensor_row(mx, my, mz, kxz, kyz, kzz);
      *px = cmk<V>(hx_.x * inv_n, hx_.y * inv_n);
      *py = cmk<V>(hy_.x * inv_n, hy_.y * inv_n);
      *pz = cmk<V>(hz_.x * inv_n, hz_.y * inv_n);
    }
    __syncthreads();
  }
  if (flags & PASS_INV) {
    V* r = cur;
    if constexpr (WIDE) fft_wide<T, true, INL, true>(cur, nlines, stride, p, tw);
    else r = fft_run<T, true, ODD, INL, false, true>(cur, oth, nlines, stride, p, tw);
    if (r != cur) {
      oth = cur;
      cur = r;
    }
  }
  if (tok) {
    for (int c = 0; c < ncomp; ++c) {
      V* dst = S + c * nspec + pbase + t;
      const V* src = cur + (long long)(c * ntx + t) * stride;
      for (int pos = pos0; pos < store_lim; pos += pstep) dst[(long long)pos * pos_stride] = src[pos];
    }
  }
}

template <typename T, bool INL, bool ODD>
__global__ void k_col_pass(FftPlan p, int ncomp, C<T>* __restrict__ S, long long nspec,
                           const C<T>* __restrict__ khat, int hx, long long plane_stride, long long pos_stride,
                           int load_lim, int store_lim, int flags, T inv_n, int tx, long long s_rstride, int lean) {
  col_pass_body<T, INL, false, ODD>(p, ncomp, S, nspec, khat, hx, plane_stride, pos_stride, load_lim, store_lim, flags,
                               inv_n, tx, s_rstride, lean);
}
// The same for the 32-value warp shapes (lengths 512 and 1024), at most 256
// threads: their registers would not fit more.
template <typename T, bool INL>
__global__ void __launch_bounds__(256) k_col_pass_wide(FftPlan p, int ncomp, C<T>* __restrict__ S, long long nspec,
                                                       const C<T>* __restrict__ khat, int hx, long long plane_stride,
                                                       long long pos_stride, int load_lim, int store_lim, int flags,
                                                       T inv_n, int tx, long long s_rstride, int lean) {
  col_pass_body<T, INL, true, false>(p, ncomp, S, nspec, khat, hx, plane_stride, pos_stride, load_lim, store_lim, flags,
                              inv_n, tx, s_rstride, lean);
}

// Column pass of FP32 films (the y lines, with the K^ product between the
// forward and the inverse transform) for lengths A B = 32, 64, 128 and 256, by
// persistent CTAs.  An item is a tile of TX kx columns of one replica; CTA i
// takes `chunk` items, consecutive replicas of one tile, so K^'s tile stays in
// shared memory (read once per CTA, before the wait on the x pass).  The next
// item's columns arrive by asynchronous copies while the current one is
// transformed, which is what the kernel is for: the register-held pass it
// replaces (three components per thread, 255 registers, 8 warps per SM) spent
// half of its time waiting for its loads.  Thread (c, b, t) of 3 B TX holds the
// values y = b + B a of component c of column t: the arithmetic of
// fft_line_cols forward, a meeting of the three components in shared memory
// for the product, and fft_line_cols inverse; each rounds as in k_col_pass, so
// the results are the same bit for bit.  Two CTAs of 192 threads per SM.
// 64 x 256^2: 48.4 -> 41 us; 4 x 256^2, a whole sweep: 22.1 -> 18.8.
template <int B>
__host__ __device__ constexpr int cp_tx() {
  return 64 / B;
}
template <int A, int B>
__host__ __device__ constexpr int cp_row() {  // transpose row: conflict-free both ways
  return B * cp_tx<B>() + (A == 8 ? 8 : 4);
}
template <int A, int B>
__host__ __device__ constexpr int cp_region() {  // one component's room: the tile's lines, then the transposes
  constexpr int L = A * B * cp_tx<B>(), T = A * cp_row<A, B>();
  return L > T ? L : T;
}
template <int A, int B>
__host__ __device__ constexpr size_t col_pipe_smem() {
  return ((size_t)6 * A * B * cp_tx<B>() + 2 * 3 * cp_region<A, B>()) * sizeof(float2);
}
// The 64 threads of one component meet (two whole warps).
__device__ __forceinline__ void cp_bar(int c) { asm volatile("bar.sync %0, 64;" ::"r"(c + 1) : "memory"); }

// The column's transform from v (positions b + B a) to v[t B + kb] = X[(b Q + t) + A kb].
template <bool INV, int A, int B>
__device__ __forceinline__ void cp_transform(float2 (&v)[A], float2* reg, const float2 (&tw)[A], int c, int b, int t) {
  constexpr int Q = A / B, TX = cp_tx<B>(), RW = cp_row<A, B>();
  RegDft<float, INV, A>::run(v);
#pragma unroll
  for (int ka = 1; ka < A; ++ka) {
    v[ka] = INV ? tmulc(v[ka], tw[ka]) : tmul(v[ka], tw[ka]);
  }
#pragma unroll
  for (int ka = 0; ka < A; ++ka) reg[ka * RW + b * TX + t] = v[ka];
  cp_bar(c);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
#pragma unroll
    for (int bb = 0; bb < B; ++bb) v[q * B + bb] = reg[(b * Q + q) * RW + bb * TX + t];
    RegDft<float, INV, B>::run(v + q * B);
  }
}

template <int A, int B>
__global__ void __launch_bounds__(192, 2)
    k_col_pipe(const __grid_constant__ FftPlan p, float2* __restrict__ S, long long nspec,
               const float2* __restrict__ khat, int hx, int pitch, int load_lim, int store_lim, int sym, float inv_n,
               int nrep, int items, int chunk) {
  using V = float2;
  constexpr int L = A * B, Q = A / B, TX = cp_tx<B>(), RG = cp_region<A, B>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* kt = reinterpret_cast<V*>(smem_raw);  // K^ tile [block][pos][t]
  V* buf0 = kt + 6 * L * TX;               // two buffers of three regions
  const int c = threadIdx.x >> 6, u = threadIdx.x & 63, t = u & (TX - 1), b = u / TX;
  const int i0 = blockIdx.x * chunk, i1 = min(items, i0 + chunk);
  // copies: thread u of a component's 64 moves the 16-byte piece lt of rows lr, lr + LR, ...
  constexpr int LR = 64 / (TX / 2);
  const int lr = u / (TX / 2), lt = 2 * (u & (TX / 2 - 1));
  auto load_k = [&](int tile) {
    const int kx = tile * TX + lt;
    if (kx < pitch) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const V* src = khat + (2 * c + q) * nspec + (long long)lr * pitch + kx;
        V* d = kt + ((2 * c + q) * L + lr) * TX + lt;
#pragma unroll 4
        for (int r = 0; r < L; r += LR) cp_async16(d + r * TX, src + (long long)r * pitch);
      }
    }
  };
  // item i's columns, rows load_lim and above 0
  auto load_item = [&](int i, V* buf) {
    const int tile = i / nrep, kx = tile * TX + lt;
    const V* src = S + ((long long)(i - tile * nrep) * 3 + c) * nspec + (long long)lr * pitch + kx;
    V* d = buf + c * RG + lr * TX + lt;
#pragma unroll
    for (int r = 0; r < L; r += LR) {
      if (lr + r < load_lim && kx < pitch)
        cp_async16(d + r * TX, src + (long long)r * pitch);
      else
        *reinterpret_cast<float4*>(d + r * TX) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  V tw[A];  // this thread's roots b ka
#pragma unroll
  for (int ka = 1; ka < A; ++ka) tw[ka] = p.tw32[p.lane_off + ka * B + b];
  int tile = i0 / nrep;
  load_k(tile);
  pdl_wait();  // the spectrum is the x pass's output
  load_item(i0, buf0);
  // row c of K^: (xx, xy, xz), (xy, yy, yz) or (xz, yz, zz) in the six blocks xx, xy, xz, yy, yz, zz
  const int o0 = c, o1 = c == 0 ? 1 : c == 1 ? 3 : 4, o2 = c == 0 ? 2 : c == 1 ? 4 : 5;
  for (int i = i0; i < i1; ++i) {
    V* buf = buf0 + ((i - i0) & 1) * 3 * RG;
    const int it = i / nrep;
    if (it != tile) {  // the chunk runs on into the next tile: every thread is past the last product
      tile = it;
      load_k(tile);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    cp_async_wait_all();
    __syncthreads();  // the item has landed; the other buffer is free
    if (i + 1 < i1) load_item(i + 1, buf0 + ((i + 1 - i0) & 1) * 3 * RG);
    V* reg = buf + c * RG;
    V v[A];
#pragma unroll
    for (int a = 0; a < A; ++a) v[a] = reg[(b + B * a) * TX + t];
    cp_bar(c);
    cp_transform<false, A, B>(v, reg, tw, c, b, t);
    cp_bar(c);
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
      for (int kb = 0; kb < B; ++kb) reg[(b * Q + q + A * kb) * TX + t] = v[q * B + kb];
    __syncthreads();
#pragma unroll
    for (int a = 0; a < A; ++a) {  // K^ . M^ / N
      const int e = (b + B * a) * TX + t;
      V k0 = kt[o0 * L * TX + e], k1 = kt[o1 * L * TX + e], k2 = kt[o2 * L * TX + e];
      if (sym) k0.y = k1.y = k2.y = 0.0f;
      V m0 = buf[e], m1 = buf[RG + e], m2 = buf[2 * RG + e];
      const V h = tensor_row(m0, m1, m2, k0, k1, k2);
      v[a] = make_float2(h.x * inv_n, h.y * inv_n);
    }
    __syncthreads();
    cp_transform<true, A, B>(v, reg, tw, c, b, t);
    const int kx = tile * TX + t;
    if (kx < hx) {
      V* dst = S + (long long)(i - it * nrep) * 3 * nspec + c * nspec + kx;
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int kb = 0; kb < B; ++kb) {
          const int pos = b * Q + q + A * kb;
          if (pos < store_lim) dst[(long long)pos * pitch] = v[q * B + kb];
        }
    }
  }
}
// Whether the pass has a k_col_pipe instance.
inline bool col_pipe_ok(const FftPlan& p) {
  return p.warp_a == 16 ? p.warp_b >= 8 : p.warp_a == 8;  // 256, 128, 64, 32
}
template <int A, int B>
cudaError_t launch_col_pipe_ab(const FftPlan& p, float2* S, long long nspec, const float2* khat, int hx, int pitch,
                               int load_lim, int store_lim, int sym, float inv_n, int nrep, cudaStream_t st) {
  const int tiles = (hx + cp_tx<B>() - 1) / cp_tx<B>();
  const long long items = (long long)tiles * nrep;
  if (items > INT_MAX) return cudaErrorInvalidValue;
  int dev = 0, nsm = 152;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int chunk = (int)((items + 2 * nsm - 1) / (2 * nsm));  // two CTAs per SM, all resident
  return launch_pdl(k_col_pipe<A, B>, dim3((unsigned)((items + chunk - 1) / chunk)), dim3(192), col_pipe_smem<A, B>(),
                    st, p, S, nspec, khat, hx, pitch, load_lim, store_lim, sym, inv_n, nrep, (int)items, chunk);
}
inline cudaError_t launch_col_pipe(const FftPlan& p, float2* S, long long nspec, const float2* khat, int hx, int pitch,
                                   int load_lim, int store_lim, int sym, float inv_n, int nrep, cudaStream_t st) {
  auto f = p.n == 256   ? launch_col_pipe_ab<16, 16>
           : p.n == 128 ? launch_col_pipe_ab<16, 8>
           : p.n == 64  ? launch_col_pipe_ab<8, 8>
                        : launch_col_pipe_ab<8, 4>;
  return f(p, S, nspec, khat, hx, pitch, load_lim, store_lim, sym, inv_n, nrep, st);
}

// One direction of an FP32 transform along y (or z), without the product:
// cl_tx columns of one component per CTA.  The lines go from global memory into
// the registers in the order the transform takes them and back from them, so
// shared memory is passed once, by the transpose, and the components and tiles
// are CTAs of their own whose loads, transforms and stores overlap.
// Bound by the latency of its loads with 16 warps per SM.  Against tiles of all
// three components staged in shared memory (k_col_pass, k_col_pass_wide), the
// demag field of a 512 x 512 x 8 slab: 97.9 -> 78.2 us, of 128 x 128 x 4 19.2 ->
// 14.1 us, of 64 x 64 x 2 14.5 -> 11.8 us.  (16 columns at length 512: the same; 4:
// 81 us; 5 CTAs per SM: 81 us.)
template <int B>
constexpr int cl_tx = B == 32 ? 4 : B == 16 ? 8 : 16;
template <bool INV, int A, int B>
__global__ void __launch_bounds__(cl_tx<B> * B, 4)
    k_col_lines(const __grid_constant__ FftPlan p, float2* __restrict__ S, long long nspec, int hx,
                long long plane_stride, long long pos_stride, int load_lim, int store_lim, long long s_rstride) {
  constexpr int TX = cl_tx<B>, Q = A / B, RW = B * TX + TX / Q;  // transpose row: conflict-free both ways
  __shared__ float2 reg[A * RW];
  const int rep = blockIdx.z / 3, c = blockIdx.z - 3 * rep;
  const int t = threadIdx.x & (TX - 1), b = threadIdx.x / TX, kx = blockIdx.x * TX + t;
  const bool mine = kx < hx;
  float2* s0 = S + rep * s_rstride + c * nspec + blockIdx.y * plane_stride + (mine ? kx : 0);
  const float2* tw = p.tw32 + p.lane_off + b;
  pdl_wait();
  float2 v[A];
#pragma unroll
  for (int a = 0; a < A; ++a) {
    const int pos = b + B * a;
    v[a] = mine && pos < load_lim ? s0[pos * pos_stride] : make_float2(0.0f, 0.0f);
  }
  RegDft<float, INV, A>::run(v);
#pragma unroll
  for (int ka = 1; ka < A; ++ka) {
    const float2 w = tw[ka * B];
    v[ka] = INV ? tmulc(v[ka], w) : tmul(v[ka], w);
  }
#pragma unroll
  for (int ka = 0; ka < A; ++ka) reg[ka * RW + b * TX + t] = v[ka];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
#pragma unroll
    for (int bb = 0; bb < B; ++bb) v[q * B + bb] = reg[(b * Q + q) * RW + bb * TX + t];
    RegDft<float, INV, B>::run(v + q * B);
  }
#pragma unroll
  for (int q = 0; q < Q; ++q)
#pragma unroll
    for (int kb = 0; kb < B; ++kb) {
      const int pos = b * Q + q + A * kb;
      if (mine && pos < store_lim) s0[pos * pos_stride] = v[q * B + kb];
    }
}
template <bool INV, int A, int B>
cudaError_t launch_col_lines_ab(const FftPlan& p, float2* S, long long nspec, int hx, int planes,
                                long long plane_stride, long long pos_stride, int load_lim, int store_lim,
                                long long s_rstride, int nrep, cudaStream_t st) {
  constexpr int TX = cl_tx<B>;
  return launch_pdl(k_col_lines<INV, A, B>, dim3((hx + TX - 1) / TX, planes, 3 * nrep), dim3(TX * B), 0, st, p, S,
                    nspec, hx, plane_stride, pos_stride, load_lim, store_lim, s_rstride);
}
template <bool INV>
cudaError_t launch_col_lines(const FftPlan& p, float2* S, long long nspec, int hx, int planes, long long plane_stride,
                             long long pos_stride, int load_lim, int store_lim, long long s_rstride, int nrep,
                             cudaStream_t st) {
  auto f = p.n == 1024  ? launch_col_lines_ab<INV, 32, 32>
           : p.n == 512 ? launch_col_lines_ab<INV, 32, 16>
           : p.n == 256 ? launch_col_lines_ab<INV, 16, 16>
           : p.n == 128 ? launch_col_lines_ab<INV, 16, 8>
           : p.n == 64  ? launch_col_lines_ab<INV, 8, 8>
                        : launch_col_lines_ab<INV, 8, 4>;
  return f(p, S, nspec, hx, planes, plane_stride, pos_stride, load_lim, store_lim, s_rstride, nrep, st);
}

// Column pass for short lines (n <= 16: the padded z axis of thin 3-D
// lattices, short y axes): csh_cols columns (kx, plane) per CTA, one thread per
// column and component with the line in registers, transformed by ThreadDft.
// For the product the threads exchange their lines through shared memory, each
// taking all three components of every third position, so that every word of
// the tensor is read once, its loads issued before the transform.
// Bound by the traffic of the tensor and the spectrum.  (One thread per column
// with all three lines: 255 registers, two CTAs per SM.)  Demag field of a
// 512 x 512 x 8 slab: 144 -> 98 us in FP32 (106 without the early tensor loads),
// 2122 -> 1215 us in FP64 with lines64.cuh's passes; 128 x 128 x 4: 23.4 -> 19.2 us.
// Same flags, product and tensor layout as k_col_pass.
template <typename T>
constexpr int csh_cols = sizeof(T) == 4 ? 64 : 32;
template <typename T, int N>
__global__ void __launch_bounds__(3 * csh_cols<T>, sizeof(T) == 4 ? 2 : 1)
    k_col_short(FftPlan p, C<T>* __restrict__ S, long long nspec, const C<T>* __restrict__ khat, FastDiv dhx, int hx,
                int total, long long plane_stride, long long pos_stride, int load_lim, int store_lim, int flags,
                T inv_n, long long s_rstride) {
  using V = C<T>;
  constexpr int CSH_COLS = csh_cols<T>, ZN = (N + 2) / 3;
  constexpr bool PRE = sizeof(T) == 4;
  __shared__ V rt[N];
  __shared__ V line[3][N][CSH_COLS];
  S += blockIdx.z * s_rstride;
  {
    const V* src = plan_tw<T>(p) + p.full_off;
    for (int i = threadIdx.x; i < N; i += blockDim.x) rt[i] = src[i];
  }
  const int c = threadIdx.x / CSH_COLS, j = threadIdx.x - c * CSH_COLS;
  const int col = blockIdx.x * CSH_COLS + j;
  const bool mine = col < total;
  const int plane = mine ? dhx.div(col) : 0, kx = mine ? col - plane * hx : 0;
  const long long base = plane * plane_stride + kx;
  V kk[PRE ? ZN : 1][6];
  if (PRE && (flags & PASS_MUL)) {
#pragma unroll
    for (int q = 0; q < ZN; ++q)
#pragma unroll
      for (int i = 0; i < 6; ++i)
        if (c + 3 * q < N) kk[q][i] = khat[i * nspec + base + (c + 3 * q) * pos_stride];
  }
  pdl_wait();
  __syncthreads();
  V* s0 = S + c * nspec + base;
  V v[N];
#pragma unroll
  for (int z = 0; z < N; ++z) v[z] = z < load_lim ? s0[z * pos_stride] : cmk<V>(0, 0);
  if (flags & PASS_FWD) ThreadDft<T, false, N, 1>::run(v, rt);
  if (flags & PASS_MUL) {
#pragma unroll
    for (int z = 0; z < N; ++z) line[c][z][j] = v[z];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < ZN; ++q) {
      const int z = c + 3 * q;
      if (z < N) {
        V k[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          k[i] = PRE ? kk[PRE ? q : 0][i] : khat[i * nspec + base + z * pos_stride];
          if (flags & PASS_SYM) k[i].y = (T)0;
        }
        const V mx = line[0][z][j], my = line[1][z][j], mz = line[2][z][j];
        const V hx_ = tensor_row(mx, my, mz, k[0], k[1], k[2]);
        const V hy_ = tensor_row(mx, my, mz, k[1], k[3], k[4]);
        const V hz_ = tensor_row(mx, my, mz, k[2], k[4], k[5]);
        line[0][z][j] = cmk<V>(hx_.x * inv_n, hx_.y * inv_n);
        line[1][z][j] = cmk<V>(hy_.x * inv_n, hy_.y * inv_n);
        line[2][z][j] = cmk<V>(hz_.x * inv_n, hz_.y * inv_n);
      }
    }
    __syncthreads();
#pragma unroll
    for (int z = 0; z < N; ++z) v[z] = line[c][z][j];
  }
  if (flags & PASS_INV) ThreadDft<T, true, N, 1>::run(v, rt);
#pragma unroll
  for (int z = 0; z < N; ++z)
    if (mine && z < store_lim) s0[z * pos_stride] = v[z];
}

// The short-line kernel for length n, or null.
template <typename T>
using ColShortFn = void (*)(FftPlan, C<T>*, long long, const C<T>*, FastDiv, int, int, long long, long long, int, int,
                            int, T, long long);
template <typename T>
ColShortFn<T> col_short_kernel(int n) {
  switch (n) {
#define MMC_CS(N_) \
  case N_:         \
    return k_col_short<T, N_>;
    MMC_CS(2) MMC_CS(3) MMC_CS(4) MMC_CS(5) MMC_CS(6) MMC_CS(7) MMC_CS(8) MMC_CS(9) MMC_CS(10) MMC_CS(11)
    MMC_CS(12) MMC_CS(13) MMC_CS(14) MMC_CS(15) MMC_CS(16)
#undef MMC_CS
    default:
      return nullptr;
  }
}

// =========================================================== lattice helpers
// Neighbour index along an axis, or -1 when the bond does not exist (open
// edge, or a periodic axis of length 1 where the neighbour is the cell itself).
__device__ __forceinline__ long long nbr_idx(const Geom& g, int x, int y, int z, int axis, int dir) {
  int c[3] = {x, y, z};
  const int n[3] = {g.nx, g.ny, g.nz};
  int v = c[axis] + dir;
  if (v < 0 || v >= n[axis]) {
    if (!g.per[axis]) return -1;
    v = v < 0 ? v + n[axis] : v - n[axis];
  }
  if (v == c[axis]) return -1;
  c[axis] = v;
  return c[0] + (long long)g.nx * (c[1] + (long long)g.ny * c[2]);
}

// nbr_idx from the cell's own index i: a step of +-stride, wrapped on a
// periodic axis; the same result without rebuilding the index.
__device__ __forceinline__ long long nbr_step(const Geom& g, long long i, int x, int y, int z, int axis, int dir) {
  const int n = axis == 0 ? g.nx : axis == 1 ? g.ny : g.nz;
  const int c = axis == 0 ? x : axis == 1 ? y : z;
  const long long stride = axis == 0 ? 1 : axis == 1 ? (long long)g.nx : (long long)g.nx * g.ny;
  const int v = c + dir;
  long long j = i + dir * stride;
  if (v < 0 || v >= n) {
    if (!g.per[axis]) return -1;
    j += v < 0 ? n * stride : -n * stride;
  }
  return n == 1 ? -1 : j;  // a periodic axis of length 1 wraps onto the cell itself
}

__device__ __forceinline__ int axis_color(int v, int n, int per) {
  if (per && (n & 1) && n > 1 && v == n - 1) return 2;
  return v & 1;
}

__device__ __forceinline__ int cell_color(const Geom& g, int x, int y, int z) {
  int s = axis_color(x, g.nx, g.per[0]) + axis_color(y, g.ny, g.per[1]) + axis_color(z, g.nz, g.per[2]);
  return g.ncolors == 2 ? (s & 1) : (s % 3);
}

// =========================================================== Metropolis sweep
//
// One sublattice colour of one sweep.  This replaces mcKernel2
// (src/mc_sampling.h:27-41, launched src/main.cu:1101-1120), whose body is not
// published.  Cells of one colour share no exchange or DMI bond, so they are
// updated in place concurrently.  For cell i:
//   F   = sum_a wex_a sum_(+-) m_nbr + DMI(nbr) + cz + cd (h_i - K0 m_i)
//   dE  = -(m' - m).F - can[(m'.u)^2 - (m.u)^2] - cd/2 [m'K0m' - mK0m]   (units of kT)
//   accept when dE <= 0 or u < exp(-dE)
// with (u0, u1, u) = Philox4x32-10(key = seed; counter = (i, sweep, stage, 0)),
// m' = (sqrt(1-z^2) cos 2 pi u1, sqrt(1-z^2) sin 2 pi u1, z = 2 u0 - 1).
template <typename T>
struct Prop;

template <>
struct Prop<double> {
  // The direction of the random words rx, ry: z = 2 u0 - 1, phi = 2 pi u1 with
  // u = (r + 1/2) 2^-32.  The steps of mmcm::u01_f64 and mmcm::sincospi, bit
  // for bit; what they do exactly (the uniforms, the split of 2 u1 into
  // quadrants) is done on the integers, which leaves 60 FP64 operations.
  static __device__ __forceinline__ double height(uint32_t rx) {  // (2 rx + 1 - 2^32) 2^-32
    return __longlong_as_double(0x4138000000000000ll + 2 * (long long)(int)(rx ^ 0x80000000u) + 1) - 0x1.8p20;
  }
  static __device__ __forceinline__ double radius(double z) {
    const double t = 1.0 - z * z;  // >= 0: |z| < 1
    return mmcm::dsqrt(t);
  }
  static __device__ __forceinline__ uint32_t halves(uint32_t ry) { return (ry >> 30) + ((ry >> 29) & 1u); }
  static __device__ __forceinline__ int quadrant(uint32_t ry) { return (int)(halves(ry) & 3u); }
  static __device__ __forceinline__ double quarter(uint32_t ry) {  // 2 u1 less its nearest half
    const int j = (int)(2u * ry + 1u - (halves(ry) << 31));
    return __longlong_as_double(0x4138000000000000ll + (long long)j) - 0x1.8p20;
  }
  static __device__ __forceinline__ void direction(uint32_t rx, uint32_t ry, double& px, double& py, double& pz) {
    pz = height(rx);
    const double s = radius(pz);
    double sn, cs;
    mmcm::sincospi_reduced(quadrant(ry), quarter(ry), &sn, &cs);
    px = s * cs;
    py = s * sn;
  }
  // The exponential's 50 operations only where the hardware's (see mc_filter)
  // cannot tell: dE is known to 2^-52 here, so the sides differ by 1e-5.
  __device__ static bool accept(double dE, double ua) {
    if (dE <= 0.0) return true;
    const float x = fminf((float)dE, 30.0f), e = __expf(-x), u = (float)ua;
    if (u > 1.00002f * e) return false;
    if (dE < 30.0 && u * 1.00002f < e) return true;
    return ua < mmcm::exp(-dE);
  }
};

template <>
struct Prop<float> {
  // FP32: the hardware sine and cosine of phi - pi in (-pi, pi), where their
  // absolute error is about 4e-7, negated (exact), and sqrt(t) as t / sqrt(t)
  // from the hardware reciprocal square root; t = 1 - z^2 >= 2^-22 because
  // u01_f32 never returns 0 or 1.
  // The flush-to-zero forms of rsqrt and ex2 skip the scaling of denormal
  // arguments and results: t is normal, and a denormal exponential loses
  // against every ua >= 2^-24 like 0 does.
  // (r >> 9) + 1/2 in units of 2^-23, as mmcm::u01_f32: the word's upper bits
  // become the mantissa of a number in [1, 2), and 1 - 2^-24 comes off exactly.
  __device__ static float u01(uint32_t r) { return __uint_as_float((r >> 9) + 0x3f800000u) - 0x1.fffffep-1f; }
  __device__ static void draw(mmcm::u32x4 r, float& px, float& py, float& pz, float& ua) {
    pz = 2.0f * u01(r.x) - 1.0f;
    const float t = 1.0f - pz * pz;
    float q;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(t));
    const float s = t * q;
    float sn, cs;
    __sincosf(6.28318530717958647692f * u01(r.y) - 3.14159265358979323846f, &sn, &cs);
    px = -(s * cs);
    py = -(s * sn);
    ua = u01(r.z);
  }
  __device__ static bool accept(float dE, float ua) {
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-dE * 1.44269504088896340736f));
    return dE <= 0.0f || ua < e;
  }
};

// Neighbour values of one trial: v[a][s] is the neighbour along axis a on side
// s (0 = -, 1 = +); has[a][s] tells whether that bond exists.
template <typename T>
struct Nbrs {
  T v[3][2][3];
  bool has[3][2];
};

// Proposal of one trial: Philox4x32-10(key = seed; counter = (cell, sweep,
// stage, 0)).  FP32: the direction m' and the acceptance uniform; FP64: the
// random words, from which the direction is made for accepted trials only.
template <typename T>
struct Proposal {
  T x, y, z, ua;
  __device__ __forceinline__ void get(T& px, T& py, T& pz) const {
    px = x;
    py = y;
    pz = z;
  }
};
template <>
struct Proposal<double> {
  uint32_t rx, ry, rz;
  __device__ __forceinline__ void get(double& px, double& py, double& pz) const {
    Prop<double>::direction(rx, ry, px, py, pz);
  }
};

template <typename T>
__device__ __forceinline__ Proposal<T> mc_propose(uint32_t key0, uint32_t key1, uint32_t cell, uint32_t stage,
                                                  uint32_t sweep) {
  mmcm::u32x4 ctr = {cell, sweep, stage, mmcm::STREAM_SWEEP};
  mmcm::u32x4 r = mmcm::philox4x32_10(ctr, key0, key1);
  Proposal<T> p;
  if constexpr (sizeof(T) == 8) {
    p.rx = r.x;
    p.ry = r.y;
    p.rz = r.z;
  } else {
    Prop<T>::draw(r, p.x, p.y, p.z, p.ua);
  }
  return p;
}

template <typename T>
__device__ __forceinline__ Proposal<T> mc_propose(const McCoef<T>& c, uint32_t cell, uint32_t stage, uint32_t sweep) {
  return mc_propose<T>(c.key0, c.key1, cell, stage, sweep);
}

// ---------------------------------------------- the FP64 trial's FP32 filter
// GB300 issues 1.7 FP64 operations per SM and cycle, so an FP64 trial costs
// what its FP64 operations cost: about 230 when everything is evaluated
// (60 for the direction, 110 for dE, 50 for the exponential).  The filter
// evaluates the same trial in FP32 with a bound on the distance from what the
// FP64 formula gives and decides when the bound allows only one answer; the
// FP64 formula decides the rest.  The decisions are the FP64 formula's, all of
// them.
//
// The bound: with M >= every |component| of m involved (at least 1), H the
// same for h, and G = gm M + gc + |cd| H >= |F_a| for each component of the
// field (McFilter), dE = -d . F in the regrouped form of mc_accept<float>.
// - On any path from an input of F to dE the FP32 evaluation makes at most 32
//   roundings of 2^-24 (2 for a truncated input, 1 for a coefficient, 16 in a
//   component of F, 3 in d and 3 in the dot product), each on terms that add up to
//   at most |d|_1 G: 1.9e-6 |d|_1 G.
// - The direction m' and the cell's own m enter d itself, by absolute errors.  An
//   error e of a component of either changes dE by at most e G (1 + |d|_1 / 4):
//   through d, and through the K0 and anisotropy terms of F, whose coefficients
//   are in G at least fourfold.  The errors add up over the components to 9.2e-7
//   for m' (rsqrtf 2 ulp, t = (1 + z)(1 - z) from two rounded factors and their
//   product, r = t / sqrt(t): 3.9e-7 of r, at most 5.5e-7 in x and y together;
//   the angle's rounding 1.3e-7; sincospif 1 ulp each 1.2e-7; the products 9e-8; z
//   3e-8) and to 2^-23 |m|_1 <= 2.1e-7 for m, truncated: together 1.13e-6 G +
//   0.28e-6 |d|_1 G.
// FP64 rounding is 1e-9 of either.  MC_FILTER_EPS = 2.2e-6 times (|d|_1 + 1) G
// covers the sum, 2.2e-6 |d|_1 G + 1.13e-6 G, for unit vectors; the rest of its
// constant part covers an m of another length.
// exp: the hardware's is within 2 + 1.173 |x| ulp, 4.5e-6 for x >= -30; below
// that the smallest uniform (2^-33) decides alone.  MC_FILTER_EXP = 2e-5 covers
// it and the rounding of the uniform.  NaN or infinity anywhere leaves both
// comparisons false: unsure.
constexpr float MC_FILTER_EPS = 2.2e-6f;
constexpr float MC_FILTER_EXP = 2e-5f;
enum McVerdict : int { MC_REJECT = 0, MC_ACCEPT = 1, MC_UNSURE = 2 };

// x truncated to FP32 by integer operations (a conversion instruction runs at
// the FP64 rate): below 2^-126 a denormal or 0, from 2^128 on NaN or infinity.
__device__ __forceinline__ float f32_trunc(double x) {
  const int hi = __double2hiint(x);
  const int e = __vimin_s32_relu((hi & 0x7fffffff) - 0x38000000, 0x0fffffff);
  const unsigned b = __funnelshift_l((unsigned)__double2loint(x), (unsigned)e, 3);
  return __uint_as_float(b | ((unsigned)hi & 0x80000000u));
}
__device__ __forceinline__ float f32_trunc(float x) { return x; }

// Neighbour values v (meaningful where has is true) and their flags, own cell
// o, demag field h (0 when the demag term is off); film: no z neighbours.
__device__ __forceinline__ McVerdict mc_filter(const McFilter& c, const float (&v)[3][2][3], const bool (&has)[3][2],
                                               float ox, float oy, float oz, float hx, float hy, float hz,
                                               uint32_t rx, uint32_t ry, uint32_t rz, bool film) {
  float Fx = c.cz[0], Fy = c.cz[1], Fz = c.cz[2];
  float M = fmaxf(fmaxf(fabsf(ox), fabsf(oy)), fmaxf(fabsf(oz), 1.0f));
  // NaN does not survive fmaxf: a sum that it does survive joins the bound
  float nan0 = 0.0f * (ox + oy + oz);
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (!has[a][s]) continue;
      const float x = v[a][s][0], y = v[a][s][1], z = v[a][s][2];
      Fx = fmaf(c.wex[a], x, Fx);
      Fy = fmaf(c.wex[a], y, Fy);
      Fz = fmaf(c.wex[a], z, Fz);
      M = fmaxf(M, fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))));
      if (a < 2) {  // DMI: (d_x m_z, d_y m_z, -d_x m_x - d_y m_y)
        const float w = s ? c.wdm[a] : -c.wdm[a];
        if (a == 0) Fx = fmaf(w, z, Fx);
        if (a == 1) Fy = fmaf(w, z, Fy);
        Fz = fmaf(-w, a == 0 ? x : y, Fz);
      }
    }
  const float a0 = fmaf((float)rx, 0x1p-31f, 0x1p-32f), a1 = fmaf((float)~rx, 0x1p-31f, 0x1p-32f);  // 1 + z, 1 - z
  const float t = a0 * a1;
  const float r = t * rsqrtf(t);
  float sn, cs;
  sincospif((float)(int)(ry ^ 0x80000000u) * 0x1p-31f, &sn, &cs);
  const float px = -(r * cs), py = -(r * sn), pz = (float)(int)(rx ^ 0x80000000u) * 0x1p-31f;
  const float dx = px - ox, dy = py - oy, dz = pz - oz;
  Fx = fmaf(c.cd, hx, Fx) + fmaf(c.k0h[0], dx, fmaf(c.k0h[1], dy, c.k0h[2] * dz));
  Fy = fmaf(c.cd, hy, Fy) + fmaf(c.k0h[1], dx, fmaf(c.k0h[3], dy, c.k0h[4] * dz));
  Fz = fmaf(c.cd, hz, Fz) + fmaf(c.k0h[2], dx, fmaf(c.k0h[4], dy, c.k0h[5] * dz));
  const float su = fmaf(px + ox, c.u[0], fmaf(py + oy, c.u[1], (pz + oz) * c.u[2]));
  const float cu = c.can * su;
  Fx = fmaf(cu, c.u[0], Fx);
  Fy = fmaf(cu, c.u[1], Fy);
  Fz = fmaf(cu, c.u[2], Fz);
  const float mdE = fmaf(dx, Fx, fmaf(dy, Fy, dz * Fz));  // -dE
  const float H = fmaxf(fabsf(hx), fmaxf(fabsf(hy), fabsf(hz)));
  nan0 += 0.0f * mdE;
  const float D = fabsf(dx) + fabsf(dy) + fabsf(dz);
  const float eps = fmaf(MC_FILTER_EPS * (D + 1.0f), fmaf(film ? c.gm : c.gm + c.gz, M, fmaf(fabsf(c.cd), H, c.gc)), nan0);
  const float ua = fmaf((float)rz, 0x1p-32f, 0x1p-33f);
  const float lo = mdE - eps, hi = fmaxf(mdE + eps, -30.0f);
  if (lo >= 0.0f || ua * (1.0f + MC_FILTER_EXP) < __expf(lo)) return MC_ACCEPT;
  // fmaxf drops a NaN: ask for a finite bound as well
  if (eps < 1e30f && ua > (1.0f + MC_FILTER_EXP) * __expf(hi)) return MC_REJECT;
  return MC_UNSURE;
}

// The Metropolis decision for one cell from its neighbour values, its own m,
// its demag field h and its proposal.  Shared by every sweep kernel, so that they
// round alike but for sep.
// sep (FP32): in the components of this mask the second neighbour's product is
// rounded before it is added, where the chain of multiply-adds rounds it with the
// sum.  k_mc_quad, k_mc_split and k_mc_pipe take what mc_sep says, every other
// form the chain; written out, it does not depend on what the compiler makes of
// the code around.
template <typename T>
__device__ __forceinline__ bool mc_accept_formula(const McCoef<T>& c, const Nbrs<T>& nb, T ox, T oy, T oz, T hx, T hy,
                                                  T hz, T px, T py, T pz, T ua, int sep = 0) {
  T Fx = 0, Fy = 0, Fz = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (!nb.has[a][s]) continue;
      if constexpr (sizeof(T) == 4) {
        const float w = c.wex[a], x = nb.v[a][s][0], y = nb.v[a][s][1], z = nb.v[a][s][2];
        const bool second = a == 0 && s == 1;
        Fx = second && (sep & 1) ? __fadd_rn(Fx, __fmul_rn(w, x)) : __fmaf_rn(w, x, Fx);
        Fy = second && (sep & 2) ? __fadd_rn(Fy, __fmul_rn(w, y)) : __fmaf_rn(w, y, Fy);
        Fz = second && (sep & 4) ? __fadd_rn(Fz, __fmul_rn(w, z)) : __fmaf_rn(w, z, Fz);
        continue;
      }
      Fx = Fx + c.wex[a] * nb.v[a][s][0];
      Fy = Fy + c.wex[a] * nb.v[a][s][1];
      Fz = Fz + c.wex[a] * nb.v[a][s][2];
    }
  const T dxmz = (nb.has[0][1] ? nb.v[0][1][2] : (T)0) - (nb.has[0][0] ? nb.v[0][0][2] : (T)0);
  const T dxmx = (nb.has[0][1] ? nb.v[0][1][0] : (T)0) - (nb.has[0][0] ? nb.v[0][0][0] : (T)0);
  const T dymz = (nb.has[1][1] ? nb.v[1][1][2] : (T)0) - (nb.has[1][0] ? nb.v[1][0][2] : (T)0);
  const T dymy = (nb.has[1][1] ? nb.v[1][1][1] : (T)0) - (nb.has[1][0] ? nb.v[1][0][1] : (T)0);
  Fx = Fx + c.wdm[0] * dxmz;
  Fy = Fy + c.wdm[1] * dymz;
  Fz = Fz - (c.wdm[0] * dxmx + c.wdm[1] * dymy);
  Fx = Fx + c.cz[0];
  Fy = Fy + c.cz[1];
  Fz = Fz + c.cz[2];
  if constexpr (sizeof(T) == 4) {
    // FP32: the same energy difference regrouped with d = m' - m, s = m' + m
    // and K0 symmetric,
    //   dE = -d . [F_local + cd h + (cd / 2) K0 d + can (s . u) u],
    // where F_local is the exchange, DMI and Zeeman part of F: the terms in
    // K0 m cancel, and the quadratic forms need no difference of squares.
    const T ddx = px - ox, ddy = py - oy, ddz = pz - oz;
    if (c.cd != (T)0) {
      Fx = Fx + c.cd * hx + (c.k0h[0] * ddx + c.k0h[1] * ddy + c.k0h[2] * ddz);
      Fy = Fy + c.cd * hy + (c.k0h[1] * ddx + c.k0h[3] * ddy + c.k0h[4] * ddz);
      Fz = Fz + c.cd * hz + (c.k0h[2] * ddx + c.k0h[4] * ddy + c.k0h[5] * ddz);
    }
    const T su = (px + ox) * c.u[0] + (py + oy) * c.u[1] + (pz + oz) * c.u[2];
    const T cs = c.can * su;
    Fx = Fx + cs * c.u[0];
    Fy = Fy + cs * c.u[1];
    Fz = Fz + cs * c.u[2];
    return Prop<T>::accept(-(ddx * Fx + ddy * Fy + ddz * Fz), ua);
  }
  if (c.cd != (T)0) {
    const T sx = c.k0[0] * ox + c.k0[1] * oy + c.k0[2] * oz;
    const T sy = c.k0[1] * ox + c.k0[3] * oy + c.k0[4] * oz;
    const T sz = c.k0[2] * ox + c.k0[4] * oy + c.k0[5] * oz;
    Fx = Fx + c.cd * (hx - sx);
    Fy = Fy + c.cd * (hy - sy);
    Fz = Fz + c.cd * (hz - sz);
  }
  const T ddx = px - ox, ddy = py - oy, ddz = pz - oz;
  T dE = -(ddx * Fx + ddy * Fy + ddz * Fz);
  const T pun = px * c.u[0] + py * c.u[1] + pz * c.u[2];
  const T puo = ox * c.u[0] + oy * c.u[1] + oz * c.u[2];
  dE = dE - c.can * (pun * pun - puo * puo);
  if (c.cd != (T)0) {
    const T qn = px * (c.k0[0] * px + c.k0[1] * py + c.k0[2] * pz) + py * (c.k0[1] * px + c.k0[3] * py + c.k0[4] * pz) +
                 pz * (c.k0[2] * px + c.k0[4] * py + c.k0[5] * pz);
    const T qo = ox * (c.k0[0] * ox + c.k0[1] * oy + c.k0[2] * oz) + oy * (c.k0[1] * ox + c.k0[3] * oy + c.k0[4] * oz) +
                 oz * (c.k0[2] * ox + c.k0[4] * oy + c.k0[5] * oz);
    dE = dE - (T)0.5 * c.cd * (qn - qo);
  }
  return Prop<T>::accept(dE, ua);
}

// The decision; p's direction is the new m where it is true.
template <typename T>
__device__ __forceinline__ bool mc_accept(const McCoef<T>& c, const Nbrs<T>& nb, T ox, T oy, T oz, T hx, T hy, T hz,
                                          const Proposal<T>& p, int sep = 0) {
  if constexpr (sizeof(T) == 8) {
    float v[3][2][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int k = 0; k < 3; ++k) v[a][s][k] = f32_trunc(nb.v[a][s][k]);
    const McVerdict w = mc_filter(c.f, v, nb.has, f32_trunc(ox), f32_trunc(oy), f32_trunc(oz), f32_trunc(hx),
                                  f32_trunc(hy), f32_trunc(hz), p.rx, p.ry, p.rz,
                                  !nb.has[2][0] && !nb.has[2][1]);
    if (w != MC_UNSURE) return w == MC_ACCEPT;
    T px, py, pz;
    p.get(px, py, pz);
    return mc_accept_formula<T>(c, nb, ox, oy, oz, hx, hy, hz, px, py, pz, mmcm::u01_f64(p.rz));
  } else {
    return mc_accept_formula<T>(c, nb, ox, oy, oz, hx, hy, hz, p.x, p.y, p.z, p.ua, sep);
  }
}

// The neighbours of cell i = (x, y, z), read as U (T, or float for the filter).
template <typename T, typename U>
__device__ __forceinline__ U mc_read(const T* p) {
  if constexpr (sizeof(T) == sizeof(U)) return *p;
  else return f32_trunc(*p);
}
template <typename T, typename U>
__device__ __forceinline__ void mc_nbrs(const Geom& g, const T* __restrict__ m, long long i, int x, int y, int z,
                                        Nbrs<U>& nb) {
  const T* mx = m;
  const T* my = m + g.n;
  const T* mz = m + 2 * g.n;
  const bool film = g.nz == 1;  // no z bonds: skip their index work and loads
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      if (a == 2 && film) {
        nb.has[a][s] = false;
        nb.v[a][s][0] = nb.v[a][s][1] = nb.v[a][s][2] = (U)0;
        continue;
      }
      const long long j = nbr_step(g, i, x, y, z, a, s ? 1 : -1);
      nb.has[a][s] = j >= 0;
      const long long jj = j >= 0 ? j : i;
      nb.v[a][s][0] = mc_read<T, U>(mx + jj);
      nb.v[a][s][1] = mc_read<T, U>(my + jj);
      nb.v[a][s][2] = mc_read<T, U>(mz + jj);
    }
}

template <typename T>
__device__ __forceinline__ bool mc_trial(const Geom& g, const McCoef<T>& c, T* __restrict__ m,
                                         const T* __restrict__ h, uint32_t stage, uint32_t sweep, int x, int y,
                                         int z) {
  const long long n = g.n;
  T* mx = m;
  T* my = m + n;
  T* mz = m + 2 * n;
  const long long i = x + (long long)g.nx * (y + (long long)g.ny * z);
  const T ox = mx[i], oy = my[i], oz = mz[i];
  Nbrs<T> nb;
  mc_nbrs<T, T>(g, m, i, x, y, z, nb);
  T hx = 0, hy = 0, hz = 0;
  if (c.cd != (T)0) {
    hx = h[i];
    hy = h[n + i];
    hz = h[2 * n + i];
  }
  const Proposal<T> p = mc_propose<T>(c, (uint32_t)i, stage, sweep);
  if (mc_accept<T>(c, nb, ox, oy, oz, hx, hy, hz, p)) {
    T px, py, pz;
    p.get(px, py, pz);
    mx[i] = px;
    my[i] = py;
    mz[i] = pz;
    return true;
  }
  return false;
}

__device__ __forceinline__ void count_accepts(bool acc, unsigned long long* counter) {
  const unsigned mask = __ballot_sync(0xffffffffu, acc);
  if ((threadIdx.x & 31) == 0 && mask) atomicAdd(counter, (unsigned long long)__popc(mask));
}

// Two-colour checkerboard: thread t -> row t / hxc, x = 2 (t mod hxc) + parity.
template <typename T>
__global__ void __launch_bounds__(256, 4) k_mc_checker(Geom g, const McCoef<T>* __restrict__ cp, T* __restrict__ m, const T* __restrict__ h,
                             const SweepCounters* __restrict__ ctr, int color, unsigned long long* acc) {
  pdl_wait();
  // replica blockIdx.z of a batch: its own coefficients, state and counter
  const McCoef<T> c = cp[blockIdx.z];
  m += blockIdx.z * 3 * g.n;
  h += blockIdx.z * 3 * g.n;
  acc += blockIdx.z;
  const int hxc = (g.nx + 1) >> 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nrows = (long long)g.ny * g.nz;
  bool accepted = false;
  if (t < nrows * hxc) {
    const int row = g.dhxc.div((int)t);
    const int j = (int)t - row * hxc;
    const int z = g.dny.div(row), y = row - z * g.ny;
    const int x = 2 * j + ((color + y + z) & 1);
    if (x < g.nx) accepted = mc_trial<T>(g, c, m, h, ctr->stage, ctr->sweep, x, y, z);
  }
  count_accepts(accepted, acc);
}

// General colouring (odd periodic axes): every thread tests its cell's colour.
template <typename T>
__global__ void __launch_bounds__(256, 4) k_mc_general(Geom g, const McCoef<T>* __restrict__ cp, T* __restrict__ m, const T* __restrict__ h,
                             const SweepCounters* __restrict__ ctr, int color, unsigned long long* acc) {
  const McCoef<T> c = cp[blockIdx.z];
  m += blockIdx.z * 3 * g.n;
  h += blockIdx.z * 3 * g.n;
  acc += blockIdx.z;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  bool accepted = false;
  if (i < g.n) {
    const int x = (int)(i % g.nx), y = (int)((i / g.nx) % g.ny), z = (int)(i / ((long long)g.nx * g.ny));
    if (cell_color(g, x, y, z) == color) accepted = mc_trial<T>(g, c, m, h, ctr->stage, ctr->sweep, x, y, z);
  }
  count_accepts(accepted, acc);
}

// One colour of an FP64 sweep (any lattice).  A thread judges MCL_TPT trials by
// the FP32 filter (mc_filter); the accepted and the unsure ones go to a list
// in shared memory, and the CTA then takes the list with full warps: the
// direction (60 FP64 operations) is made for those trials only, and the FP64
// formula decides the unsure ones.  Cells of one colour do not see each other,
// so the stores may come after all of the CTA's decisions.  Bound by FP64
// issue (1.7 operations per SM and cycle): per trial 60 x the acceptance rate
// instead of the 230 that every lane of a warp paid.
constexpr int MCL_THREADS = 128;
template <int TPT>
__global__ void __launch_bounds__(MCL_THREADS) k_mc_list(Geom g, const McCoef<double>* __restrict__ cp,
                                                         double* __restrict__ m, const double* __restrict__ h,
                                                         const SweepCounters* __restrict__ ctr, int color,
                                                         unsigned long long* acc) {
  __shared__ uint4 list[MCL_THREADS * TPT];  // cell (top bit: unsure), random words
  __shared__ double part[3][MCL_THREADS * TPT];
  __shared__ int count;
  if (threadIdx.x == 0) count = 0;
  pdl_wait();
  const McCoef<double>& c = cp[blockIdx.z];
  const long long n = g.n;
  m += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  const uint32_t stage = ctr->stage, sweep = ctr->sweep;
  const bool dm = c.cd != 0.0;
  const bool two = g.ncolors == 2;
  const int hxc = (g.nx + 1) >> 1;
  const int total = two ? g.ny * g.nz * hxc : (int)n;  // fits: n < 2^31
  __syncthreads();
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
    const long long tl = ((long long)blockIdx.x * TPT + u) * MCL_THREADS + threadIdx.x;
    McVerdict w = MC_REJECT;
    Proposal<double> p{};
    int cell = 0;
    if (tl < total) {
      const int t = (int)tl;
      int x, y, z, row;
      bool mine;
      if (two) {
        row = g.dhxc.div(t);
        z = g.dny.div(row);
        y = row - z * g.ny;
        x = 2 * (t - row * hxc) + ((color + y + z) & 1);
        mine = x < g.nx;
      } else {
        row = g.dnx.div(t);
        x = t - row * g.nx;
        z = g.dny.div(row);
        y = row - z * g.ny;
        mine = cell_color(g, x, y, z) == color;
      }
      if (mine) {
        cell = x + g.nx * row;
        Nbrs<float> nb;
        mc_nbrs<double, float>(g, m, cell, x, y, z, nb);
        float hx = 0, hy = 0, hz = 0;
        if (dm) {
          hx = f32_trunc(h[cell]);
          hy = f32_trunc(h[n + cell]);
          hz = f32_trunc(h[2 * n + cell]);
        }
        p = mc_propose<double>(c, (uint32_t)cell, stage, sweep);
        w = mc_filter(c.f, nb.v, nb.has, f32_trunc(m[cell]), f32_trunc(m[n + cell]), f32_trunc(m[2 * n + cell]), hx,
                      hy, hz, p.rx, p.ry, p.rz, g.nz == 1);
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, w != MC_REJECT);
    if (mask) {
      const int lane = threadIdx.x & 31;
      int base = 0;
      if (lane == 0) base = atomicAdd(&count, __popc(mask));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (w != MC_REJECT)
        list[base + __popc(mask & ((1u << lane) - 1u))] =
            make_uint4((uint32_t)cell | (w == MC_UNSURE ? 0x80000000u : 0u), p.rx, p.ry, p.rz);
    }
  }
  __syncthreads();
  const int cnt = count;
  // the listed trials' directions, in three pieces of about 25 FP64 operations
  // on warps of their own: a warp's FP64 instructions issue one per 64 cycles
  const int lane = threadIdx.x & 31, groups = (cnt + 31) >> 5;
  for (int task = threadIdx.x >> 5; task < 3 * groups; task += MCL_THREADS / 32) {
    const int piece = task / groups, i = (task - piece * groups) * 32 + lane;
    if (i >= cnt) continue;
    const uint4 e = list[i];
    double v;
    if (piece == 2) {
      v = Prop<double>::radius(Prop<double>::height(e.y));
    } else {
      double y, w;
      mmcm::pi_angle(Prop<double>::quarter(e.z), &y, &w);
      v = piece == 0 ? mmcm::sin_taylor(y, w) : mmcm::cos_taylor(w);
    }
    part[piece][i] = v;
  }
  __syncthreads();
  for (int i0 = 0; i0 < cnt; i0 += MCL_THREADS) {
    const int i = i0 + threadIdx.x;
    bool ok = i < cnt;
    if (ok) {
      const uint4 e = list[i];
      const int cell = (int)(e.x & 0x7fffffffu);
      double sn, cs;
      mmcm::sincos_quadrant(Prop<double>::quadrant(e.z), part[0][i], part[1][i], &sn, &cs);
      const double s = part[2][i];
      const double px = s * cs, py = s * sn, pz = Prop<double>::height(e.y);
      if (e.x >> 31) {
        const int row = g.dnx.div(cell), x = cell - row * g.nx;
        const int z = g.dny.div(row), y = row - z * g.ny;
        Nbrs<double> nb;
        mc_nbrs<double, double>(g, m, cell, x, y, z, nb);
        ok = mc_accept_formula<double>(c, nb, m[cell], m[n + cell], m[2 * n + cell], dm ? h[cell] : 0.0,
                                       dm ? h[n + cell] : 0.0, dm ? h[2 * n + cell] : 0.0, px, py, pz,
                                       mmcm::u01_f64(e.w));
      }
      if (ok) {
        m[cell] = px;
        m[n + cell] = py;
        m[2 * n + cell] = pz;
      }
    }
    count_accepts(ok, acc + blockIdx.z);
  }
}

// One colour of a two-colour film sweep (nz = 1, nx a multiple of 4) with
// 16-byte loads: a thread owns a segment of 4 consecutive cells of one row
// and makes the decisions of its 2 cells of this colour.  The row segment, the
// same segment of the rows above and below, and one cell on each side are
// loaded as whole vectors; the segment is stored back whole (its cells of the
// other colour are written with the values just read, which no thread of this
// launch changes).  Decisions are those of k_mc_checker (same mc_accept, same
// inputs).
template <typename T>
struct Vec4 {
  T v[4];
};
template <typename T>
__device__ __forceinline__ Vec4<T> ld4(const T* p) {
  Vec4<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    r.v[0] = a.x, r.v[1] = a.y, r.v[2] = a.z, r.v[3] = a.w;
  } else {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    r.v[0] = a.x, r.v[1] = a.y, r.v[2] = b.x, r.v[3] = b.y;
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void st4(T* p, const Vec4<T>& r) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
  } else {
    reinterpret_cast<double2*>(p)[0] = make_double2(r.v[0], r.v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(r.v[2], r.v[3]);
  }
}

// The components whose second exchange product a vectorised form rounds
// separately (mc_accept_formula; bit 0 = x) for cell q of a thread's two, at x
// offset p0 + 2 q of its u-th segment.  This is how each form has rounded from
// the beginning, and it keeps a seed's run the same; about two trials in 1e10 are
// decided by it, so a long run in one of these forms leaves the scalar forms'
// path there.  u < 0: the scalar forms' chain (k_mc_band); k_mc_pipe takes u = 1;
// k_mc_quad and k_mc_split the number of the thread's segment.
// The segments of a thread are a grid's threads apart, so these two fix u for every
// cell; k_mc_quad and k_mc_split, which take runs of one seed in turn (by the
// run's length), must share them.
constexpr int MCQ_THREADS = 128, MCQ_UNITS = 2;
template <bool ALLB, bool Z3>
__device__ __forceinline__ int mc_sep(int q, int u, int p0) {
  if (q || u < 0) return 0;
  if (ALLB) return !Z3 || u == 1 ? 7 : p0;
  return u == 1 || p0 == 0 ? 7 : Z3 ? 0 : 4;
}

// The decisions of the two cells at offsets P0 and P0 + 2 of a segment.
// ALLB: every x and y bond exists (both axes periodic, ny > 1), so the
// availability flags are compile-time true.  Z3: a 3-D lattice, with the
// segments of the layers below (zd) and above (zu) and their flags; films
// pass anything there.
template <typename T, int P0, bool ALLB, bool Z3 = false>
__device__ __forceinline__ bool quad_cells(const McCoef<T>& c, Vec4<T> (&own)[3], const Vec4<T> (&up)[3],
                                           const Vec4<T> (&dn)[3], const T (&lft)[3], const T (&rgt)[3],
                                           const Vec4<T> (&hh)[3], bool hl, bool hr, bool hd, bool hu,
                                           uint32_t cell0, uint32_t stage, uint32_t sweep, unsigned int& mine, int u,
                                           const Vec4<T> (&zd)[3], const Vec4<T> (&zu)[3], bool hzd, bool hzu) {
  if constexpr (ALLB) hl = hr = hd = hu = true;
  if constexpr (!Z3) hzd = hzu = false;
  bool changed = false;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int o = P0 + 2 * q;  // compile-time after unrolling
    Nbrs<T> nb;
    const bool lin = o > 0, rin = o < 3;
    nb.has[0][0] = lin || hl;
    nb.has[0][1] = rin || hr;
    nb.has[1][0] = hd;
    nb.has[1][1] = hu;
    nb.has[2][0] = hzd;
    nb.has[2][1] = hzu;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const T ov = own[k].v[o];
      nb.v[0][0][k] = lin ? own[k].v[(o + 3) & 3] : (hl ? lft[k] : ov);
      nb.v[0][1][k] = rin ? own[k].v[(o + 1) & 3] : (hr ? rgt[k] : ov);
      nb.v[1][0][k] = hd ? dn[k].v[o] : ov;
      nb.v[1][1][k] = hu ? up[k].v[o] : ov;
      nb.v[2][0][k] = hzd ? zd[k].v[o] : ov;
      nb.v[2][1][k] = hzu ? zu[k].v[o] : ov;
    }
    const Proposal<T> pr = mc_propose<T>(c, cell0 + (uint32_t)o, stage, sweep);
    if (mc_accept<T>(c, nb, own[0].v[o], own[1].v[o], own[2].v[o], hh[0].v[o], hh[1].v[o], hh[2].v[o], pr,
                     mc_sep<ALLB, Z3>(q, u, P0))) {
      pr.get(own[0].v[o], own[1].v[o], own[2].v[o]);
      changed = true;
      ++mine;
    }
  }
  return changed;
}

__host__ __device__ inline bool mc_quad_ok(const Geom& g) { return g.ncolors == 2 && g.nx % 4 == 0; }
// every x and y bond of a film exists
__host__ __device__ inline bool mc_all_bonds(const Geom& g) { return g.per[0] && g.per[1] && g.nx > 1 && g.ny > 1; }
// the staged form (k_mc_band) for the same lattices, up to 1024 cells per row
// (a band of one row then fits in 96 KB of shared memory in FP64)
constexpr size_t MC_BAND_SMEM_MAX = 96 * 1024;
__host__ __device__ inline bool mc_band_ok(const Geom& g) { return g.nz == 1 && mc_quad_ok(g) && g.nx <= 1024; }

// Z3: 3-D lattices (nz > 1), with the segments of the layers below and above.
template <typename T, bool ALLB, bool Z3>
__global__ void __launch_bounds__(256) k_mc_quad(Geom g, const McCoef<T>* __restrict__ cp, T* __restrict__ m,
                                                 const T* __restrict__ h, const SweepCounters* __restrict__ ctr,
                                                 int color, unsigned long long* acc) {
  pdl_wait();
  const McCoef<T> c = cp[blockIdx.z];
  const long long n = g.n;
  m += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  acc += blockIdx.z;
  const int nseg = g.nx >> 2;
  // two segments per thread, a grid-stride apart: the coefficients and the
  // set-up are shared by both, and the second segment's loads overlap the
  // first one's work (measured 4 us faster per batched sweep than one segment)
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int tstride = gridDim.x * blockDim.x;
  unsigned int mine = 0;
#pragma unroll
  for (int u = 0; u < MCQ_UNITS; ++u) {
    const int t = t0 + u * tstride;
    if (t < nseg * g.ny * g.nz) {
      // t / (nx / 4) == (4 t) / nx: the multiply-shift divider by nx, no run-time division
      const int row = g.dnx.div(4 * t), s = t - row * nseg;
      int z = 0, y = row;
      if constexpr (Z3) {
        z = g.dny.div(row);
        y = row - z * g.ny;
      }
      const int x0 = 4 * s;
      const long long rowb = (long long)row * g.nx;
      const long long plane = (long long)g.nx * g.ny;
      // neighbour rows: wrapped on a periodic axis, missing at an open edge or
      // when the axis has length 1
      int yu = y + 1, yd = y - 1;
      bool hu = true, hd = true;
      if (yu >= g.ny) { if (g.per[1]) yu -= g.ny; else hu = false; }
      if (yd < 0) { if (g.per[1]) yd += g.ny; else hd = false; }
      if (g.ny == 1) hu = hd = false;
      int zu = z + 1, zd = z - 1;
      bool hzu = Z3, hzd = Z3;
      if constexpr (Z3) {
        if (zu >= g.nz) { if (g.per[2]) zu -= g.nz; else hzu = false; }
        if (zd < 0) { if (g.per[2]) zd += g.nz; else hzd = false; }
      }
      // side cells
      int xl = x0 - 1, xr = x0 + 4;
      bool hl = true, hr = true;
      if (xl < 0) { if (g.per[0]) xl += g.nx; else hl = false; }
      if (xr >= g.nx) { if (g.per[0]) xr -= g.nx; else hr = false; }
      if constexpr (ALLB) hu = hd = hl = hr = true;
      // this colour's cells sit at offsets p0 and p0 + 2 (x0 is even), so only
      // one side cell is a neighbour: the left one for p0 = 0, the right one
      // for p0 = 1
      const int p0 = (color + y + z) & 1;
      const long long zbase = (long long)z * plane;
      Vec4<T> own[3], up[3], dn[3], zup[3], zdn[3];
      T lft[3], rgt[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const T* base = m + k * n;
        own[k] = ld4<T>(base + rowb + x0);
        up[k] = hu ? ld4<T>(base + zbase + (long long)yu * g.nx + x0) : own[k];
        dn[k] = hd ? ld4<T>(base + zbase + (long long)yd * g.nx + x0) : own[k];
        if constexpr (Z3) {
          zup[k] = hzu ? ld4<T>(base + (long long)zu * plane + (long long)y * g.nx + x0) : own[k];
          zdn[k] = hzd ? ld4<T>(base + (long long)zd * plane + (long long)y * g.nx + x0) : own[k];
        } else {
          zup[k] = zdn[k] = own[k];
        }
        lft[k] = (hl && p0 == 0) ? base[rowb + xl] : (T)0;
        rgt[k] = (hr && p0 == 1) ? base[rowb + xr] : (T)0;
      }
      Vec4<T> hh[3];
      const bool dm = c.cd != (T)0;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (dm) hh[k] = ld4<T>(h + k * n + rowb + x0);
        else hh[k].v[0] = hh[k].v[1] = hh[k].v[2] = hh[k].v[3] = (T)0;
      }
      // the offsets are compile-time inside quad_cells so the vectors stay in
      // registers
      bool changed;
      if (p0 == 0)
        changed = quad_cells<T, 0, ALLB, Z3>(c, own, up, dn, lft, rgt, hh, hl, hr, hd, hu, (uint32_t)(rowb + x0),
                                             ctr->stage, ctr->sweep, mine, u, zdn, zup, hzd, hzu);
      else
        changed = quad_cells<T, 1, ALLB, Z3>(c, own, up, dn, lft, rgt, hh, hl, hr, hd, hu, (uint32_t)(rowb + x0),
                                             ctr->stage, ctr->sweep, mine, u, zdn, zup, hzd, hzu);
      if (changed) {
#pragma unroll
        for (int k = 0; k < 3; ++k) st4<T>(m + k * n + rowb + x0, own[k]);
      }
    }
  }
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, (unsigned long long)v);
}

// --------------------------------------------------- colour-split Metropolis
// One colour of a two-colour FP32 sweep on rows stored colour by colour: the
// nx / 2 cells of colour 0 of row (y, z) first, then those of colour 1
// (split_pos).  The cells of a launch's colour are then contiguous, and so are
// their neighbours, all of the other colour: cell j of the row sees cell j of the
// rows above and below and cells j and j - 1 (or j + 1, by the row's parity) of
// its own row.  A thread takes two cells: it reads 15 pairs and 3 side cells
// where k_mc_quad read 12 vectors of 4 and 3 side cells for two trials, of which
// half were cells of no use to it.  Runs of at least MC_SPLIT_SWEEPS sweeps
// convert m once at either end (k_split_rows); the x passes read and write the
// split order at no cost.  Decisions: mc_propose / mc_accept on the same inputs
// as every other form but for mc_sep.  Latency and issue share the bound (58 % issue, loads the
// top stall): the coefficients stay in shared memory so that 80 registers hold 24
// warps per SM (102 registers and 16 warps with them in registers: 29 us; one
// cell per thread, 32 warps: 31 us for its index work).  128 x 64^2: 17.6 -> 13.3
// us per sweep against k_mc_quad, 64 x 256^2: 53 -> 49.
__host__ __device__ inline bool mc_split_geom_ok(const Geom& g) { return g.ncolors == 2 && g.nx % 4 == 0; }
template <typename T>
inline bool mc_split_ok(const Geom& g, const FftPlan& px) {
  return sizeof(T) == 4 && mc_split_geom_ok(g) && px.warp_a != 0;
}
constexpr int MCSP_THREADS = MCQ_THREADS;
template <bool ALLB, bool Z3>
__global__ void __launch_bounds__(MCSP_THREADS, 6) k_mc_split(Geom g, const McCoef<float>* __restrict__ cp,
                                                           float* __restrict__ m, const float* __restrict__ h,
                                                           const SweepCounters* __restrict__ ctr, int color,
                                                           int upt, FastDiv dunit, unsigned long long* acc) {
  // the coefficients stay in shared memory and are read again for each trial:
  // 26 registers less
  __shared__ McCoef<float> c;
  pdl_wait();
  if (threadIdx.x < sizeof(c) / 4)
    reinterpret_cast<uint32_t*>(&c)[threadIdx.x] = reinterpret_cast<const uint32_t*>(cp + blockIdx.z)[threadIdx.x];
  const long long n = g.n;
  m += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  acc += blockIdx.z;
  const uint32_t stage = ctr->stage, sweep = ctr->sweep;
  __syncthreads();
  const bool dm = c.cd != 0.0f;
  const int half = g.nx >> 1, upr = g.nx >> 2;  // cells of a colour, units of a row
  const int total = upr * g.ny * g.nz, tstride = gridDim.x * MCSP_THREADS;
  const int own0 = color ? half : 0, oth0 = color ? 0 : half;
  unsigned int mine = 0;
  int t = blockIdx.x * MCSP_THREADS + threadIdx.x;
  for (int u = 0; u < upt; ++u, t += tstride) {
    if (t >= total) break;
    const int row = dunit.div(t), j0 = 2 * (t - row * upr);
    int z = 0, y = row;
    if constexpr (Z3) {
      z = g.dny.div(row);
      y = row - z * g.ny;
    }
    const int p = (color + y + z) & 1;
    int yu = y + 1, yd = y - 1;
    bool hu = true, hd = true;
    if (yu >= g.ny) { if (g.per[1]) yu -= g.ny; else hu = false; }
    if (yd < 0) { if (g.per[1]) yd += g.ny; else hd = false; }
    if (g.ny == 1) hu = hd = false;
    int zu = z + 1, zd = z - 1;
    bool hzu = Z3, hzd = Z3;
    if constexpr (Z3) {
      if (zu >= g.nz) { if (g.per[2]) zu -= g.nz; else hzu = false; }
      if (zd < 0) { if (g.per[2]) zd += g.nz; else hzd = false; }
    }
    int js = p ? j0 + 2 : j0 - 1;  // the side cell
    bool hs = true;
    if (js < 0) { if (g.per[0]) js += half; else hs = false; }
    if (js >= half) { if (g.per[0]) js -= half; else hs = false; }
    if constexpr (ALLB) hu = hd = hs = true;
    const int rb = row * g.nx, ro = rb + own0 + j0, rt = rb + oth0;
    const int ru = (z * g.ny + yu) * g.nx + oth0 + j0, rd = (z * g.ny + yd) * g.nx + oth0 + j0;
    const int rzu = (zu * g.ny + y) * g.nx + oth0 + j0, rzd = (zd * g.ny + y) * g.nx + oth0 + j0;
    float2 own[3], oth[3], up[3], dn[3], zup[3], zdn[3], hh[3];
    float side[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float* base = m + k * n;
      own[k] = *reinterpret_cast<const float2*>(base + ro);
      oth[k] = *reinterpret_cast<const float2*>(base + rt + j0);
      side[k] = hs ? base[rt + js] : 0.0f;
      up[k] = hu ? *reinterpret_cast<const float2*>(base + ru) : own[k];
      dn[k] = hd ? *reinterpret_cast<const float2*>(base + rd) : own[k];
      if constexpr (Z3) {
        zup[k] = hzu ? *reinterpret_cast<const float2*>(base + rzu) : own[k];
        zdn[k] = hzd ? *reinterpret_cast<const float2*>(base + rzd) : own[k];
      } else {
        zup[k] = zdn[k] = own[k];
      }
      hh[k] = dm ? *reinterpret_cast<const float2*>(h + k * n + ro) : make_float2(0.0f, 0.0f);
    }
    bool changed = false;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      asm volatile("" ::: "memory");
      Nbrs<float> nb;
      // q = 0: (side, oth.x) or (oth.x, oth.y); q = 1: (oth.x, oth.y) or (oth.y, side)
      nb.has[0][0] = q == 0 ? (p || hs) : true;
      nb.has[0][1] = q == 1 ? (!p || hs) : true;
      if constexpr (ALLB) nb.has[0][0] = nb.has[0][1] = true;
      nb.has[1][0] = hd;
      nb.has[1][1] = hu;
      nb.has[2][0] = hzd;
      nb.has[2][1] = hzu;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nb.v[0][0][k] = q == 0 ? (p ? oth[k].x : side[k]) : (p ? oth[k].y : oth[k].x);
        nb.v[0][1][k] = q == 0 ? (p ? oth[k].y : oth[k].x) : (p ? side[k] : oth[k].y);
        nb.v[1][0][k] = q ? dn[k].y : dn[k].x;
        nb.v[1][1][k] = q ? up[k].y : up[k].x;
        nb.v[2][0][k] = q ? zdn[k].y : zdn[k].x;
        nb.v[2][1][k] = q ? zup[k].y : zup[k].x;
      }
      const Proposal<float> pr = mc_propose<float>(c, (uint32_t)(rb + 2 * (j0 + q) + p), stage, sweep);
      float& ox = q ? own[0].y : own[0].x;
      float& oy = q ? own[1].y : own[1].x;
      float& oz = q ? own[2].y : own[2].x;
      if (mc_accept<float>(c, nb, ox, oy, oz, q ? hh[0].y : hh[0].x, q ? hh[1].y : hh[1].x, q ? hh[2].y : hh[2].x,
                           pr, mc_sep<ALLB, Z3>(q, u, p))) {
        pr.get(ox, oy, oz);
        changed = true;
        ++mine;
      }
    }
    if (changed) {
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<float2*>(m + k * n + ro) = own[k];
    }
  }
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, (unsigned long long)v);
}

// Rows of `a` (nrows rows of nx values, components and replicas back to back;
// row r has y + z = yz of lattice row r mod nyz) between the natural and the
// colour-split order, in place: a CTA holds a row in shared memory in between.
static __global__ void k_split_rows(float* __restrict__ a, int nx, FastDiv dnyz, FastDiv dny, int to_split) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* line = reinterpret_cast<float*>(smem_raw);
  const int r = blockIdx.x, row = r - dnyz.div(r) * (int)dnyz.d, z = dny.div(row), yz = row - z * (int)dny.d + z;
  float* p = a + (long long)r * nx;
  for (int x = threadIdx.x; x < nx; x += blockDim.x) line[x] = p[x];
  __syncthreads();
  for (int x = threadIdx.x; x < nx; x += blockDim.x) {
    const int q = split_pos(x, yz, nx);
    if (to_split) p[q] = line[x];
    else p[x] = line[q];
  }
}

// One colour of a two-colour film sweep (the k_mc_quad film cases) with the rows
// a CTA needs staged in shared memory first: the CTA owns a band of `band`
// rows of one replica, copies m rows y0-1 .. y0+band (wrapped on a periodic
// axis) and h rows y0 .. y0+band-1 with 16-byte asynchronous copies, which
// hold no registers while they land, and then runs k_mc_quad's per-thread
// work (4-cell segments, the same quad_cells) from shared memory.  Fewer
// registers per thread than k_mc_quad, whose vector loads all sit in
// registers at once, so more warps per SM hide the copies' latency.
// Shared memory: (band + 2) x 3 rows of m and band x 3 rows of h.

template <typename T>
__host__ __device__ inline size_t mc_band_smem(const Geom& g, int band) {
  return (size_t)(2 * band + 2) * 3 * g.nx * sizeof(T);
}
// rows per CTA: about one 4-cell segment per thread
template <typename T>
inline int mc_band_rows(const Geom& g, int threads) {
  int band = std::max(1, std::min(g.ny, 4 * threads / g.nx));
  while (band > 1 && mc_band_smem<T>(g, band) > MC_BAND_SMEM_MAX) band /= 2;
  return band;
}

// The decisions of this colour on rows y0 .. y0+nb-1 of one replica from rows
// staged in shared memory -- ms[slot][comp][x] with slot s = row y0-1+s, hs
// [row][comp][x] (read when dm) -- the CTA's threads striding over the rows'
// 4-cell segments (k_mc_quad's per-thread work, the same quad_cells); the
// segments that changed are stored to m (this replica's), and accepts are
// added to mine.
template <typename T, bool ALLB>
__device__ __forceinline__ void band_segments(const Geom& g, const McCoef<T>& c, const T* ms, const T* hs,
                                              T* __restrict__ m, int y0, int nb, int color, bool dm,
                                              const FastDiv& dseg, uint32_t stage, uint32_t sweep,
                                              unsigned int& mine, int u) {
  const int nx = g.nx, ny = g.ny;
  const long long n = g.n;
  const int nseg = (int)dseg.d;
  for (int t = threadIdx.x; t < nb * nseg; t += blockDim.x) {
    const int rr = dseg.div(t), s = t - rr * nseg;
    const int y = y0 + rr;
    const int x0 = 4 * s;
    bool hu = true, hd = true;
    if (y + 1 >= ny && !g.per[1]) hu = false;
    if (y - 1 < 0 && !g.per[1]) hd = false;
    if (ny == 1) hu = hd = false;
    int xl = x0 - 1, xr = x0 + 4;
    bool hl = true, hr = true;
    if (xl < 0) { if (g.per[0]) xl += nx; else hl = false; }
    if (xr >= nx) { if (g.per[0]) xr -= nx; else hr = false; }
    if constexpr (ALLB) hu = hd = hl = hr = true;
    const int p0 = (color + y) & 1;
    const T* own_r = ms + (size_t)(rr + 1) * 3 * nx;
    const T* up_r = own_r + 3 * nx;
    const T* dn_r = own_r - 3 * nx;
    Vec4<T> own[3], up[3], dn[3], hh[3];
    T lft[3], rgt[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      own[k] = ld4<T>(own_r + k * nx + x0);
      up[k] = hu ? ld4<T>(up_r + k * nx + x0) : own[k];
      dn[k] = hd ? ld4<T>(dn_r + k * nx + x0) : own[k];
      lft[k] = (hl && p0 == 0) ? own_r[k * nx + xl] : (T)0;
      rgt[k] = (hr && p0 == 1) ? own_r[k * nx + xr] : (T)0;
      if (dm) hh[k] = ld4<T>(hs + ((size_t)rr * 3 + k) * nx + x0);
      else hh[k].v[0] = hh[k].v[1] = hh[k].v[2] = hh[k].v[3] = (T)0;
    }
    const long long rowb = (long long)y * nx;
    bool changed;
    if (p0 == 0)
      changed = quad_cells<T, 0, ALLB>(c, own, up, dn, lft, rgt, hh, hl, hr, hd, hu, (uint32_t)(rowb + x0), stage,
                                       sweep, mine, u, own, own, false, false);
    else
      changed = quad_cells<T, 1, ALLB>(c, own, up, dn, lft, rgt, hh, hl, hr, hd, hu, (uint32_t)(rowb + x0), stage,
                                       sweep, mine, u, own, own, false, false);
    if (changed) {
#pragma unroll
      for (int k = 0; k < 3; ++k) st4<T>(m + k * n + rowb + x0, own[k]);
    }
  }
}

// (Three CTAs of 256 threads per SM in FP32 -- 80 registers, a few spilled
// -- and two in FP64.)
template <typename T, bool ALLB>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 2) k_mc_band(Geom g, const McCoef<T>* __restrict__ cp, T* __restrict__ m,
                                                    const T* __restrict__ h, const SweepCounters* __restrict__ ctr,
                                                    int color, int band, FastDiv dchunk, FastDiv dseg,
                                                    unsigned long long* acc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = g.nx, ny = g.ny;
  const long long n = g.n;
  T* ms = reinterpret_cast<T*>(smem_raw);  // [slot][comp][x], slot s = row y0 - 1 + s
  T* hs = ms + (size_t)(band + 2) * 3 * nx;  // [row][comp][x]
  const McCoef<T> c = cp[blockIdx.z];
  m += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  acc += blockIdx.z;
  const int y0 = blockIdx.x * band;
  const int nb = min(band, ny - y0);
  const bool dm = c.cd != (T)0;
  const int per = (int)dchunk.d;  // 16-byte chunks per row
  constexpr int E = 16 / (int)sizeof(T);
  const int nm = (nb + 2) * 3 * per, nh = dm ? nb * 3 * per : 0;
  for (int i = threadIdx.x; i < nm + nh; i += blockDim.x) {
    const bool isM = i < nm;
    const int j = isM ? i : i - nm;
    const int row = dchunk.div(j), q = j - row * per;  // row = slot * 3 + comp (m) or r * 3 + comp (h)
    const int slot = row / 3, comp = row - slot * 3;
    if (isM) {
      int y = y0 - 1 + slot;
      if (y < 0 || y >= ny) {
        if (!g.per[1] || ny == 1) continue;
        y = y < 0 ? y + ny : y - ny;
      }
      cp_async16(ms + (size_t)row * nx + q * E, m + comp * n + (long long)y * nx + q * E);
    } else {
      cp_async16(hs + (size_t)row * nx + q * E, h + comp * n + (long long)(y0 + slot) * nx + q * E);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  unsigned int mine = 0;
  band_segments<T, ALLB>(g, c, ms, hs, m, y0, nb, color, dm, dseg, ctr->stage, ctr->sweep, mine, -1);
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, (unsigned long long)v);
}

// ---------------------------------------------- pipelined staged Metropolis
// One colour of a two-colour film sweep (the k_mc_band lattices) by
// persistent CTAs.  Work items are (replica, band of rows); CTA b takes the
// items [b chunk, (b + 1) chunk), consecutive bands of one replica, so its
// coefficients change rarely.  A band's rows -- m rows y0-1 .. y0+nb (wrapped
// on a periodic axis) and h rows y0 .. y0+nb-1, whole rows of one component
// each -- are fetched by bulk asynchronous copies (cp.async.bulk, the TMA
// engine) into one of nst (2-4) shared-memory buffers, their completion
// counted by that buffer's mbarrier (transaction bytes).  Warp 0 issues the
// copies of item i + nst as soon as item i's buffer is free (after the CTA
// barrier that ends item i), so the loads of later bands land while the CTA
// decides the current ones: no registers or issue slots spent on copying, and
// none of the load latency on the decisions' critical path.  Every warp waits
// on its buffer's mbarrier itself, so no warp waits for the producer's
// issuing; the producer reads the next item's replica flag (demag on or off)
// before the decisions, so its latency is hidden too.  The decisions are
// band_segments', i.e. k_mc_band's and k_mc_quad's (same quad_cells on the
// same inputs).  Measured at 32 x 256^2 in FP32: 49 us per batched sweep
// against k_mc_quad's 30.7 -- 128 registers hold 2 CTAs (16 warps) per SM at
// 36-39 % issue, against k_mc_quad's 24 warps at 54 %, the top stall being
// the barrier that ends each item (ncu); taking the loads off the decisions'
// path does not pay where the decisions themselves are latency- and
// issue-bound and k_mc_quad's warps already hide its L2 loads.  Two segments
// per thread unrolled together: 51 us.  It is an autotuner candidate.
//
// Every wait on a buffer is bounded (MCP_WAIT_NS of the global timer): a warp
// whose wait runs out sets the CTA's abort flag and *err; after the item's
// barrier the CTA skips the remaining items, thread 0 waits (bounded again)
// for the copies still in flight, and the CTA returns; the host reads *err
// after the run.
constexpr int MCP_THREADS = 256;
constexpr int MCP_MIN_STAGES = 2;
constexpr int MCP_MAX_STAGES = 3;
constexpr int MCP_HDR = 128;  // bytes ahead of the stage buffers: the mbarriers, the abort flag
constexpr unsigned long long MCP_WAIT_NS = 2000000000ull;
__host__ __device__ inline bool mc_pipe_ok(const Geom& g) { return mc_band_ok(g); }
// rows per band: one 4-cell segment per thread (two, unrolled together so
// that their decisions interleave, measured no faster and spilled)
inline int mc_pipe_rows(const Geom& g) { return std::max(1, std::min(g.ny, 4 * MCP_THREADS / g.nx)); }
// elements of one stage buffer: m rows y0-1 .. y0+band, h rows y0 .. y0+band-1
__host__ __device__ inline size_t mc_pipe_stage_elems(const Geom& g, int band) {
  return (size_t)(2 * band + 2) * 3 * g.nx;
}
template <typename T>
inline size_t mc_pipe_smem(const Geom& g, int nst = MCP_MIN_STAGES) {
  return MCP_HDR + nst * mc_pipe_stage_elems(g, mc_pipe_rows(g)) * sizeof(T);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ unsigned long long mcp_now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits until the phase with the given parity has completed, at most limit_ns.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, unsigned parity, unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = mcp_now_ns();
  while (!mbar_try_wait(bar, parity))
    if (mcp_now_ns() - t0 > limit_ns) return false;
  return true;
}
// Bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned) from
// global to shared memory, completing as transaction bytes on bar.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Warp 0: the copies of item i into buffer `buf` (see k_mc_pipe); dm: the
// item's replica has demag on (its h rows are needed).
template <typename T>
__device__ __forceinline__ void mc_pipe_issue(const Geom& g, const T* m, const T* h, int i, int band, int nbands,
                                              bool dm, T* buf, uint64_t* bar) {
  const int nx = g.nx, ny = g.ny;
  const long long n = g.n;
  const int r = i / nbands;
  const int y0 = (i - r * nbands) * band;
  const int nb = min(band, ny - y0);
  const bool wrap = g.per[1] && ny > 1;
  const int lo = (y0 > 0 || wrap) ? 0 : 1;             // first m slot present
  const int hi = (y0 + nb < ny || wrap) ? nb + 1 : nb;  // last m slot present
  const int nm = 3 * (hi - lo + 1), nh = dm ? 3 * nb : 0;
  const unsigned rowb = (unsigned)(nx * sizeof(T));
  const T* mr = m + (long long)r * 3 * n;
  const T* hr = h + (long long)r * 3 * n;
  T* hs = buf + (size_t)(band + 2) * 3 * nx;
  const int lane = threadIdx.x & 31;
  // the CTA's reads of this buffer (ordered before by a barrier) come before
  // the copies that overwrite it
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (lane == 0) mbar_arrive_expect_tx(bar, (unsigned)(nm + nh) * rowb);
  __syncwarp();
  for (int q = lane; q < nm + nh; q += 32) {
    if (q < nm) {
      const int slot = lo + q / 3, comp = q - (q / 3) * 3;
      int y = y0 - 1 + slot;
      if (y < 0) y += ny;
      else if (y >= ny) y -= ny;
      bulk_g2s(buf + ((size_t)slot * 3 + comp) * nx, mr + comp * n + (long long)y * nx, rowb, bar);
    } else {
      const int j = q - nm, rr = j / 3, comp = j - rr * 3;
      bulk_g2s(hs + ((size_t)rr * 3 + comp) * nx, hr + comp * n + (long long)(y0 + rr) * nx, rowb, bar);
    }
  }
}

__device__ __forceinline__ void flush_accepts(unsigned int& mine, unsigned long long* counter) {
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(counter, (unsigned long long)v);
  mine = 0;
}

// m, h, acc and cp cover every replica (items = replicas x nbands); nst
// buffers (MCP_MIN_STAGES .. MCP_MAX_STAGES).
template <typename T, bool ALLB>
__global__ void __launch_bounds__(MCP_THREADS, 2)
    k_mc_pipe(Geom g, const McCoef<T>* __restrict__ cp, T* __restrict__ m, const T* __restrict__ h,
              const SweepCounters* __restrict__ ctr, int color, int band, int nbands, int items, int chunk, int nst,
              FastDiv dseg, unsigned long long* acc, int* err) {
  // no static shared memory: the dynamic limit is raised to the device's whole
  // opt-in size
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
  volatile int& abort_s = *reinterpret_cast<int*>(smem_raw + 64);
  T* buf0 = reinterpret_cast<T*>(smem_raw + MCP_HDR);
  const size_t selems = mc_pipe_stage_elems(g, band);
  const long long n = g.n;
  const int i0 = blockIdx.x * chunk, i1 = min(items, i0 + chunk);
  if (i0 >= i1) return;
  const bool producer = threadIdx.x < 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < nst; ++s) mbar_init(&bars[s], 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();  // m and h are the previous kernels' output
  if (producer)
    for (int k = 0; k < nst && i0 + k < i1; ++k)
      mc_pipe_issue<T>(g, m, h, i0 + k, band, nbands, cp[(i0 + k) / nbands].cd != (T)0, buf0 + k * selems,
                       &bars[k]);
  const uint32_t stage = ctr->stage, sweep = ctr->sweep;
  McCoef<T> c;
  int rc = -1;
  unsigned int mine = 0;
  int failed = -1;  // the item whose wait ran out
  for (int i = i0; i < i1; ++i) {
    const int k = i - i0, s = k % nst;
    const int inext = i + nst;
    const bool dm_next = producer && inext < i1 && cp[inext / nbands].cd != (T)0;
    // warp-uniform: every lane sees the phase complete, or the warp gives up
    const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], (unsigned)(k / nst) & 1u, MCP_WAIT_NS));
    if (!ok) {
      abort_s = 1;
    } else {
      const int r = i / nbands, y0 = (i - r * nbands) * band;
      if (r != rc) {
        if (rc >= 0) flush_accepts(mine, acc + rc);
        rc = r;
        c = cp[r];
      }
      const T* ms = buf0 + s * selems;
      band_segments<T, ALLB>(g, c, ms, ms + (size_t)(band + 2) * 3 * g.nx, m + (long long)r * 3 * n, y0,
                             min(band, g.ny - y0), color, c.cd != (T)0, dseg, stage, sweep, mine, 1);
    }
    __syncthreads();  // buffer s is free; abort_s is final for this item
    if (abort_s) {
      failed = i;
      break;
    }
    if (producer && inext < i1) mc_pipe_issue<T>(g, m, h, inext, band, nbands, dm_next, buf0 + s * selems, &bars[s]);
  }
  if (rc >= 0) flush_accepts(mine, acc + rc);
  if (failed >= 0 && threadIdx.x == 0) {
    atomicExch(err, 1);
    // the copies still in flight: items failed .. failed + nst - 1
    for (int i = failed; i < min(i1, failed + nst); ++i) {
      const int k = i - i0;
      mbar_wait_bounded(&bars[k % nst], (unsigned)(k / nst) & 1u, MCP_WAIT_NS);
    }
  }
}

// Both colours of a two-colour film sweep (nz = 1) in one launch.  A CTA owns
// an MCT x MCT tile of one replica and holds, in shared memory, m on the tile
// plus a 2-cell margin and h on the tile plus a 1-cell margin.  Colour 0 runs
// on the tile and on the ring of cells next to it (without the corners): the
// ring cells belong to neighbouring tiles, and this CTA repeats, bit for bit,
// the decisions their owners make -- same inputs, same Philox counter -- so
// that colour 1 on the tile sees exactly the colour-0 state of the two-launch
// sweep.  Only tile cells are written and counted, to the other copy of m: a
// neighbour that starts later (another wave of CTAs, a cold instruction cache)
// still has to read this tile's margin as it was before the sweep.  Periodic
// axes must be whole tiles and at least two tiles long, so the margin never wraps
// onto the tile itself.
constexpr int MCT = 32;

// One 4- or 8-byte global -> shared copy through the async path (no register
// round trip, so a thread can have many in flight).
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* smem, const T* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (sizeof(T) == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(gmem) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
constexpr int MCT_B = MCT + 4;  // m box side
constexpr int MCT_H = MCT + 2;  // h box side

__host__ __device__ inline bool mc_tile_ok(const Geom& g) {
  return g.nz == 1 && g.ncolors == 2 && (!g.per[0] || (g.nx % MCT == 0 && g.nx >= 2 * MCT)) &&
         (!g.per[1] || (g.ny % MCT == 0 && g.ny >= 2 * MCT));
}
template <typename T>
__host__ __device__ inline size_t mc_tile_smem() {
  return (size_t)3 * (MCT_B * MCT_B + MCT_H * MCT_H) * sizeof(T);
}

template <typename T>
__global__ void __launch_bounds__(256) k_mc_tile(Geom g, const McCoef<T>* __restrict__ cp,
                                                 const T* __restrict__ m, T* __restrict__ mo,
                                                 const T* __restrict__ h, const SweepCounters* __restrict__ ctr,
                                                 unsigned long long* acc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);  // [comp][by][bx], MCT_B^2 per component
  T* sh = sm + 3 * MCT_B * MCT_B;           // [comp][hy][hx], MCT_H^2 per component
  __shared__ int colx[MCT_B], rowy[MCT_B];  // box column / row -> lattice x / y, -1 outside an open edge
  const McCoef<T> c = cp[blockIdx.z];
  const long long n = g.n;
  m += blockIdx.z * 3 * n;
  mo += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  acc += blockIdx.z;
  const uint32_t stage = ctr->stage, sweep = ctr->sweep;
  const int x0 = blockIdx.x * MCT, y0 = blockIdx.y * MCT;
  if (threadIdx.x < MCT_B) {
    int v = x0 - 2 + (int)threadIdx.x;
    if (v < 0 || v >= g.nx) v = g.per[0] ? (v + g.nx) % g.nx : -1;
    colx[threadIdx.x] = v;
    int w = y0 - 2 + (int)threadIdx.x;
    if (w < 0 || w >= g.ny) w = g.per[1] ? (w + g.ny) % g.ny : -1;
    rowy[threadIdx.x] = w;
  }
  __syncthreads();
  constexpr int BB = MCT_B * MCT_B, HH = MCT_H * MCT_H;
  // asynchronous element copies, all in flight at once; cells outside an open
  // edge are zero
  for (int idx = threadIdx.x; idx < 3 * BB; idx += blockDim.x) {
    const int cc = idx / BB, r = idx - cc * BB, by = r / MCT_B, bx = r - by * MCT_B;
    const int gx = colx[bx], gy = rowy[by];
    if (gx >= 0 && gy >= 0)
      cp_async_elem<T>(sm + idx, m + cc * n + (long long)gy * g.nx + gx);
    else
      sm[idx] = (T)0;
  }
  const bool with_h = c.cd != (T)0;
  for (int idx = threadIdx.x; idx < 3 * HH; idx += blockDim.x) {
    const int cc = idx / HH, r = idx - cc * HH, hy = r / MCT_H, hx = r - hy * MCT_H;
    const int gx = colx[hx + 1], gy = rowy[hy + 1];
    if (with_h && gx >= 0 && gy >= 0)
      cp_async_elem<T>(sh + idx, h + cc * n + (long long)gy * g.nx + gx);
    else
      sh[idx] = (T)0;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // one trial at box cell (bx, by); returns whether it was accepted
  auto trial = [&](int bx, int by) -> bool {
    const int gx = colx[bx], gy = rowy[by];
    if (gx < 0 || gy < 0) return false;
    Nbrs<T> nb;
    T* own = sm + by * MCT_B + bx;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int ex = bx + (s ? 1 : -1), ey = by + (s ? 1 : -1);
      const bool okx = colx[ex] >= 0, oky = rowy[ey] >= 0;
      nb.has[0][s] = okx;
      nb.has[1][s] = oky;
      nb.has[2][s] = false;
      const T* px = okx ? sm + by * MCT_B + ex : own;
      const T* py = oky ? sm + ey * MCT_B + bx : own;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        nb.v[0][s][k] = px[k * BB];
        nb.v[1][s][k] = py[k * BB];
        nb.v[2][s][k] = own[k * BB];
      }
    }
    const T* hp = sh + (by - 1) * MCT_H + (bx - 1);
    const Proposal<T> p = mc_propose<T>(c, (uint32_t)(gx + g.nx * gy), stage, sweep);
    if (mc_accept<T>(c, nb, own[0], own[BB], own[2 * BB], hp[0], hp[HH], hp[2 * HH], p)) {
      p.get(own[0], own[BB], own[2 * BB]);
      return true;
    }
    return false;
  };
  // the colour of box cell (bx, by) is (bx + by) & 1: x0 - 2 and y0 - 2 are even
  // and periodic axes have even length
  unsigned int mine = 0;
  // colour 0 on box rows 1 .. MCT + 2 (tile rows -1 .. MCT), box columns
  // 1 .. MCT + 2, without the four corners
  constexpr int HALF0 = (MCT + 2) / 2;
  for (int idx = threadIdx.x; idx < (MCT + 2) * HALF0; idx += blockDim.x) {
    const int by = 1 + idx / HALF0, k = idx - (by - 1) * HALF0;
    const int bx = 1 + 2 * k + ((by + 1) & 1);
    const bool edge_row = by == 1 || by == MCT + 2;
    if (edge_row && (bx == 1 || bx == MCT + 2)) continue;
    const bool acc_ok = trial(bx, by);
    if (acc_ok && by >= 2 && by < MCT + 2 && bx >= 2 && bx < MCT + 2) ++mine;
  }
  __syncthreads();
  // colour 1 on the tile
  constexpr int HALF1 = MCT / 2;
  for (int idx = threadIdx.x; idx < MCT * HALF1; idx += blockDim.x) {
    const int by = 2 + idx / HALF1, k = idx - (by - 2) * HALF1;
    const int bx = 2 + 2 * k + ((by + 1) & 1);
    if (trial(bx, by)) ++mine;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 3 * MCT * MCT; idx += blockDim.x) {
    const int cc = idx / (MCT * MCT), r = idx - cc * MCT * MCT, ty = r / MCT, tx = r - ty * MCT;
    const int gx = colx[tx + 2], gy = rowy[ty + 2];
    if (gx >= 0 && gy >= 0 && x0 + tx < g.nx && y0 + ty < g.ny)
      mo[cc * n + (long long)gy * g.nx + gx] = sm[cc * BB + (ty + 2) * MCT_B + tx + 2];
  }
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, (unsigned long long)v);
}

// Both colours of a two-colour film sweep (nz = 1, nx a multiple of 4) in one
// launch, by strips of rows.  A CTA owns `rows` consecutive rows of one
// replica (the last strip may be shorter) and stages the m rows y0 - 2 ..
// y0 + rows + 1 in shared memory (slot s holds row y0 - 2 + s, wrapped on a
// periodic y axis, absent beyond an open edge).  Colour 0 runs on its own
// rows and on the two rows next to them (y0 - 1 and y0 + rows): the owners of
// those rows make the same decisions from the same inputs, since the
// neighbours of a colour-0 cell are colour-1 cells, unchanged until colour 1.
// Colour 1 then runs on the own rows, reading the colour-0 values just
// decided.  A thread owns pairs of cells (2k, 2k + 1) of a row, one of each
// colour, and reads the pair's h once for both decisions.  The strip reads m
// from `m_in` and writes its own rows to `m_out`, a different buffer: other
// strips still read the rows it changes.  Each trial is mc_propose /
// mc_accept on the same inputs as in the per-colour forms, so the decisions
// are theirs bit for bit.  m is read once and written once per sweep, h is
// read once, and one launch replaces two.
constexpr int MCS_THREADS = 256;
constexpr int MCS_IPT = 4;  // own-row pairs per thread
__host__ __device__ inline bool mc_strip_ok(const Geom& g) {
  return g.nz == 1 && g.ncolors == 2 && g.nx % 4 == 0 && g.nx >= 4 && g.nx <= 2048;
}
// rows per strip: the own-row pairs of a strip fill the CTA's MCS_IPT pairs
// per thread, at most 32 rows
__host__ __device__ inline int mc_strip_rows(const Geom& g) {
  const int r = MCS_IPT * MCS_THREADS / (g.nx / 2);
  return r < 1 ? 1 : r > 32 ? 32 : (r > g.ny ? g.ny : r);
}
template <typename T>
__host__ __device__ inline size_t mc_strip_smem(const Geom& g) {
  return (size_t)(mc_strip_rows(g) + 4) * 3 * g.nx * sizeof(T);
}

// Lattice row of slot s of the strip starting at y0, or -1 (absent).
__device__ __forceinline__ int strip_slot_row(const Geom& g, int y0, int s) {
  int y = y0 - 2 + s;
  if (y < 0 || y >= g.ny) {
    if (!g.per[1]) return -1;
    y %= g.ny;
    if (y < 0) y += g.ny;
  }
  return y;
}

// One trial at x of slot s (lattice row y) with the given h; neighbours from
// the staged rows.  ALLB: every x and y bond exists.
template <typename T, bool ALLB>
__device__ __forceinline__ bool strip_trial(const Geom& g, const McCoef<T>& c, T* __restrict__ sm, int s, int y,
                                            int x, bool hdn, bool hup, T hx, T hy, T hz, uint32_t stage,
                                            uint32_t sweep) {
  const int nx = g.nx, rs = 3 * nx;
  T* own = sm + s * rs + x;
  int xl = x - 1, xr = x + 1;
  bool hl = true, hr = true;
  if (xl < 0) {
    if (g.per[0]) xl += nx;
    else hl = false;
  }
  if (xr >= nx) {
    if (g.per[0]) xr -= nx;
    else hr = false;
  }
  if constexpr (ALLB) hl = hr = hdn = hup = true;
  Nbrs<T> nb;
  nb.has[0][0] = hl;
  nb.has[0][1] = hr;
  nb.has[1][0] = hdn;
  nb.has[1][1] = hup;
  nb.has[2][0] = nb.has[2][1] = false;
  const T* row = sm + s * rs;
  T ov[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ov[k] = own[k * nx];
    nb.v[0][0][k] = hl ? row[k * nx + xl] : ov[k];
    nb.v[0][1][k] = hr ? row[k * nx + xr] : ov[k];
    nb.v[1][0][k] = hdn ? own[k * nx - rs] : ov[k];
    nb.v[1][1][k] = hup ? own[k * nx + rs] : ov[k];
    nb.v[2][0][k] = nb.v[2][1][k] = ov[k];
  }
  const Proposal<T> p = mc_propose<T>(c, (uint32_t)(y * nx + x), stage, sweep);
  if (mc_accept<T>(c, nb, ov[0], ov[1], ov[2], hx, hy, hz, p)) {
    p.get(own[0], own[nx], own[2 * nx]);
    return true;
  }
  return false;
}

template <typename T>
struct Pair2 {
  T a, b;
};
template <typename T>
__device__ __forceinline__ Pair2<T> ld2(const T* p) {
  if constexpr (sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return {v.x, v.y};
  } else {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return {v.x, v.y};
  }
}

template <typename T, bool ALLB>
__global__ void __launch_bounds__(MCS_THREADS) k_mc_strip(Geom g, const McCoef<T>* __restrict__ cp,
                                                          const T* __restrict__ m_in, T* __restrict__ m_out,
                                                          const T* __restrict__ h,
                                                          const SweepCounters* __restrict__ ctr, int rows,
                                                          FastDiv dq, FastDiv dp, unsigned long long* acc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);  // [slot][comp][x]
  pdl_wait();  // coefficients (tempering swaps), counters, m and h come from earlier kernels
  const McCoef<T> c = cp[blockIdx.z];
  const long long n = g.n;
  const int nx = g.nx, P = nx >> 1, Q = nx >> 2, rs = 3 * nx;
  const int y0 = blockIdx.x * rows;
  const int nown = min(rows, g.ny - y0);
  const int nslots = nown + 4;
  m_in += blockIdx.z * 3 * n;
  m_out += blockIdx.z * 3 * n;
  h += blockIdx.z * 3 * n;
  acc += blockIdx.z;
  const bool dm = c.cd != (T)0;
  const bool ybonds = g.ny > 1;
  const uint32_t stage = ctr->stage, sweep = ctr->sweep;
  // stage the slots (16-byte loads and stores, x fastest)
  for (int idx = threadIdx.x; idx < nslots * 3 * Q; idx += blockDim.x) {
    const int sk = dq.div(idx), q = idx - sk * Q;
    const int sl = sk / 3, k = sk - 3 * sl;
    const int y = strip_slot_row(g, y0, sl);
    if (y >= 0) st4<T>(sm + sl * rs + k * nx + 4 * q, ld4<T>(m_in + k * n + (long long)y * nx + 4 * q));
  }
  __syncthreads();
  // colour 0 on the own rows (slots 2 .. nown + 1), keeping the colour-1
  // cells' h for the second phase
  T h1[MCS_IPT][3];
  unsigned int mine = 0;
#pragma unroll
  for (int i = 0; i < MCS_IPT; ++i) {
    const int item = threadIdx.x + i * MCS_THREADS;
    if (item < nown * P) {
      const int r = dp.div(item), k = item - r * P;
      const int sl = 2 + r, y = y0 + r;
      const int p0 = y & 1;
      T hc[3] = {(T)0, (T)0, (T)0};
      if (dm) {
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          const Pair2<T> hv = ld2<T>(h + cc * n + (long long)y * nx + 2 * k);
          hc[cc] = p0 ? hv.b : hv.a;
          h1[i][cc] = p0 ? hv.a : hv.b;
        }
      } else {
        h1[i][0] = h1[i][1] = h1[i][2] = (T)0;
      }
      const bool hdn = ybonds && (ALLB || strip_slot_row(g, y0, sl - 1) >= 0);
      const bool hup = ybonds && (ALLB || strip_slot_row(g, y0, sl + 1) >= 0);
      if (strip_trial<T, ALLB>(g, c, sm, sl, y, 2 * k + p0, hdn, hup, hc[0], hc[1], hc[2], stage, sweep)) ++mine;
    }
  }
  // colour 0 on the rows next to the strip (slots 1 and nown + 2): the
  // neighbouring strips' decisions, recomputed, not counted
  for (int item = threadIdx.x; item < 2 * P; item += blockDim.x) {
    const int side = item >= P, k = item - side * P;
    const int sl = side ? nown + 2 : 1;
    const int y = strip_slot_row(g, y0, sl);
    if (y < 0) continue;
    const int x = 2 * k + (y & 1);
    T hc[3] = {(T)0, (T)0, (T)0};
    if (dm) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) hc[cc] = h[cc * n + (long long)y * nx + x];
    }
    const bool hdn = ybonds && (ALLB || strip_slot_row(g, y0, sl - 1) >= 0);
    const bool hup = ybonds && (ALLB || strip_slot_row(g, y0, sl + 1) >= 0);
    strip_trial<T, ALLB>(g, c, sm, sl, y, x, hdn, hup, hc[0], hc[1], hc[2], stage, sweep);
  }
  __syncthreads();
  // colour 1 on the own rows
#pragma unroll
  for (int i = 0; i < MCS_IPT; ++i) {
    const int item = threadIdx.x + i * MCS_THREADS;
    if (item < nown * P) {
      const int r = dp.div(item), k = item - r * P;
      const int sl = 2 + r, y = y0 + r;
      const int p1 = (y & 1) ^ 1;
      const bool hdn = ybonds && (ALLB || strip_slot_row(g, y0, sl - 1) >= 0);
      const bool hup = ybonds && (ALLB || strip_slot_row(g, y0, sl + 1) >= 0);
      if (strip_trial<T, ALLB>(g, c, sm, sl, y, 2 * k + p1, hdn, hup, h1[i][0], h1[i][1], h1[i][2], stage, sweep))
        ++mine;
    }
  }
  __syncthreads();
  // own rows back, whole
  for (int idx = threadIdx.x; idx < nown * 3 * Q; idx += blockDim.x) {
    const int sk = dq.div(idx), q = idx - sk * Q;
    const int r = sk / 3, k = sk - 3 * r;
    st4<T>(m_out + k * n + (long long)(y0 + r) * nx + 4 * q, ld4<T>(sm + (r + 2) * rs + k * nx + 4 * q));
  }
  unsigned int v = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(acc, (unsigned long long)v);
}

// =========================================================== energy
// Per-cell energies in FP64 whatever T is (calEnergyKernel,
// src/effective_H.h:35-43, + thrust::reduce, src/main.cu:945-948), reduced
// per block in a fixed order; a second single-block kernel sums the blocks.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Per-cell terms of the energy reduction: q[0..4] the five energies with the
// prefactors of e, q[5..7] m, q[8] (with_q) the solid angle of the two
// triangles of the plaquette at (x, y).
template <typename T>
__device__ __forceinline__ void energy_terms_at(const Geom& g, const EnCoef& e, const T* __restrict__ m,
                                                const T* __restrict__ h, long long i, bool with_q, double q[NQ]) {
  const long long n = g.n;
  const T* mx = m;
  const T* my = m + n;
  const T* mz = m + 2 * n;
  // cell coordinates by the multiply-shift dividers (n < 2^31)
  const int row = g.dnx.div((int)i), x = (int)i - row * g.nx;
  const int z = g.dny.div(row), y = row - z * g.ny;
  const double ax = mx[i], ay = my[i], az = mz[i];
  for (int a = 0; a < 3; ++a) {
    const long long j = nbr_idx(g, x, y, z, a, 1);
    if (j < 0) continue;
    const double ddx = (double)mx[j] - ax, ddy = (double)my[j] - ay, ddz = (double)mz[j] - az;
    q[0] += e.aexV_d2[a] * (ddx * ddx + ddy * ddy + ddz * ddz);
  }
  const long long xp = nbr_idx(g, x, y, z, 0, 1), xm = nbr_idx(g, x, y, z, 0, -1);
  const long long yp = nbr_idx(g, x, y, z, 1, 1), ym = nbr_idx(g, x, y, z, 1, -1);
  const double dxmz = (xp >= 0 ? (double)mz[xp] : 0.0) - (xm >= 0 ? (double)mz[xm] : 0.0);
  const double dxmx = (xp >= 0 ? (double)mx[xp] : 0.0) - (xm >= 0 ? (double)mx[xm] : 0.0);
  const double dymz = (yp >= 0 ? (double)mz[yp] : 0.0) - (ym >= 0 ? (double)mz[ym] : 0.0);
  const double dymy = (yp >= 0 ? (double)my[yp] : 0.0) - (ym >= 0 ? (double)my[ym] : 0.0);
  q[1] = -(ax * e.dV_2d[0] * dxmz + ay * e.dV_2d[1] * dymz - az * (e.dV_2d[0] * dxmx + e.dV_2d[1] * dymy));
  const double mu = ax * e.u[0] + ay * e.u[1] + az * e.u[2];
  q[2] = -e.kuV * mu * mu;
  q[3] = -(ax * e.msVB[0] + ay * e.msVB[1] + az * e.msVB[2]);
  if (e.demag != 0.0 && h) q[4] = -e.demag * (ax * (double)h[i] + ay * (double)h[n + i] + az * (double)h[2 * n + i]);
  q[5] = ax;
  q[6] = ay;
  q[7] = az;
  if (!with_q) return;
  const long long i2 = nbr_idx(g, x, y, z, 0, 1);
  const long long i4 = nbr_idx(g, x, y, z, 1, 1);
  if (i2 >= 0 && i4 >= 0) {
    const int x2 = (int)i2 - g.dnx.div((int)i2) * g.nx;
    const long long i3 = nbr_idx(g, x2, y, z, 1, 1);
    const long long tri[2][3] = {{i, i2, i3}, {i, i3, i4}};
    for (int t = 0; t < 2; ++t) {
      const long long a = tri[t][0], b = tri[t][1], cc = tri[t][2];
      const double pax = mx[a], pay = my[a], paz = mz[a];
      const double pbx = mx[b], pby = my[b], pbz = mz[b];
      const double pcx = mx[cc], pcy = my[cc], pcz = mz[cc];
      const double trip =
          pax * (pby * pcz - pbz * pcy) + pay * (pbz * pcx - pbx * pcz) + paz * (pbx * pcy - pby * pcx);
      const double den = 1.0 + (pax * pbx + pay * pby + paz * pbz) + (pbx * pcx + pby * pcy + pbz * pcz) +
                         (pcx * pax + pcy * pay + pcz * paz);
      q[8] += 2.0 * atan2(trip, den);
    }
  }
}

// Block sums of q[0..NQ) in a fixed order -> partials[blockIdx.x * NQ + k].
__device__ __forceinline__ void block_sum_nq(const double q[NQ], double* __restrict__ partials) {
  __shared__ double red[NQ][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NQ; ++k) {
    const double v = warp_sum(q[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
    partials[(long long)blockIdx.x * NQ + threadIdx.x] = s;
  }
}

// with_q = 0: the five energies (and m) only, without the solid angles of the
// topological charge -- FP64 atan2 per plaquette, the dearest part on a GPU
// whose FP64 rate is a small fraction of its FP32 rate; the energies are the
// same bit for bit.  Parallel-tempering swaps need only the energies.
template <typename T>
__global__ void __launch_bounds__(256) k_energy(Geom g, const EnCoef* __restrict__ ep, const T* __restrict__ m,
                                                const T* __restrict__ h, double* __restrict__ partials,
                                                int with_q) {
  const EnCoef e = ep[blockIdx.z];
  m += blockIdx.z * 3 * g.n;
  if (h) h += blockIdx.z * 3 * g.n;
  partials += (long long)blockIdx.z * gridDim.x * NQ;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double q[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) q[k] = 0;
  if (i < g.n) energy_terms_at<T>(g, e, m, h, i, with_q != 0, q);
  block_sum_nq(q, partials);
}

// The five energies of FP32 replicas for parallel-tempering swaps: each cell's
// terms in FP32 (the working precision of the replicas' own updates), summed
// per thread over ENL_CELLS cells in FP32 and from there in FP64.  Within
// ~1e-6 relative of the FP64-per-cell evaluation (k_energy) of the same state,
// far below what a swap decision resolves (kT ~ 1e-3 of these energies), at
// a small fraction of its cost on a GPU with a low FP64 rate.  q[5..8] are 0.
constexpr int ENL_CELLS = 8;
// SPLIT: m and h in the colour-split order.
template <bool SPLIT>
__global__ void __launch_bounds__(256) k_energy_lean(Geom g, const EnCoef* __restrict__ ep,
                                                     const float* __restrict__ m, const float* __restrict__ h,
                                                     double* __restrict__ partials) {
  const EnCoef e = ep[blockIdx.z];
  const int n = (int)g.n;
  m += blockIdx.z * 3 * g.n;
  if (h) h += blockIdx.z * 3 * g.n;
  partials += (long long)blockIdx.z * gridDim.x * NQ;
  const float* mx = m;
  const float* my = m + n;
  const float* mz = m + 2 * n;
  const float aex[3] = {(float)e.aexV_d2[0], (float)e.aexV_d2[1], (float)e.aexV_d2[2]};
  const float dv0 = (float)e.dV_2d[0], dv1 = (float)e.dV_2d[1], kuv = (float)e.kuV;
  const float u0 = (float)e.u[0], u1 = (float)e.u[1], u2 = (float)e.u[2];
  const float b0 = (float)e.msVB[0], b1 = (float)e.msVB[1], b2 = (float)e.msVB[2];
  const float dmg = (float)e.demag;
  float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int row = g.dnx.div(i), x = i - row * g.nx;
    const int z = g.dny.div(row), y = row - z * g.ny;
    const auto at = [&](long long j) -> int {  // where cell j is stored
      if constexpr (!SPLIT) return (int)j;
      const int r = g.dnx.div((int)j), zz = g.dny.div(r);
      return r * g.nx + split_pos((int)j - r * g.nx, r - zz * g.ny + zz, g.nx);
    };
    const int is = at(i);
    const float ax = mx[is], ay = my[is], az = mz[is];
    for (int a = 0; a < 3; ++a) {
      long long j = nbr_idx(g, x, y, z, a, 1);
      if (j < 0) continue;
      j = at(j);
      const float ddx = mx[j] - ax, ddy = my[j] - ay, ddz = mz[j] - az;
      acc[0] += aex[a] * (ddx * ddx + ddy * ddy + ddz * ddz);
    }
    long long xp = nbr_idx(g, x, y, z, 0, 1), xm = nbr_idx(g, x, y, z, 0, -1);
    long long yp = nbr_idx(g, x, y, z, 1, 1), ym = nbr_idx(g, x, y, z, 1, -1);
    xp = xp < 0 ? xp : at(xp);
    xm = xm < 0 ? xm : at(xm);
    yp = yp < 0 ? yp : at(yp);
    ym = ym < 0 ? ym : at(ym);
    const float dxmz = (xp >= 0 ? mz[xp] : 0.f) - (xm >= 0 ? mz[xm] : 0.f);
    const float dxmx = (xp >= 0 ? mx[xp] : 0.f) - (xm >= 0 ? mx[xm] : 0.f);
    const float dymz = (yp >= 0 ? mz[yp] : 0.f) - (ym >= 0 ? mz[ym] : 0.f);
    const float dymy = (yp >= 0 ? my[yp] : 0.f) - (ym >= 0 ? my[ym] : 0.f);
    acc[1] -= ax * dv0 * dxmz + ay * dv1 * dymz - az * (dv0 * dxmx + dv1 * dymy);
    const float mu = ax * u0 + ay * u1 + az * u2;
    acc[2] -= kuv * mu * mu;
    acc[3] -= ax * b0 + ay * b1 + az * b2;
    if (h) acc[4] -= dmg * (ax * h[is] + ay * h[n + is] + az * h[2 * n + is]);
  }
  double q[NQ];
#pragma unroll
  for (int k = 0; k < NQ; ++k) q[k] = k < 5 ? (double)acc[k] : 0.0;
  block_sum_nq(q, partials);
}

static __global__ void __launch_bounds__(256) k_reduce_partials(const double* __restrict__ partials, int nblocks,
                                                                double* __restrict__ out) {
  partials += (long long)blockIdx.x * nblocks * NQ;  // one block per replica
  out += blockIdx.x * NQ;
  __shared__ double red[NQ][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = 0; k < NQ; ++k) {
    double s = 0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += partials[(long long)b * NQ + k];
    s = warp_sum(s);
    if (lane == 0) red[k][warp] = s;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
    out[threadIdx.x] = s;
  }
}

// =========================================================== effective field
// Per-term H in A/m (the DEBUG_H_FIELD dumps of src/main.cu:965-1086).
// H of one term (0-4) or of all (5) at cell i, A/m.
template <typename T>
__device__ __forceinline__ void field_at(const Geom& g, const HCoef& c, int term, const T* __restrict__ m,
                                         const T* __restrict__ h, long long i, double f[3]) {
  const long long n = g.n;
  const T* mx = m;
  const T* my = m + n;
  const T* mz = m + 2 * n;
  // cell coordinates by the multiply-shift dividers (n < 2^31)
  const int row = g.dnx.div((int)i), x = (int)i - row * g.nx;
  const int z = g.dny.div(row), y = row - z * g.ny;
  const double ax = mx[i], ay = my[i], az = mz[i];
  double f0 = 0, f1 = 0, f2 = 0;
  const bool all = term == 5;
  if (term == 0 || all) {
    for (int a = 0; a < 3; ++a)
      for (int dir = -1; dir <= 1; dir += 2) {
        const long long j = nbr_idx(g, x, y, z, a, dir);
        if (j < 0) continue;
        f0 += c.ex_d2[a] * ((double)mx[j] - ax);
        f1 += c.ex_d2[a] * ((double)my[j] - ay);
        f2 += c.ex_d2[a] * ((double)mz[j] - az);
      }
  }
  if (term == 1 || all) {
    const long long xp = nbr_idx(g, x, y, z, 0, 1), xm = nbr_idx(g, x, y, z, 0, -1);
    const long long yp = nbr_idx(g, x, y, z, 1, 1), ym = nbr_idx(g, x, y, z, 1, -1);
    const double dxmz = (xp >= 0 ? (double)mz[xp] : 0.0) - (xm >= 0 ? (double)mz[xm] : 0.0);
    const double dxmx = (xp >= 0 ? (double)mx[xp] : 0.0) - (xm >= 0 ? (double)mx[xm] : 0.0);
    const double dymz = (yp >= 0 ? (double)mz[yp] : 0.0) - (ym >= 0 ? (double)mz[ym] : 0.0);
    const double dymy = (yp >= 0 ? (double)my[yp] : 0.0) - (ym >= 0 ? (double)my[ym] : 0.0);
    f0 += c.dm_2d[0] * dxmz;
    f1 += c.dm_2d[1] * dymz;
    f2 += -(c.dm_2d[0] * dxmx + c.dm_2d[1] * dymy);
  }
  if (term == 2 || all) {
    const double mu = ax * c.u[0] + ay * c.u[1] + az * c.u[2];
    f0 += c.an * mu * c.u[0];
    f1 += c.an * mu * c.u[1];
    f2 += c.an * mu * c.u[2];
  }
  if (term == 3 || all) {
    f0 += c.b[0];
    f1 += c.b[1];
    f2 += c.b[2];
  }
  if ((term == 4 || all) && c.ms != 0.0 && h) {
    f0 += c.ms * (double)h[i];
    f1 += c.ms * (double)h[n + i];
    f2 += c.ms * (double)h[2 * n + i];
  }
  f[0] = f0;
  f[1] = f1;
  f[2] = f2;
}

// Per-term H in A/m (the DEBUG_H_FIELD dumps of src/main.cu:965-1086).
template <typename T>
__global__ void k_field(Geom g, HCoef c, int term, const T* __restrict__ m, const T* __restrict__ h,
                        double* __restrict__ out) {
  const long long n = g.n;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double f[3];
  field_at<T>(g, c, term, m, h, i, f);
  out[i] = f[0];
  out[n + i] = f[1];
  out[2 * n + i] = f[2];
}

// =========================================================== init / utility
// Uniform directions from Philox(key = seed; counter = (i, 0, 0, STREAM_INIT)),
// computed in FP64 and rounded to T (replaces randInitMx, src/mx_init.h:21-97).
template <typename T>
__global__ void k_init(long long n, uint32_t k0, uint32_t k1, T* __restrict__ m) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  mmcm::u32x4 ctr = {(uint32_t)i, 0u, 0u, mmcm::STREAM_INIT};
  mmcm::u32x4 r = mmcm::philox4x32_10(ctr, k0, k1);
  double z = 2.0 * mmcm::u01_f64(r.x) - 1.0;
  double t = 1.0 - z * z;
  if (t < 0) t = 0;
  double s = mmcm::dsqrt(t), sn, cs;
  mmcm::sincospi(2.0 * mmcm::u01_f64(r.y), &sn, &cs);
  m[i] = (T)(s * cs);
  m[n + i] = (T)(s * sn);
  m[2 * n + i] = (T)z;
}

template <typename T>
__global__ void k_from_f64(long long n, const double* __restrict__ src, T* __restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (T)src[i];
}
template <typename T>
__global__ void k_to_f64(long long n, const T* __restrict__ src, double* __restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (double)src[i];
}
template <typename T>
__global__ void k_khat_store(long long count, const double2* __restrict__ src, C<T>* __restrict__ dst) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) dst[i] = cmk<C<T>>((T)src[i].x, (T)src[i].y);
}

// =========================================================== host launchers
#define MMC_TRY_ATTR(x)                  \
  do {                                   \
    cudaError_t e_ = (x);                \
    if (e_ != cudaSuccess) return e_;    \
  } while (0)
inline size_t x_pass_smem(const FftPlan& p, int lines_per_row, int rows, size_t csize) {
  return ((size_t)((p.tw_total + 1) & ~1) + 2 * (size_t)rows * lines_per_row * p.n) * csize;
}
inline size_t col_pass_smem_lean(const FftPlan& p, int ncomp, int tx, size_t csize) {
  return ((size_t)((p.tw_total + 1) & ~1) + (size_t)ncomp * tx * col_line_stride(p, csize)) * csize;
}
inline size_t col_pass_smem(const FftPlan& p, int ncomp, int tx, size_t csize, bool mul) {
  return ((size_t)((p.tw_total + 1) & ~1) + 2 * (size_t)ncomp * tx * col_line_stride(p, csize) +
          (mul ? 6 * (size_t)p.n * tx : 0)) *
         csize;
}
// Two line buffers and no tensor tile (the tensor read from global memory).
inline size_t col_pass_smem_kglobal(const FftPlan& p, int ncomp, int tx, size_t csize) {
  return col_pass_smem(p, ncomp, tx, csize, false);
}

// The warp-shaped x-pass kernels for the plan's (A, B), or null.
template <typename T>
struct XPassW {
  void (*fwd)(FftPlan, int, FastDiv, int, const T*, long long, C<T>*, long long, int, int, int, int, long long,
              long long);
  void (*inv)(FftPlan, const C<T>*, long long, int, int, int, FastDiv, FastDiv, int, T*, long long, int, long long,
              long long);
};
template <typename T, bool SPLIT = false>
XPassW<T> x_pass_w(const FftPlan& p) {
  if constexpr (__is_same(T, double)) return {nullptr, nullptr};  // lines64.cuh
  else {
#define MMC_XW(A_, B_) \
  if (p.warp_a == A_ && p.warp_b == B_) {                                                    \
    if constexpr (sizeof(T) == 4)                                                           \
      return {k_x_forward_r<A_, B_, SPLIT>, k_x_inverse_r<A_, B_, SPLIT>};                  \
    else                                                                                    \
      return {k_x_forward_w<T, A_, B_>, k_x_inverse_w<T, A_, B_>};                          \
  }
  MMC_XW(32, 32)
  MMC_XW(32, 16)
  MMC_XW(16, 16)
  MMC_XW(16, 8)
  MMC_XW(8, 8)
  MMC_XW(16, 2)
  MMC_XW(8, 4)
#undef MMC_XW
  return {nullptr, nullptr};
  }
}
inline size_t x_pass_w_smem(const FftPlan& p, int rows, int threads, size_t csize) {
  // a line's room per row and pair, or (FP32) per line in flight
  const size_t lines = csize == 8 ? (size_t)(threads / p.warp_b) : 2 * (size_t)rows;
  return ((size_t)p.n + lines * (p.n + p.warp_a)) * csize;
}

// Raises the dynamic shared-memory limit of the FFT pass kernels to the
// device's opt-in maximum.  Called once per device at handle creation, never
// inside a stream capture.
template <typename T>
cudaError_t prepare_passes(int max_dyn_smem) {
  const void* fns[] = {(const void*)k_x_forward<T, 3, false>,    (const void*)k_x_forward<T, 3, true>,
                       (const void*)k_x_inverse<T, false>,       (const void*)k_x_inverse<T, true>,
                       (const void*)k_col_pass<T, false, false>, (const void*)k_col_pass<T, true, false>,
                       (const void*)k_col_pass<T, false, true>};
  for (const void* f : fns) MMC_TRY_ATTR(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
  if constexpr (__is_same(T, double)) return l64_prepare(max_dyn_smem);
  else {
    const void* wide[] = {(const void*)k_col_pass_wide<T, false>, (const void*)k_col_pass_wide<T, true>};
    for (const void* f : wide) MMC_TRY_ATTR(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
    if constexpr (__is_same(T, f64s))  // the tensor's six blocks
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_x_forward<T, 6, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
    for (int s = 0; s < 7; ++s) {
      FftPlan p{};
      const int ab[7][2] = {{32, 32}, {32, 16}, {16, 16}, {16, 8}, {8, 8}, {16, 2}, {8, 4}};
      p.warp_a = ab[s][0];
      p.warp_b = ab[s][1];
      const XPassW<T> w = x_pass_w<T>(p);
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)w.fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)w.inv, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
      if constexpr (sizeof(T) == 4) {
        const XPassW<T> ws = x_pass_w<T, true>(p);
        MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)ws.fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
        MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)ws.inv, cudaFuncAttributeMaxDynamicSharedMemorySize, max_dyn_smem));
      }
    }
    if constexpr (sizeof(T) == 4) {
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_col_pipe<16, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)col_pipe_smem<16, 16>()));
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_col_pipe<16, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)col_pipe_smem<16, 8>()));
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_col_pipe<8, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)col_pipe_smem<8, 8>()));
      MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_col_pipe<8, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)col_pipe_smem<8, 4>()));
    }
    return cudaSuccess;
  }
}
template <typename T>
cudaError_t prepare_impl(int max_dyn_smem) {
  MMC_TRY_ATTR(prepare_passes<T>(max_dyn_smem));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_tile<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)mc_tile_smem<T>()));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_band<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)MC_BAND_SMEM_MAX));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_band<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)MC_BAND_SMEM_MAX));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_strip<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    max_dyn_smem));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_strip<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    max_dyn_smem));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_pipe<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    max_dyn_smem));
  MMC_TRY_ATTR(cudaFuncSetAttribute((const void*)k_mc_pipe<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    max_dyn_smem));
  // the error word's address, looked up now rather than during a graph capture
  if (!mc_pipe_err_word()) return cudaErrorInvalidDevice;
  return cudaSuccess;
}

template <typename T>
cudaError_t run_x_forward(const FftPlan& p, int ncomp, int xdata, int ydata, int nrows, const T* in,
                          long long in_cstride, C<T>* S, long long nspec, int nyp, int hx, int pitch, int rpc,
                          int threads, cudaStream_t st, int nrep = 1, long long in_rstride = 0,
                          long long s_rstride = 0, bool split = false) {
  if (ncomp == 3) {
    XPassW<T> w = x_pass_w<T>(p);
    if constexpr (sizeof(T) == 4) {
      if (split) w = x_pass_w<T, true>(p);
    }
    if (w.fwd) {
      dim3 grid((nrows + rpc - 1) / rpc, 1, nrep);
      return launch_pdl(w.fwd, grid, dim3(threads), x_pass_w_smem(p, rpc, threads, sizeof(C<T>)), st, p, xdata,
                        FastDiv((uint32_t)ydata), nrows, in, in_cstride, S, nspec, nyp, hx, pitch, rpc, in_rstride,
                        s_rstride);
    }
  }
  if (ncomp == 3 && p.warp_a == 32) return cudaErrorInvalidValue;  // the wide shapes have warp-shaped x passes
  const int lines = (ncomp + 1) / 2;
  size_t sm = x_pass_smem(p, lines, rpc, sizeof(C<T>));
  dim3 grid((nrows + rpc - 1) / rpc, 1, nrep);
  auto kern = plan_odd(p) ? k_x_forward<T, 3, true> : k_x_forward<T, 3, false>;
  if constexpr (__is_same(T, f64s)) {
    if (ncomp == 6) kern = k_x_forward<T, 6, true>;  // the tensor's six blocks
  }
  if (ncomp != 3 && !(ncomp == 6 && __is_same(T, f64s))) return cudaErrorInvalidValue;
  kern<<<grid, threads, sm, st>>>(p, xdata, FastDiv((uint32_t)ydata), nrows, in, in_cstride, S, nspec, nyp,
                                  FastDiv((uint32_t)hx), pitch, rpc, in_rstride, s_rstride);
  return cudaGetLastError();
}

// Whether a launch shape takes the pipelined film column pass (col_lean 2 or 3).
inline int col_regs(const DemagTuning& tun) { return tun.col_lean >= 2 ? 1 : 0; }
template <typename T>
cudaError_t run_col_pass(const FftPlan& p, int ncomp, C<T>* S, long long nspec, const C<T>* khat, int hx,
                         int planes, long long plane_stride, long long pos_stride, int load_lim, int store_lim,
                         int flags, T inv_n, int tx, int threads, cudaStream_t st, int nrep = 1,
                         long long s_rstride = 0, bool inl = false, bool lean = false, int regs = 0) {
  if (ncomp == 3 && p.n <= 16 && p.full_off > 0) {  // short lines: one thread per column and component
    const ColShortFn<T> ks = col_short_kernel<T>(p.n);
    constexpr int CSH_COLS = csh_cols<T>;
    if (ks && (long long)hx * planes < INT_MAX - CSH_COLS) {
      const int total = hx * planes;
      dim3 grid((total + CSH_COLS - 1) / CSH_COLS, 1, nrep);
      return launch_pdl(ks, grid, dim3(3 * CSH_COLS), 0, st, p, S, nspec, khat, FastDiv((uint32_t)hx), hx, total,
                        plane_stride, pos_stride, load_lim, store_lim, flags, inv_n, s_rstride);
    }
  }
  if constexpr (__is_same(T, double)) {
    L64Fns f;
    if (ncomp == 3 && l64_pick(p, (long long)hx * planes * nrep, f)) {
      const int mode = (flags & PASS_MUL) ? 2 : (flags & PASS_INV) ? 1 : 0;
      return launch_pdl(f.col[mode], dim3((hx + f.tile - 1) / f.tile, planes, nrep), dim3(f.threads), f.smem, st, p, S,
                        nspec, khat, hx, plane_stride, pos_stride, load_lim, store_lim, (flags & PASS_SYM) ? 1 : 0,
                        inv_n, s_rstride);
    }
  }
  if constexpr (sizeof(T) == 4) {
    if (ncomp == 3 && p.warp_a && (flags == PASS_FWD || flags == PASS_INV) && planes <= 65535 && nrep <= 21845)
      return flags == PASS_FWD ? launch_col_lines<false>(p, S, nspec, hx, planes, plane_stride, pos_stride, load_lim,
                                                         store_lim, s_rstride, nrep, st)
                               : launch_col_lines<true>(p, S, nspec, hx, planes, plane_stride, pos_stride, load_lim,
                                                        store_lim, s_rstride, nrep, st);
    if (regs && ncomp == 3 && planes == 1 && (flags & ~PASS_SYM) == (PASS_FWD | PASS_MUL | PASS_INV) &&
        pos_stride < (1LL << 31) && (nrep == 1 || s_rstride == 3 * nspec) && col_pipe_ok(p) &&
        (reinterpret_cast<uintptr_t>(S) & 15) == 0)  // its copies are of 16 bytes; a caller's scratch may lie on 8
      return launch_col_pipe(p, S, nspec, khat, hx, (int)pos_stride, load_lim, store_lim, (flags & PASS_SYM) ? 1 : 0,
                             inv_n, nrep, st);
  }
  if (tx < 1 || (tx & (tx - 1)) != 0 || threads % tx != 0) return cudaErrorInvalidValue;  // see k_col_pass
  // in-place transforms exist for the warp path only
  int lmode = lean && p.warp_a != 0 ? 1 : 0;
  size_t sm = lmode ? col_pass_smem_lean(p, ncomp, tx, sizeof(C<T>))
                    : col_pass_smem(p, ncomp, tx, sizeof(C<T>), (flags & PASS_MUL) != 0);
  if (!lmode && (flags & PASS_MUL) && sm > 48 * 1024) {
    // a tensor tile that does not fit beside the two line buffers is read from
    // global memory in the product instead (the same values, so the same results)
    int dev = 0, optin = 0;
    MMC_TRY_ATTR(cudaGetDevice(&dev));
    MMC_TRY_ATTR(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (sm > (size_t)optin) {
      lmode = 2;
      sm = col_pass_smem_kglobal(p, ncomp, tx, sizeof(C<T>));
    }
  }
  dim3 grid((hx + tx - 1) / tx, planes, nrep);
  auto kern = plan_odd(p) ? k_col_pass<T, false, true> : inl ? k_col_pass<T, true, false> : k_col_pass<T, false, false>;
  if constexpr (!__is_same(T, double)) {
    if (p.warp_a == 32) kern = inl ? k_col_pass_wide<T, true> : k_col_pass_wide<T, false>;
  }
  // no more threads than the kernel's registers allow (the split of the work
  // does not change the results)
  cudaFuncAttributes fa;
  MMC_TRY_ATTR(cudaFuncGetAttributes(&fa, (const void*)kern));
  threads = std::min(threads, fa.maxThreadsPerBlock & ~31);
  threads -= threads % std::max(tx, 32);
  if (threads < 32) return cudaErrorInvalidValue;
  return launch_pdl(kern, grid, dim3(threads), sm, st, p, ncomp, S, nspec, khat, hx, plane_stride, pos_stride,
                    load_lim, store_lim, flags, inv_n, tx, s_rstride, lmode);
}

#define MMC_TRY(x)                       \
  do {                                   \
    cudaError_t e_ = (x);                \
    if (e_ != cudaSuccess) return e_;    \
  } while (0)

template <typename T>
cudaError_t demag_impl(const Geom& g, const FftPlan& px, const FftPlan& py, const FftPlan& pz,
                       const DemagTuning& tun, const T* m, T* h, void* spec, const void* khat, cudaStream_t st,
                       int nrep, cudaEvent_t* ev, int mul_flags = 0, bool split = false) {
  C<T>* S = reinterpret_cast<C<T>*>(spec);
  const C<T>* K = reinterpret_cast<const C<T>*>(khat);
  const long long ns = g.nspec;
  const long long mr = 3 * g.n, sr = 3 * ns;  // replica strides
  T inv_n = (T)(1.0 / (double)g.np);
  const int rows = g.ny * g.nz;
  if (ev) MMC_TRY(cudaEventRecord(ev[0], st));
  bool x64 = false;  // the FP64 x passes of lines64.cuh
  if constexpr (__is_same(T, double)) {
    L64Fns f;
    x64 = l64_pick(px, (long long)((rows + 1) / 2) * nrep, f);
    if (x64) {
      dim3 grid(((rows + 1) / 2 + f.tile - 1) / f.tile, 1, nrep);
      MMC_TRY(launch_pdl(f.xf, grid, dim3(f.threads), f.smem, st, px, g.nx, g.dny, rows, m, g.n, S, ns, g.nyp, g.hxp,
                         mr, sr));
      inv_n *= 0.5;  // the forward pass leaves the spectra doubled
    }
  }
  if (!x64)
    MMC_TRY(run_x_forward<T>(px, 3, g.nx, g.ny, rows, m, g.n, S, ns, g.nyp, g.hx, g.hxp, tun.x_rows_per_cta,
                           tun.x_threads, st, nrep, mr, sr, split));
  if (ev) MMC_TRY(cudaEventRecord(ev[1], st));
  const long long ystride = g.hxp, yplane = (long long)g.nyp * g.hxp;
  if (g.nzp == 1) {
    MMC_TRY(run_col_pass<T>(py, 3, S, ns, K, g.hx, 1, yplane, ystride, g.ny, g.ny,
                            PASS_FWD | PASS_MUL | PASS_INV | mul_flags, inv_n, tun.col_tx, tun.col_threads, st, nrep,
                            sr, tun.fft_inline != 0, tun.col_lean != 0, col_regs(tun)));
  } else {
    MMC_TRY(run_col_pass<T>(py, 3, S, ns, K, g.hx, g.nz, yplane, ystride, g.ny, g.nyp, PASS_FWD, inv_n, tun.col_tx,
                            tun.col_threads, st, nrep, sr, tun.fft_inline != 0, tun.col_lean != 0));
    MMC_TRY(run_col_pass<T>(pz, 3, S, ns, K, g.hx, g.nyp, ystride, yplane, g.nz, g.nz,
                            PASS_FWD | PASS_MUL | PASS_INV | mul_flags, inv_n, tun.col_tx_z, tun.col_threads, st, nrep,
                            sr, tun.fft_inline != 0, tun.col_lean != 0));
    MMC_TRY(run_col_pass<T>(py, 3, S, ns, K, g.hx, g.nz, yplane, ystride, g.nyp, g.ny, PASS_INV, inv_n, tun.col_tx,
                            tun.col_threads, st, nrep, sr, tun.fft_inline != 0, tun.col_lean != 0));
  }
  if (ev) MMC_TRY(cudaEventRecord(ev[2], st));
  const int rpc = tun.x_rows_per_cta;
  dim3 grid((rows + rpc - 1) / rpc, 1, nrep);
  XPassW<T> w = x_pass_w<T>(px);
  if constexpr (sizeof(T) == 4) {
    if (split) w = x_pass_w<T, true>(px);
  }
  if (x64) {
    if constexpr (__is_same(T, double)) {
      L64Fns f;
      l64_pick(px, (long long)((rows + 1) / 2) * nrep, f);
      MMC_TRY(launch_pdl(f.xi, dim3(((rows + 1) / 2 + f.tile - 1) / f.tile, 1, nrep), dim3(f.threads), f.smem, st, px,
                         (const double2*)S, ns, g.nyp, g.hxp, g.nx, g.dny, rows, h, g.n, sr, mr));
    }
  } else if (w.inv) {
    MMC_TRY(launch_pdl(w.inv, grid, dim3(tun.x_threads), x_pass_w_smem(px, rpc, tun.x_threads, sizeof(C<T>)), st, px,
                       (const C<T>*)S, ns, g.nyp, g.hx, g.hxp, g.dnx, g.dny, rows, h, g.n, rpc, sr, mr));
  } else {
    if (px.warp_a == 32) return cudaErrorInvalidValue;  // the wide shapes have warp-shaped x passes
    size_t sm = x_pass_smem(px, 2, rpc, sizeof(C<T>));
    auto kinv = plan_odd(px) ? k_x_inverse<T, true> : k_x_inverse<T, false>;
    kinv<<<grid, tun.x_threads, sm, st>>>(px, S, ns, g.nyp, g.hx, g.hxp, g.dnx, g.dny, rows, h, g.n, rpc, sr, mr);
  }
  MMC_TRY(cudaGetLastError());
  if (ev) MMC_TRY(cudaEventRecord(ev[3], st));
  return cudaSuccess;
}

template <typename T>
cudaError_t mc_impl(const Geom& g, const McCoef<T>* c, T* m, const T* h, const SweepCounters* ctr, int color,
                    unsigned long long* acc, cudaStream_t st, int nrep, int form) {
  const int threads = 256;
  // the forms that work in place, one launch per colour (the others: launch_mc_out)
  if (color < 0) {  // every colour of the sweep
    for (int col = 0; col < g.ncolors; ++col) MMC_TRY(mc_impl<T>(g, c, m, h, ctr, col, acc, st, nrep, form));
    return cudaSuccess;
  }
  if (form == MC_FORM_PIPE && mc_pipe_ok(g)) {
    const int band = mc_pipe_rows(g);
    const int nbands = (g.ny + band - 1) / band;
    const long long items = (long long)nrep * nbands;
    auto kern = mc_all_bonds(g) ? k_mc_pipe<T, true> : k_mc_pipe<T, false>;
    int* err = mc_pipe_err_word();
    // the bulk copies need 16-byte aligned rows: nx * sizeof(T) is a multiple
    // of 16 (nx % 4 == 0), so aligned bases suffice
    if (!err || items > INT_MAX || ((uintptr_t)m | (uintptr_t)h) % 16 != 0) return cudaErrorInvalidValue;
    int dev = 0, nsm = 0, optin = 0, per_sm = 0;
    MMC_TRY(cudaGetDevice(&dev));
    MMC_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    MMC_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    // as many buffers as keep the CTAs per SM the registers allow (at most
    // MCP_MAX_STAGES, at least MCP_MIN_STAGES)
    int nst = MCP_MIN_STAGES;
    MMC_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, MCP_THREADS, mc_pipe_smem<T>(g, nst)));
    for (int k = nst + 1; k <= MCP_MAX_STAGES && mc_pipe_smem<T>(g, k) <= (size_t)optin; ++k) {
      int q = 0;
      MMC_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, kern, MCP_THREADS, mc_pipe_smem<T>(g, k)));
      if (q < per_sm) break;
      nst = k;
    }
    const size_t smem = mc_pipe_smem<T>(g, nst);
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    // a static chunk of consecutive items per CTA, every CTA resident at once
    const long long ctas = (long long)nsm * per_sm;
    const int chunk = (int)((items + ctas - 1) / ctas);
    const int grid = (int)((items + chunk - 1) / chunk);
    return launch_pdl(kern, dim3(grid), dim3(MCP_THREADS), smem, st, g, c, m, h, ctr, color, band, nbands,
                      (int)items, chunk, nst, FastDiv((uint32_t)(g.nx / 4)), acc, err);
  }
  if (form == MC_FORM_BAND && mc_band_ok(g)) {
    const int band = mc_band_rows<T>(g, threads);
    dim3 grid((unsigned)((g.ny + band - 1) / band), 1, nrep);
    auto kern = mc_all_bonds(g) ? k_mc_band<T, true> : k_mc_band<T, false>;
    kern<<<grid, threads, mc_band_smem<T>(g, band), st>>>(
        g, c, m, h, ctr, color, band, FastDiv((uint32_t)(g.nx * sizeof(T) / 16)), FastDiv((uint32_t)(g.nx / 4)), acc);
    return cudaGetLastError();
  }
  if (form == MC_FORM_SPLIT) {
    if constexpr (sizeof(T) == 4) {
      if (!mc_split_geom_ok(g)) return cudaErrorInvalidValue;
      const long long total = (long long)g.ny * g.nz * (g.nx >> 2);
      const int upt = MCQ_UNITS;  // units per thread (1: 28.6 us at 64 x 256^2 instead of 24.3)
      dim3 grid((unsigned)((total + upt * MCSP_THREADS - 1) / (upt * MCSP_THREADS)), 1, nrep);
      auto kern = g.nz > 1 ? (mc_all_bonds(g) ? k_mc_split<true, true> : k_mc_split<false, true>)
                           : (mc_all_bonds(g) ? k_mc_split<true, false> : k_mc_split<false, false>);
      return launch_pdl(kern, grid, dim3(MCSP_THREADS), 0, st, g, c, m, h, ctr, color, upt,
                        FastDiv((uint32_t)(g.nx >> 2)), acc);
    }
    return cudaErrorInvalidValue;
  }
  if (form == MC_FORM_QUAD && mc_quad_ok(g)) {
    // 128-thread CTAs: the same warps per SM as 256 (the registers limit
    // them), in finer pieces, measured 2 us faster per batched sweep
    const int qthreads = MCQ_THREADS;
    const long long total = (long long)g.ny * g.nz * (g.nx >> 2);  // segments, two per thread
    dim3 grid((unsigned)((total + MCQ_UNITS * qthreads - 1) / (MCQ_UNITS * qthreads)), 1, nrep);
    auto kern = g.nz > 1 ? (mc_all_bonds(g) ? k_mc_quad<T, true, true> : k_mc_quad<T, false, true>)
                         : (mc_all_bonds(g) ? k_mc_quad<T, true, false> : k_mc_quad<T, false, false>);
    return launch_pdl(kern, grid, dim3(qthreads), 0, st, g, c, m, h, ctr, color, acc);
  }
  if constexpr (sizeof(T) == 8) {
    // one trial per thread; two (fuller warps of accepted trials) once the
    // launch has more CTAs than the SMs hold at a time
    const long long total = g.ncolors == 2 ? (long long)g.ny * g.nz * ((g.nx + 1) / 2) : g.n;
    const int tpt = total * nrep >= 2LL * MCL_THREADS * 152 * 8 ? 2 : 1;
    dim3 grid((unsigned)((total + tpt * MCL_THREADS - 1) / (tpt * MCL_THREADS)), 1, nrep);
    return launch_pdl(tpt == 2 ? k_mc_list<2> : k_mc_list<1>, grid, dim3(MCL_THREADS), 0, st, g, c, m, h, ctr, color,
                      acc);
  } else if (g.ncolors == 2) {
    const long long total = (long long)g.ny * g.nz * ((g.nx + 1) / 2);
    dim3 grid((unsigned)((total + threads - 1) / threads), 1, nrep);
    MMC_TRY(launch_pdl(k_mc_checker<T>, grid, dim3(threads), 0, st, g, c, m, h, ctr, color, acc));
  } else {
    dim3 grid((unsigned)((g.n + threads - 1) / threads), 1, nrep);
    k_mc_general<T><<<grid, threads, 0, st>>>(g, c, m, h, ctr, color, acc);
  }
  return cudaGetLastError();
}

inline int energy_blocks(const Geom& g) { return (int)((g.n + 255) / 256); }

template <typename T>
cudaError_t energy_impl(const Geom& g, const EnCoef* e, const T* m, const T* h, double* partials, int npartials,
                        double* out, cudaStream_t st, int nrep, int with_q) {
  const int nb = energy_blocks(g);
  if (nb > npartials) return cudaErrorInvalidValue;
  k_energy<T><<<dim3(nb, 1, nrep), 256, 0, st>>>(g, e, m, h, partials, with_q);
  MMC_TRY(cudaGetLastError());
  k_reduce_partials<<<nrep, 256, 0, st>>>(partials, nb, out);
  return cudaGetLastError();
}

// with_q < 0: the energies for tempering swaps (k_energy_lean for FP32 replicas).
template <typename T>
cudaError_t energy_swap_impl(const Geom& g, const EnCoef* e, const T* m, const T* h, double* partials,
                             int npartials, double* out, cudaStream_t st, int nrep, bool split) {
  if constexpr (sizeof(T) == 4) {
    const int nb = std::max(1, energy_blocks(g) / ENL_CELLS);
    if (nb > npartials || g.n >= (1LL << 31)) return cudaErrorInvalidValue;
    (split ? k_energy_lean<true> : k_energy_lean<false>)<<<dim3(nb, 1, nrep), 256, 0, st>>>(g, e, m, h, partials);
    MMC_TRY(cudaGetLastError());
    k_reduce_partials<<<nrep, 256, 0, st>>>(partials, nb, out);
    return cudaGetLastError();
  } else {
    return energy_impl<T>(g, e, m, h, partials, npartials, out, st, nrep, 0);
  }
}

template <typename T>
cudaError_t field_impl(const Geom& g, const HCoef& c, int term, const T* m, const T* h, double* out,
                       cudaStream_t st) {
  k_field<T><<<(unsigned)((g.n + 255) / 256), 256, 0, st>>>(g, c, term, m, h, out);
  return cudaGetLastError();
}

template <typename T>
cudaError_t init_impl(const Geom& g, uint64_t seed, T* m, cudaStream_t st) {
  k_init<T><<<(unsigned)((g.n + 255) / 256), 256, 0, st>>>(g.n, (uint32_t)(seed & 0xffffffffu),
                                                          (uint32_t)(seed >> 32), m);
  return cudaGetLastError();
}

// ----------------------------------------------------------- launcher bodies
// Explicitly instantiated for float in kernels_f32.cu and for double in kernels_f64.cu.
template <typename T>
cudaError_t launch_demag(const Geom& g, const FftPlan& px, const FftPlan& py, const FftPlan& pz,
                         const DemagTuning& tun, const T* m, T* h, void* spec, const void* khat, cudaStream_t st,
                         int nrep, cudaEvent_t* ev, bool split) {
  if (split && !mc_split_ok<T>(g, px)) return cudaErrorInvalidValue;
  return demag_impl<T>(g, px, py, pz, tun, m, h, spec, khat, st, nrep, ev, 0, split);
}
template <typename T>
cudaError_t launch_demag_sym(const Geom& g, const FftPlan& px, const FftPlan& py, const FftPlan& pz,
                             const DemagTuning& tun, const T* m, T* h, void* spec, const void* khat, cudaStream_t st) {
  return demag_impl<T>(g, px, py, pz, tun, m, h, spec, khat, st, 1, nullptr, PASS_SYM);
}
template <typename T>
cudaError_t launch_mc(const Geom& g, const McCoef<T>* c, T* m, const T* h, const SweepCounters* ctr, int color,
                      unsigned long long* acc, cudaStream_t st, int nrep, int form) {
  return mc_impl<T>(g, c, m, h, ctr, color, acc, st, nrep, form);
}
template <typename T>
cudaError_t launch_mc_out(const Geom& g, const McCoef<T>* c, const T* m_in, T* m_out, const T* h,
                          const SweepCounters* ctr, unsigned long long* acc, cudaStream_t st, int nrep, int form) {
  if (m_in == m_out) return cudaErrorInvalidValue;
  if (form == MC_FORM_TILE) {
    if (!mc_tile_ok(g)) return cudaErrorInvalidValue;
    dim3 grid((unsigned)((g.nx + MCT - 1) / MCT), (unsigned)((g.ny + MCT - 1) / MCT), nrep);
    k_mc_tile<T><<<grid, 256, mc_tile_smem<T>(), st>>>(g, c, m_in, m_out, h, ctr, acc);
    return cudaGetLastError();
  }
  if (form != MC_FORM_STRIP || !mc_strip_ok(g)) return cudaErrorInvalidValue;
  const int rows = mc_strip_rows(g);
  dim3 grid((unsigned)((g.ny + rows - 1) / rows), 1, nrep);
  auto kern = mc_all_bonds(g) ? k_mc_strip<T, true> : k_mc_strip<T, false>;
  return launch_pdl(kern, grid, dim3(MCS_THREADS), mc_strip_smem<T>(g), st, g, c, m_in, m_out, h, ctr, rows,
                    FastDiv((uint32_t)(g.nx / 4)), FastDiv((uint32_t)(g.nx / 2)), acc);
}
template <typename T>
cudaError_t launch_energy(const Geom& g, const EnCoef* e, const T* m, const T* h, double* partials, int npartials,
                          double* out, cudaStream_t st, int nrep, int with_q, bool split) {
  if (with_q < 0) return energy_swap_impl<T>(g, e, m, h, partials, npartials, out, st, nrep, split);
  if (split) return cudaErrorInvalidValue;
  return energy_impl<T>(g, e, m, h, partials, npartials, out, st, nrep, with_q);
}
template <typename T>
cudaError_t launch_field(const Geom& g, const HCoef& c, int term, const T* m, const T* h, double* out,
                         cudaStream_t st) {
  return field_impl<T>(g, c, term, m, h, out, st);
}
template <typename T>
cudaError_t launch_init(const Geom& g, uint64_t seed, T* m, cudaStream_t st) {
  return init_impl<T>(g, seed, m, st);
}
template <typename T>
cudaError_t launch_col_pass_2d(const Geom& g, const FftPlan& py, const DemagTuning& tun, void* spec,
                               const void* khat, cudaStream_t st, int nrep) {
  const T inv_n = (T)(1.0 / (double)g.np);
  return run_col_pass<T>(py, 3, reinterpret_cast<C<T>*>(spec), g.nspec, reinterpret_cast<const C<T>*>(khat), g.hx, 1,
                         (long long)g.nyp * g.hxp, g.hxp, g.ny, g.ny, PASS_FWD | PASS_MUL | PASS_INV, inv_n,
                         tun.col_tx, tun.col_threads, st, nrep, 3 * g.nspec, tun.fft_inline != 0,
                         tun.col_lean != 0, col_regs(tun));
}
template <typename T>
cudaError_t launch_prepare(int max_dyn_smem) {
  return prepare_impl<T>(max_dyn_smem);
}
template <typename T>
cudaError_t launch_from_f64(long long count, const double* src, T* dst, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_from_f64<T><<<(unsigned)((count + 255) / 256), 256, 0, st>>>(count, src, dst);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_to_f64(long long count, const T* src, double* dst, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_to_f64<T><<<(unsigned)((count + 255) / 256), 256, 0, st>>>(count, src, dst);
  return cudaGetLastError();
}
template <typename T>
cudaError_t launch_khat_store(long long count, const double2* spec64, void* khat, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  k_khat_store<T><<<(unsigned)((count + 255) / 256), 256, 0, st>>>(count, spec64, reinterpret_cast<C<T>*>(khat));
  return cudaGetLastError();
}

#define MMC_INSTANTIATE_LAUNCHERS(T)                                                                          \
  template cudaError_t launch_demag<T>(const Geom&, const FftPlan&, const FftPlan&, const FftPlan&,           \
                                       const DemagTuning&, const T*, T*, void*, const void*, cudaStream_t, int, \
                                       cudaEvent_t*, bool);                                                    \
  template cudaError_t launch_demag_sym<T>(const Geom&, const FftPlan&, const FftPlan&, const FftPlan&,       \
                                           const DemagTuning&, const T*, T*, void*, const void*, cudaStream_t); \
  template cudaError_t launch_mc<T>(const Geom&, const McCoef<T>*, T*, const T*, const SweepCounters*, int,   \
                                    unsigned long long*, cudaStream_t, int, int);                             \
  template cudaError_t launch_mc_out<T>(const Geom&, const McCoef<T>*, const T*, T*, const T*,               \
                                        const SweepCounters*, unsigned long long*, cudaStream_t, int, int);    \
  template cudaError_t launch_energy<T>(const Geom&, const EnCoef*, const T*, const T*, double*, int, double*, \
                                        cudaStream_t, int, int, bool);                                         \
  template cudaError_t launch_field<T>(const Geom&, const HCoef&, int, const T*, const T*, double*,            \
                                       cudaStream_t);                                                          \
  template cudaError_t launch_init<T>(const Geom&, uint64_t, T*, cudaStream_t);                               \
  template cudaError_t launch_prepare<T>(int);                                                                \
  template cudaError_t launch_col_pass_2d<T>(const Geom&, const FftPlan&, const DemagTuning&, void*, const void*, \
                                             cudaStream_t, int);                                              \
  template cudaError_t launch_from_f64<T>(long long, const double*, T*, cudaStream_t);                        \
  template cudaError_t launch_to_f64<T>(long long, const T*, double*, cudaStream_t);                          \
  template cudaError_t launch_khat_store<T>(long long, const double2*, void*, cudaStream_t);

}  // namespace mmc

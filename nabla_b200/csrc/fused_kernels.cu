// Memory-bound fused kernels for sm_100a: LayerNorm fwd/bwd, softmax / log-softmax,
// cross-entropy fwd/bwd, AdamW / SGD steps, embedding gather / scatter-add, activation
// backward, column sums (bias gradients), casts, Philox RNG, dropout, NF4 dequantisation,
// pooling and a direct NHWC convolution for small channel counts.
//
// These replace compositions of primitive ops in the reference:
//   layer_norm         nabla/nn/functional/layers.py:38-56   (9 primitive ops)
//   cross_entropy      nabla/nn/functional/losses.py:20-44   (logsoftmax, one-hot mul, sum)
//   adamw_step         nabla/nn/optim/functional.py:116-162  (~15 primitive ops per leaf)
//   embedding          nabla/nn/functional/layers.py:84-98 + nabla/ops/view/indexing.py
//   dequantize_nf4     nabla/nn/finetune/qlora.py:77-98
//   pooling            nabla/ops/pooling.py:53-137 (python loop of slices)
// All of them are bandwidth bound: 16-byte vector accesses, fp32 math, one pass over DRAM
// where the row fits in registers / L1.
#include <cuda_runtime.h>
#include <cfloat>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "launch.cuh"
#include "nb_debug.cuh"

namespace nbk {

typedef __nv_bfloat16 bf16;

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16(v); }

// 16-byte vector of T
template <typename T> struct Vec { static constexpr int N = 16 / sizeof(T); };

template <typename T>
__device__ __forceinline__ void load_vec(const T* p, float* out) {
  uint4 raw = *reinterpret_cast<const uint4*>(p);
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < Vec<T>::N; ++i) out[i] = to_f<T>(e[i]);
}
template <typename T>
__device__ __forceinline__ void store_vec(T* p, const float* in) {
  uint4 raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < Vec<T>::N; ++i) e[i] = from_f<T>(in[i]);
  *reinterpret_cast<uint4*>(p) = raw;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int NW>
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = 0.f;
#pragma unroll
  for (int i = 0; i < NW; ++i) r += sh[i];
  return r;
}
template <int NW>
__device__ __forceinline__ float block_max(float v, float* sh) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = -INFINITY;
#pragma unroll
  for (int i = 0; i < NW; ++i) r = fmaxf(r, sh[i]);
  return r;
}

// ============================================================== LayerNorm
template <typename T>
__device__ __forceinline__ void unpack_vec(const uint4& raw, float* out) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < Vec<T>::N; ++i) out[i] = to_f<T>(e[i]);
}

// 16-byte vector <-> pairs of floats, for the packed two-wide fp32 instructions (fma.rn.f32x2).
template <typename T> __device__ __forceinline__ void unpack_pairs(const uint4& raw, float2* out);
template <> __device__ __forceinline__ void unpack_pairs<float>(const uint4& raw, float2* out) {
  out[0] = make_float2(__uint_as_float(raw.x), __uint_as_float(raw.y));
  out[1] = make_float2(__uint_as_float(raw.z), __uint_as_float(raw.w));
}
template <> __device__ __forceinline__ void unpack_pairs<bf16>(const uint4& raw, float2* out) {
  const unsigned w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) out[k] = make_float2(__uint_as_float(w[k] << 16), __uint_as_float(w[k] & 0xffff0000u));
}
template <typename T> __device__ __forceinline__ uint4 pack_pairs(const float2* in);
template <> __device__ __forceinline__ uint4 pack_pairs<float>(const float2* in) {
  return make_uint4(__float_as_uint(in[0].x), __float_as_uint(in[0].y), __float_as_uint(in[1].x), __float_as_uint(in[1].y));
}
template <> __device__ __forceinline__ uint4 pack_pairs<bf16>(const float2* in) {
  unsigned w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    __nv_bfloat162 h = __float22bfloat162_rn(in[k]);
    w[k] = *reinterpret_cast<unsigned*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One warp per row. The row is read once and stays in registers in its packed 16-byte form
// (D <= 32 * VPL * Vec::N); it is unpacked for the mean, the variance and the output, which keeps
// the register count low enough for the number of rows in flight that a bandwidth-bound pass needs. The arithmetic on bf16 is two elements wide:
// that, twice the elements of fp32 in the same bytes, was bound by instructions (16384 x 2048 30.4 us, 26.1 so; HBM's copy rate is
// 20.5), and wider rows have the registers that they need (8192 x 4096 51.3, 32.8, with 64 they spilled).
template <typename T, int VPL>
__global__ void __launch_bounds__(128, VPL <= 4 || (VPL <= 8 && sizeof(T) == 4) ? 8 : VPL <= 8 ? 7 : 4) layernorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ gamma,
                                                              const T* __restrict__ beta, T* __restrict__ y,
                                                              float* __restrict__ mean, float* __restrict__ rstd,
                                                              int rows, int D, float eps) {
  // (of wider rows 16384 x 2048 24.2 us, 25.7 by ending)
  nb::follow_grid_when(VPL > 1 || gridDim.x <= nb::MANY_BLOCKS, x, gamma, beta);
  constexpr int V = Vec<T>::N, P = V / 2;
  constexpr bool PAIRS = sizeof(T) == 2;             // (16384 x 1024 fp32 25.0 us one at a time, 27.4 two)
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + (size_t)row * D;
  uint4 raw[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) raw[i] = *reinterpret_cast<const uint4*>(xr + c);
  }
  // one pass over the registers for both moments (shifted by the row's first element so that the
  // E[x^2] - E[x]^2 form does not cancel for rows with a large common offset), one pair of warp
  // reductions issued back to back
  const float shift = __shfl_sync(0xffffffffu, to_f<T>(reinterpret_cast<const T*>(&raw[0])[0]), 0);
  float s = 0.f, q = 0.f;
  float2 s2 = make_float2(0.f, 0.f), q2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) {
      float2 v[P];
      unpack_pairs<T>(raw[i], v);
#pragma unroll
      for (int j = 0; j < P; ++j) {
        if (PAIRS) {
          const float2 d = __fadd2_rn(v[j], make_float2(-shift, -shift));
          s2 = __fadd2_rn(s2, d);
          q2 = __ffma2_rn(d, d, q2);
        } else {
          const float a = v[j].x - shift, b = v[j].y - shift;
          s += a;
          q = fmaf(a, a, q);
          s += b;
          q = fmaf(b, b, q);
        }
      }
    }
  }
  if (PAIRS) { s = s2.x + s2.y; q = q2.x + q2.y; }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    q += __shfl_xor_sync(0xffffffffu, q, o);
  }
  const float ms = s / D;
  const float mu = ms + shift;
  const float rs = rsqrtf(fmaxf(q / D - ms * ms, 0.f) + eps);
  if (lane == 0) {
    if (mean) mean[row] = mu;
    if (rstd) rstd[row] = rs;
  }
  T* yr = y + (size_t)row * D;
  const float2 rs2 = make_float2(rs, rs), nmr2 = make_float2(-mu * rs, -mu * rs);
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) {
      float2 v[P], g[P], b[P];
      unpack_pairs<T>(raw[i], v);
      if (gamma) unpack_pairs<T>(*reinterpret_cast<const uint4*>(gamma + c), g);
      if (beta) unpack_pairs<T>(*reinterpret_cast<const uint4*>(beta + c), b);
#pragma unroll
      for (int j = 0; j < P; ++j) {
        if (PAIRS) {
          const float2 n = __ffma2_rn(v[j], rs2, nmr2);
          v[j] = gamma ? (beta ? __ffma2_rn(n, g[j], b[j]) : __fmul2_rn(n, g[j])) : beta ? __fadd2_rn(n, b[j]) : n;
        } else {
          const float m = fmaf(v[j].x, rs, nmr2.x), n = fmaf(v[j].y, rs, nmr2.y);
          v[j].x = gamma ? fmaf(m, g[j].x, beta ? b[j].x : 0.f) : m + (beta ? b[j].x : 0.f);
          v[j].y = gamma ? fmaf(n, g[j].y, beta ? b[j].y : 0.f) : n + (beta ? b[j].y : 0.f);
        }
      }
      *reinterpret_cast<uint4*>(yr + c) = pack_pairs<T>(v);
    }
  }
}

// 16 bytes from global to shared memory without a register in between; the copying thread alone waits for them and reads them.
__device__ __forceinline__ void async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Backward, part 1: dx. One warp per row. The row's x and dy stay in registers in their packed
// 16-byte form (half the registers of keeping them as floats, so twice as many rows are in flight
// per SM for this bandwidth-bound pass) and are unpacked once for the two sums and once for dx.
template <typename T, int VPL>
__global__ void __launch_bounds__(128, 4) layernorm_bwd_dx_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                              const T* __restrict__ gamma, const float* __restrict__ mean,
                                                              const float* __restrict__ rstd, T* __restrict__ dx,
                                                              int rows, int D) {
  nb::follow_grid(dy, x, gamma, mean, rstd);
  constexpr int V = Vec<T>::N;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + (size_t)row * D;
  const T* dyr = dy + (size_t)row * D;
  uint4 xraw[VPL], draw[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) {
      xraw[i] = *reinterpret_cast<const uint4*>(xr + c);
      draw[i] = *reinterpret_cast<const uint4*>(dyr + c);
    }
  }
  const float mu = mean[row], rs = rstd[row];
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) {
      float xv[V], dv[V], gm[V];
      unpack_vec<T>(xraw[i], xv);
      unpack_vec<T>(draw[i], dv);
      if (gamma) load_vec<T>(gamma + c, gm);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float g = dv[j] * (gamma ? gm[j] : 1.f);
        s1 += g;
        s2 += g * (xv[j] - mu) * rs;
      }
    }
  }
  s1 = warp_sum(s1) / D;
  s2 = warp_sum(s2) / D;
  T* dxr = dx + (size_t)row * D;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int c = (i * 32 + lane) * V;
    if (c < D) {
      float xv[V], dv[V], gm[V], o[V];
      unpack_vec<T>(xraw[i], xv);
      unpack_vec<T>(draw[i], dv);
      if (gamma) load_vec<T>(gamma + c, gm);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const float g = dv[j] * (gamma ? gm[j] : 1.f);
        o[j] = (g - s1 - (xv[j] - mu) * rs * s2) * rs;
      }
      store_vec<T>(dxr + c, o);
    }
  }
}

// Backward in one pass (rows of one vector per lane): a persistent grid of warps walks the rows,
// each warp computing dx of its row as above while it also adds the row's dy * xhat and dy into
// register accumulators of its lanes' columns, so dy and x are read from DRAM once
// instead of twice. At the end the four warps of a block fold their accumulators through shared
// memory and the block writes one row of `partial` ([gridDim.x][2][D] fp32), which
// colsum_partials_kernel adds up into dgamma / dbeta.
// ADD: dx += add, the gradient that reaches x beside the norm (a residual connection), rounded once.
template <typename T, bool ADD>
__global__ void __launch_bounds__(128, 4)
    layernorm_bwd_fused_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                               const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ add,
                               T* __restrict__ dx, float* __restrict__ partial, int rows, int D) {
  nb::follow_grid(dy, x, gamma, mean, rstd, add);
  constexpr int V = Vec<T>::N, P = V / 2;
  __shared__ float sh[2][32 * V];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = lane * V;
  const bool act = c < D;
  float2 ag[P], ab[P];
#pragma unroll
  for (int k = 0; k < P; ++k) ag[k] = ab[k] = make_float2(0.f, 0.f);
  for (int row = blockIdx.x * 4 + warp; row < rows; row += gridDim.x * 4) {
    uint4 xraw, draw, araw;
    if (act) {
      if (ADD) araw = *reinterpret_cast<const uint4*>(add + (size_t)row * D + c);
      xraw = *reinterpret_cast<const uint4*>(x + (size_t)row * D + c);
      draw = *reinterpret_cast<const uint4*>(dy + (size_t)row * D + c);
    }
    const float mu = mean[row], rs = rstd[row];
    const float2 rs2 = make_float2(rs, rs), nmr2 = make_float2(-mu * rs, -mu * rs);
    float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f), xv[P], dv[P], gm[P];
    if (act) {
      unpack_pairs<T>(xraw, xv);
      unpack_pairs<T>(draw, dv);
      if (gamma) unpack_pairs<T>(*reinterpret_cast<const uint4*>(gamma + c), gm);
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const float2 xh = __ffma2_rn(xv[k], rs2, nmr2);              // (x - mean) * rstd
        const float2 g = gamma ? __fmul2_rn(dv[k], gm[k]) : dv[k];
        s1 = __fadd2_rn(s1, g);
        s2 = __ffma2_rn(g, xh, s2);
        ag[k] = __ffma2_rn(dv[k], xh, ag[k]);
        ab[k] = __fadd2_rn(ab[k], dv[k]);
      }
    }
    const float m1 = warp_sum(s1.x + s1.y) / D;
    const float m2 = warp_sum(s2.x + s2.y) / D;
    if (act) {
      // dx = rstd * (g - m1 - xhat * m2) = g * rstd + (xhat * (-rstd * m2) + (-rstd * m1))
      const float2 a2 = make_float2(-rs * m2, -rs * m2), b2 = make_float2(-rs * m1, -rs * m1);
      float2 o[P];
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const float2 xh = __ffma2_rn(xv[k], rs2, nmr2);
        const float2 g = gamma ? __fmul2_rn(dv[k], gm[k]) : dv[k];
        o[k] = __ffma2_rn(g, rs2, __ffma2_rn(xh, a2, b2));
      }
      if (ADD) {
        float2 e[P];
        unpack_pairs<T>(araw, e);
#pragma unroll
        for (int k = 0; k < P; ++k) o[k] = __fadd2_rn(o[k], e[k]);
      }
      *reinterpret_cast<uint4*>(dx + (size_t)row * D + c) = pack_pairs<T>(o);
    }
  }
  for (int w = 0; w < 4; ++w) {
    if (warp == w && act) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        sh[0][c + 2 * k] = (w == 0 ? 0.f : sh[0][c + 2 * k]) + ag[k].x;
        sh[0][c + 2 * k + 1] = (w == 0 ? 0.f : sh[0][c + 2 * k + 1]) + ag[k].y;
        sh[1][c + 2 * k] = (w == 0 ? 0.f : sh[1][c + 2 * k]) + ab[k].x;
        sh[1][c + 2 * k + 1] = (w == 0 ? 0.f : sh[1][c + 2 * k + 1]) + ab[k].y;
      }
    }
    __syncthreads();
  }
  float* prow = partial + (size_t)blockIdx.x * 2 * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) {
    prow[i] = sh[0][i];
    prow[D + i] = sh[1][i];
  }
}

// Backward in one pass for wider rows: NW warps share a row, one 16-byte vector of x and dy per thread, so
// gamma and the column sums of a thread's V columns sit in registers for the whole launch and 32 warps fit
// an SM (a warp per row holds 8 vectors per lane and their sums in 200 registers: 8 warps per SM, and half
// of HBM's rate left unused). RB = 8 / NW rows per block at a time, two of them in flight per thread; the row
// sums meet in shared memory, double buffered, one barrier per two rows. 16384 x 2048 bf16: 83 -> 52 us with the
// column sums' second launch; 8192 x 4096: 165 -> 65 us. Each block writes one row of
// `partial` as above.
constexpr int LN_MAX_WARPS = 16;
template <typename T, bool ADD>
__global__ void __launch_bounds__(32 * LN_MAX_WARPS, 2)
    layernorm_bwd_rows_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ gamma,
                              const float* __restrict__ mean, const float* __restrict__ rstd, const T* __restrict__ add,
                              T* __restrict__ dx, float* __restrict__ partial, int rows, int D, int NW, int RB) {
  nb::follow_grid(dy, x, gamma, mean, rstd, add);
  constexpr int V = Vec<T>::N, P = V / 2;
  __shared__ float red[2][LN_MAX_WARPS][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, slot = wid / NW, c = ((wid - slot * NW) * 32 + lane) * V;
  const bool act = c < D;
  const float inv_d = 1.f / D;
  float2 gm[P], ag[P], ab[P];
#pragma unroll
  for (int k = 0; k < P; ++k) { gm[k] = make_float2(1.f, 1.f); ag[k] = ab[k] = make_float2(0.f, 0.f); }
  if (gamma && act) unpack_pairs<T>(*reinterpret_cast<const uint4*>(gamma + c), gm);
  const int stride = gridDim.x * RB;
  // The next pair of rows is on its way to shared memory while a pair is worked on: a thread's own vectors, which it alone waits for
  // and reads. With the loads in front of their use the memory waited for a block's sums and barrier. us with the column sums' launch, before and
  // with this and the shorter exchange of the sums: 16384 x 2048 bf16 52.5, 49.3, with `add` 67.9, 57.5; 8192 x 4096 58.8, 51.1; 8192 x 2048 fp32 49.0, 38.1.
  constexpr int W = ADD ? 3 : 2, AHEAD = 1;
  extern __shared__ uint4 ln_ring[];
  auto ask = [&](int base, int stage) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = base + u * stride + slot;
      if (row < rows && act && NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, (long long)row * D + c + V - 1, (long long)rows * D)) {
        uint4* to = ln_ring + ((stage * 2 + u) * W) * blockDim.x + threadIdx.x;
        async16(to, x + (size_t)row * D + c);
        async16(to + blockDim.x, dy + (size_t)row * D + c);
        if (ADD) async16(to + 2 * blockDim.x, add + (size_t)row * D + c);
      }
    }
    async_commit();
  };
  auto moments = [&](int base, float (&m)[2], float (&r)[2]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = base + u * stride + slot;
      m[u] = row < rows ? mean[row] : 0.f;
      r[u] = row < rows ? rstd[row] : 0.f;
    }
  };
  int buf = 0, stage = 0;
  float mn[2], rn[2];
  moments(blockIdx.x * RB, mn, rn);
#pragma unroll
  for (int k = 0; k < AHEAD; ++k) ask(blockIdx.x * RB + 2 * k * stride, k);
  for (int base = blockIdx.x * RB; base < rows; base += 2 * stride, buf ^= 1, stage = stage == AHEAD ? 0 : stage + 1) {
    float rs[2], nmr[2];
    ask(base + 2 * AHEAD * stride, stage == 0 ? AHEAD : stage - 1);
#pragma unroll
    for (int u = 0; u < 2; ++u) { rs[u] = rn[u]; nmr[u] = -mn[u] * rn[u]; }
    moments(base + 2 * stride, mn, rn);
    async_wait<AHEAD>();
    const uint4* from = ln_ring + stage * 2 * W * blockDim.x + threadIdx.x;       // [u][x, dy, add]
    float s[4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f), xv[P], dv[P];
      const float2 rs2 = make_float2(rs[u], rs[u]), nmr2 = make_float2(nmr[u], nmr[u]);
      if (act && base + u * stride + slot < rows) {
        unpack_pairs<T>(from[u * W * blockDim.x], xv);
        unpack_pairs<T>(from[(u * W + 1) * blockDim.x], dv);
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const float2 xh = __ffma2_rn(xv[k], rs2, nmr2);              // (x - mean) * rstd
          const float2 g = __fmul2_rn(dv[k], gm[k]);
          s1 = __fadd2_rn(s1, g);
          s2 = __ffma2_rn(g, xh, s2);
          ag[k] = __ffma2_rn(dv[k], xh, ag[k]);
          ab[k] = __fadd2_rn(ab[k], dv[k]);
        }
      }
      s[2 * u] = s1.x + s1.y;
      s[2 * u + 1] = s2.x + s2.y;
    }
    // The four sums over the warp, each to an eighth of its lanes, then over the row's warps by eight lanes each: what an exchange of
    // all four by all lanes and a loop over the warps take 80 instructions for, of some 230, takes 30.
    const bool upper = lane & 16, odd8 = lane & 8;
    const float a0 = (upper ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, upper ? s[0] : s[2], 16);
    const float a1 = (upper ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, upper ? s[1] : s[3], 16);
    float a = (odd8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, odd8 ? a0 : a1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const int which = lane >> 3, of = lane & 7;      // lanes 8 k .. 8 k + 7: sum k
    if (of == 0) red[buf][wid][which] = a;
    __syncthreads();
    a = of < NW ? red[buf][slot * NW + of][which] : 0.f;
    if (of + 8 < NW) a += red[buf][slot * NW + of + 8][which];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    float4 t;
    t.x = __shfl_sync(0xffffffffu, a, 0);
    t.y = __shfl_sync(0xffffffffu, a, 8);
    t.z = __shfl_sync(0xffffffffu, a, 16);
    t.w = __shfl_sync(0xffffffffu, a, 24);
    const float m1[2] = {t.x * inv_d, t.z * inv_d}, m2[2] = {t.y * inv_d, t.w * inv_d};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int row = base + u * stride + slot;
      if (act && row < rows && NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, (long long)row * D + c + V - 1, (long long)rows * D)) {
        // dx = rstd * (g - m1 - xhat * m2) = g * rstd + (xhat * (-rstd * m2) + (-rstd * m1))
        const float2 rs2 = make_float2(rs[u], rs[u]), nmr2 = make_float2(nmr[u], nmr[u]);
        const float2 a2 = make_float2(-rs[u] * m2[u], -rs[u] * m2[u]), b2 = make_float2(-rs[u] * m1[u], -rs[u] * m1[u]);
        float2 xv[P], dv[P], o[P];
        unpack_pairs<T>(from[u * W * blockDim.x], xv);
        unpack_pairs<T>(from[(u * W + 1) * blockDim.x], dv);
#pragma unroll
        for (int k = 0; k < P; ++k)
          o[k] = __ffma2_rn(__fmul2_rn(dv[k], gm[k]), rs2, __ffma2_rn(__ffma2_rn(xv[k], rs2, nmr2), a2, b2));
        if (ADD) {
          float2 e[P];
          unpack_pairs<T>(from[(u * W + 2) * blockDim.x], e);
#pragma unroll
          for (int k = 0; k < P; ++k) o[k] = __fadd2_rn(o[k], e[k]);
        }
        *reinterpret_cast<uint4*>(dx + (size_t)row * D + c) = pack_pairs<T>(o);
      }
    }
  }
  float* prow = partial + (size_t)blockIdx.x * 2 * D;
  float(*sh)[4 * 32 * V] = reinterpret_cast<float(*)[4 * 32 * V]>(ln_ring);      // the ring has been read; RB > 1 means NW <= 4
  async_wait<0>();
  __syncthreads();
  for (int r = 0; r < RB; ++r) {                     // fold the row slots, in order
    if (slot == r && act) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        float2 g = ag[k], b = ab[k];
        if (r > 0) {
          g.x += sh[0][c + 2 * k]; g.y += sh[0][c + 2 * k + 1];
          b.x += sh[1][c + 2 * k]; b.y += sh[1][c + 2 * k + 1];
        }
        if (r == RB - 1) {
          *reinterpret_cast<float2*>(prow + c + 2 * k) = g;
          *reinterpret_cast<float2*>(prow + D + c + 2 * k) = b;
        } else {
          sh[0][c + 2 * k] = g.x; sh[0][c + 2 * k + 1] = g.y;
          sh[1][c + 2 * k] = b.x; sh[1][c + 2 * k + 1] = b.y;
        }
      }
    }
    if (RB > 1) __syncthreads();
  }
}

// Backward, part 2 of the two-kernel layout (comparisons only): dgamma = sum_rows dy * xhat, dbeta = sum_rows dy. Block = 32*V columns x a
// slab of rows; 8 warps stride over the slab's rows with register accumulators; partial sums go
// to `partial` ([gridDim.y][2][D] fp32) and are folded by colsum_partials_kernel.
template <typename T>
__global__ void __launch_bounds__(256) layernorm_bwd_dgb_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                               const float* __restrict__ mean,
                                                               const float* __restrict__ rstd,
                                                               float* __restrict__ partial, int rows, int D,
                                                               int rows_per_block) {
  nb::follow_grid(dy, x, mean, rstd);
  constexpr int V = Vec<T>::N;
  __shared__ float sh[2][8][32 * V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * V;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float ag[V], ab[V];
#pragma unroll
  for (int j = 0; j < V; ++j) { ag[j] = 0.f; ab[j] = 0.f; }
  if (c < D) {
    for (int r = r0 + warp; r < r1; r += 8) {
      float xv[V], dv[V];
      load_vec<T>(x + (size_t)r * D + c, xv);
      load_vec<T>(dy + (size_t)r * D + c, dv);
      const float mu = mean[r], rs = rstd[r];
#pragma unroll
      for (int j = 0; j < V; ++j) {
        ag[j] += dv[j] * (xv[j] - mu) * rs;
        ab[j] += dv[j];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < V; ++j) { sh[0][warp][lane * V + j] = ag[j]; sh[1][warp][lane * V + j] = ab[j]; }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * V; i += blockDim.x) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { a += sh[0][w][i]; b += sh[1][w][i]; }
    const int col = blockIdx.x * 32 * V + i;
    if (col < D) {
      partial[(size_t)blockIdx.y * 2 * D + col] = a;
      partial[(size_t)blockIdx.y * 2 * D + D + col] = b;
    }
  }
}

// out0[c] = sum_b partial[b][0][c], out1[c] = sum_b partial[b][1][c]  (two planes of width D per row
// of `partial`). A block covers 32 columns of one plane; its 32 warps take every 32nd row, so several hundred
// rows of partials are a dozen or two loads per thread.
template <typename T>
__global__ void __launch_bounds__(1024) colsum_partials_kernel(const float* __restrict__ partial, T* __restrict__ out0,
                                                              T* __restrict__ out1, int nblocks, int D) {
  nb::follow_grid(partial);
  __shared__ float sh[32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float a = 0.f;
  if (c < D) {
#pragma unroll 8
    for (int i = w; i < nblocks; i += 32) a += partial[((size_t)i * 2 + blockIdx.y) * D + c];
  }
  sh[w][lane] = a;
  __syncthreads();
  a = warp_sum(sh[lane][w]);                         // warp w: column w of the block's 32
  T* out = blockIdx.y ? out1 : out0;
  if (lane == 0 && blockIdx.x * 32 + w < D && out) out[blockIdx.x * 32 + w] = from_f<T>(a);
}

// Sum of eight numbers in pairs: three roundings deep.
__device__ __forceinline__ float sum8(const float (&a)[8]) { return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7])); }

// out[i] = sum_z part[z][i], fp32 slices of n: 32 results per block, its WARPS warps take every WARPS-th slice and meet
// in a tree. 32 warps from 64 slices on, so that no chain of additions is long: several hundred slices added by 8
// warps rounded more than the blocks that made them.
template <typename T, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) fold_slices_kernel(const float* __restrict__ part, T* __restrict__ out, size_t n,
                                                                int slices) {
  nb::follow_grid(part);
  __shared__ float sh[WARPS][33];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const size_t i0 = (size_t)blockIdx.x * 32, i = i0 + lane;
  float s = 0.f;
  if (i < n) {
#pragma unroll 8
    for (int z = wq; z < slices; z += WARPS) s += part[(size_t)z * n + i];
  }
  sh[wq][lane] = s;
  __syncthreads();
  if constexpr (WARPS == 32) {                       // warp w: result w of the block's 32
    s = warp_sum(sh[lane][wq]);
    if (lane == 0 && i0 + wq < n) out[i0 + wq] = from_f<T>(s);
  } else if (wq == 0 && i < n) {
    float a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = sh[q][lane];
    out[i] = from_f<T>(sum8(a));
  }
}
template <typename T>
static void fold_slices(const float* part, void* out, size_t n, int slices, cudaStream_t stream) {
  const unsigned grid = (unsigned)((n + 31) / 32);
  if (slices < 64) nb::launch_following(fold_slices_kernel<T, 8>, grid, 256, 0, stream, part, (T*)out, n, slices);
  else nb::launch_following(fold_slices_kernel<T, 32>, grid, 1024, 0, stream, part, (T*)out, n, slices);
}

// ============================================================== small fp32 products
// out[M][N] = A B + bias for fp32 operands of any strides: the linear layers of small fp32 networks, few results of long
// sums, whose time is latency. 32 x 32 results per block, 32 steps of K staged through shared memory, the next
// ones on their way meanwhile; K is cut into gridDim.z slices (fp32 partial sums, folded by a second launch) so that the
// chip has some 300 blocks. What the library took 24.2 us for (256 x 1568 times 1568 x 10: 64-wide tiles, its own slices and
// an add for the bias) takes 7.5; 1568 x 256 times 256 x 10: 8.1 -> 7.2.
constexpr int SG = 32;
struct SgemmArgs {
  const float *a, *b, *bias;
  float* out;                                        // [M][N], or [gridDim.z][M][N] partial sums
  int M, N, K, per;                                  // per: K of a slice, a multiple of SG
  long long a_m, a_k, b_k, b_n;
};
__global__ void __launch_bounds__(256) sgemm_kernel(const SgemmArgs g) {
  nb::follow_grid();
  __shared__ float sa[SG][SG + 1], sb[SG][SG + 1];   // [k][m], [k][n]
  const int t = threadIdx.x, m0 = blockIdx.y * SG, n0 = blockIdx.x * SG;
  const int k_lo = blockIdx.z * g.per, k_hi = min(g.K, k_lo + g.per);
  // consecutive threads along the operand's unit stride
  const bool a_along_k = g.a_k == 1, b_along_n = g.b_n == 1;
  float ra[4], rb[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = t & 31, j = (t >> 5) + u * 8;
      const int am = m0 + (a_along_k ? j : i), ak = k0 + (a_along_k ? i : j);
      ra[u] = am < g.M && ak < k_hi && NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, ak, g.K) ? g.a[am * g.a_m + ak * g.a_k] : 0.f;
      const int bn = n0 + (b_along_n ? i : j), bk = k0 + (b_along_n ? j : i);
      rb[u] = bn < g.N && bk < k_hi && NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, bk, g.K) ? g.b[bk * g.b_k + bn * g.b_n] : 0.f;
    }
  };
  // thread: rows ty and ty + 16, columns tx and tx + 16
  const int tx = t & 15, ty = t >> 4;
  float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  fetch(k_lo);
  for (int k0 = k_lo; k0 < k_hi; k0 += SG) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = t & 31, j = (t >> 5) + u * 8;
      if (a_along_k) sa[i][j] = ra[u]; else sa[j][i] = ra[u];
      if (b_along_n) sb[j][i] = rb[u]; else sb[i][j] = rb[u];
    }
    __syncthreads();
    if (k0 + SG < k_hi) fetch(k0 + SG);
    const int steps = min(SG, k_hi - k0);            // (a padded step would turn an infinite operand into NaN)
    for (int k = 0; k < steps; ++k) {
      const float a0 = sa[k][ty], a1 = sa[k][ty + 16], b0 = sb[k][tx], b1 = sb[k][tx + 16];
      acc[0][0] = fmaf(a0, b0, acc[0][0]); acc[0][1] = fmaf(a0, b1, acc[0][1]);
      acc[1][0] = fmaf(a1, b0, acc[1][0]); acc[1][1] = fmaf(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
  float* out = g.out + (size_t)blockIdx.z * g.M * g.N;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int m = m0 + ty + 16 * r, n = n0 + tx + 16 * c;
      if (m < g.M && n < g.N) out[(size_t)m * g.N + n] = acc[r][c] + (g.bias != nullptr && gridDim.z == 1 ? g.bias[n] : 0.f);
    }
}
// out[m][n] = sum of the slices + bias[n]; eight lanes per result.
__global__ void __launch_bounds__(256) sgemm_fold_kernel(const float* __restrict__ part, const float* __restrict__ bias,
                                                        float* __restrict__ out, int MN, int N, int slices) {
  nb::follow_grid(part, bias);
  const int i = (blockIdx.x * 256 + threadIdx.x) % 32 + blockIdx.x * 32, q = threadIdx.x >> 5;
  __shared__ float sh[8][33];
  float s = 0.f;
  if (i < MN)
    for (int z = q; z < slices; z += 8) s += part[(size_t)z * MN + i];
  sh[q][threadIdx.x & 31] = s;
  __syncthreads();
  if (q == 0 && i < MN) {
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = sh[k][threadIdx.x];
    out[i] = sum8(a) + (bias != nullptr ? bias[i % N] : 0.f);
  }
}

// ============================================================== column sum (bias gradient)
// x [rows][N] -> partial[gridDim.y][N] ; each block sums a slab of rows for 32*V columns.
template <typename T>
__global__ void __launch_bounds__(256) colsum_kernel(const T* __restrict__ x, float* __restrict__ partial, int rows,
                                                    int N, int rows_per_block) {
  nb::follow_grid(x);
  constexpr int V = Vec<T>::N;
  __shared__ float sh[8][32 * V];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * V;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = 0.f;
  if (c < N) {
#pragma unroll 4
    for (int r = r0 + warp; r < r1; r += 8) {
      float v[V];
      load_vec<T>(x + (size_t)r * N + c, v);
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < V; ++j) sh[warp][lane * V + j] = acc[j];
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * V; i += blockDim.x) {
    float a[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) a[w] = sh[w][i];
    const int col = blockIdx.x * 32 * V + i;
    if (col < N) partial[(size_t)blockIdx.y * N + col] = sum8(a);
  }
}
// Column sums of a tall, narrow matrix (the bias gradient of a convolution: 200704 x 16): the block's 256
// threads cover 256 / (N / V) whole rows at a time, so every lane loads whatever N is; colsum_kernel gives a
// warp one row's 32 vectors and leaves 28 of 32 lanes without one there. 200704 x 16 fp32: 81 -> 15 us.
template <typename T>
__global__ void __launch_bounds__(256) colsum_narrow_kernel(const T* __restrict__ x, float* __restrict__ partial, int rows,
                                                           int N, int rows_per_block) {
  nb::follow_grid(x);
  constexpr int V = Vec<T>::N;
  __shared__ float sh[256 * V];
  const int nv = N / V, rpp = 256 / nv, r_in = threadIdx.x / nv, c = threadIdx.x % nv;
  const int r0 = blockIdx.x * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = 0.f;
  if (r_in < rpp) {
#pragma unroll 4
    for (int r = r0 + r_in; r < r1; r += rpp) {
      if (!NB_IN_BOUNDS(NB_SITE_REDUCE_INDEX, ((long long)r * N + c * V) + V - 1, (long long)rows * N)) break;
      float v[V];
      load_vec<T>(x + (size_t)r * N + c * V, v);
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < V; ++j) sh[threadIdx.x * V + j] = acc[j];
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += 256) {        // element i of row slot k sits at k * N + i
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int k = 0;
    for (; k + 8 <= rpp; k += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) a[u] += sh[(k + u) * N + i];
    }
    float s = 0.f;
    for (; k < rpp; ++k) s += sh[k * N + i];
    a[0] += s;
    partial[(size_t)blockIdx.x * N + i] = sum8(a);
  }
}

// Column sums of several matrices in one launch, without a second one that folds slabs: the blocks of a cluster share a
// tile of L vectors of columns, walk every row of it between them and meet in distributed shared memory. A block is 256 / L
// row slots, whose rows are interleaved over the cluster; a thread asks for eight rows before it adds the first and adds
// them as a tree, so no value goes through more than ceil(rows / (64 * 256 / L)) + 8 + log2(32 / L) additions that round (three in the tree, one a
// round, the slots of a warp, eight warps, eight blocks): 14 for 8192 rows and L = 8, 16 for 4096 and L = 32. Rows that are not whole aligned
// vectors go element by element (`vec` of a leaf is 0). Latency bounds it: three dependent rounds (rows, cluster, result) and the
// launch. 2002 x 512 bf16 5.2 us as slabs and fold, 3.5 so; where the line lies: colsum_clusters in native/kernels.py.
constexpr int COLSUM_GROUP = 32, COLSUM_CLUSTER = 8;
struct ColsumGroup {
  struct Leaf {
    const void* x;
    void* out;
    int rows, N;
    unsigned tile0;                                  // first column tile of the leaf
    int vec, out_bf16;
  } leaf[COLSUM_GROUP];
  int count;
};
template <typename T, int L, bool VEC>
__device__ __forceinline__ void colsum_slot(const T* __restrict__ x, int rows, int N, int c, int row, float (&acc)[Vec<T>::N]) {
  constexpr int V = VEC ? Vec<T>::N : 1, STEP = COLSUM_CLUSTER * (256 / L);
  for (int r = row; r < rows; r += 8 * STEP) {
    float v[8][V];
    if constexpr (VEC) {
      uint4 raw[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        raw[u] = make_uint4(0, 0, 0, 0);
        if (r + u * STEP < rows && NB_IN_BOUNDS(NB_SITE_REDUCE_INDEX, (long long)(r + u * STEP) * N + c + V - 1, (long long)rows * N))
          raw[u] = *reinterpret_cast<const uint4*>(x + (size_t)(r + u * STEP) * N + c);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) unpack_vec<T>(raw[u], v[u]);
    } else {
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u][0] = r + u * STEP < rows ? to_f<T>(x[(size_t)(r + u * STEP) * N + c]) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < V; ++j)
      acc[j] += ((v[0][j] + v[1][j]) + (v[2][j] + v[3][j])) + ((v[4][j] + v[5][j]) + (v[6][j] + v[7][j]));
  }
}
template <typename T, int L>
__global__ void __launch_bounds__(256) __cluster_dims__(1, COLSUM_CLUSTER, 1) colsum_group_kernel(const __grid_constant__ ColsumGroup g) {
  nb::follow_grid();
  constexpr int V = Vec<T>::N;
  __shared__ float sh[8][L * V];
  __shared__ float tot[L * V];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  int l = 0;
  while (l + 1 < g.count && blockIdx.x >= g.leaf[l + 1].tile0) ++l;
  const ColsumGroup::Leaf& t = g.leaf[l];
  const int lane = threadIdx.x % L, slot = threadIdx.x / L, rank = blockIdx.y;
  const int width = t.vec ? L * V : L, c0 = (int)(blockIdx.x - t.tile0) * width, c = c0 + lane * (t.vec ? V : 1);
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = 0.f;
  if (c < t.N) {
    const int row = rank * (256 / L) + slot;
    if (t.vec) colsum_slot<T, L, true>((const T*)t.x, t.rows, t.N, c, row, acc);
    else colsum_slot<T, L, false>((const T*)t.x, t.rows, t.N, c, row, acc);
  }
#pragma unroll
  for (int o = L; o < 32; o <<= 1)                   // slots that share a warp
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  if ((threadIdx.x & 31) < L) {
#pragma unroll
    for (int j = 0; j < V; ++j) sh[threadIdx.x >> 5][lane * V + j] = acc[j];
  }
  __syncthreads();
  // (of a leaf without vectors, element lane * V of a row of `sh` holds column lane)
  const int i = threadIdx.x, at = t.vec ? i : i * V;
  if (i < width) {
    float a[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) a[w] = sh[w][at];
    tot[i] = sum8(a);
  }
  cluster.sync();
  if (rank == 0 && i < width && c0 + i < t.N) {
    float a[8];
#pragma unroll
    for (int w = 0; w < 8; ++w) a[w] = cluster.map_shared_rank(tot, w)[i];
    const float s = sum8(a);
    if (t.out_bf16) ((bf16*)t.out)[c0 + i] = __float2bfloat16(s);
    else ((float*)t.out)[c0 + i] = s;
  }
  cluster.sync();                                    // a block's shared memory is read until here
}

// ============================================================== softmax / log-softmax (last dim)
template <typename T, bool LOG>
__global__ void __launch_bounds__(256) softmax_kernel(const T* __restrict__ x, T* __restrict__ y, int rows, int D) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS || D > 4096, x);
  __shared__ float sh[8];
  const int row = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, row, rows)) return;   // debug build: one block per row
  const T* xr = x + (size_t)row * D;
  T* yr = y + (size_t)row * D;
  float m = -INFINITY, s = 0.f;
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    const float v = to_f<T>(xr[c]);
    if (v > m) { s = s * __expf(m - v); m = v; }
    s += __expf(v - m);
  }
  const float gm = block_max<8>(m, sh);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum<8>(s, sh);
  const float lse = gm + logf(gs);
  const float inv = 1.f / gs;
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    const float v = to_f<T>(xr[c]);
    yr[c] = from_f<T>(LOG ? (v - lse) : __expf(v - gm) * inv);
  }
}

// ============================================================== cross entropy building blocks
// Per row: lse = logsumexp(logits_row); picked = logits_row[target] when 0 <= target < D else 0.
// A vocabulary shard passes targets shifted by its offset, so out-of-range simply means
// "another shard holds this class"; the caller combines shards with max/sum reductions.
//
// Rows of any width and alignment move in 16-byte vectors: the elements before a row's first 16-byte
// boundary and behind its last are taken one by one (a vocabulary that is not a multiple of 8 gives every
// row another offset). 4096 x 10001 bf16: forward 95 us with scalar rows, 33 so; gradient 98 and 37. WHOLE: all rows are
// whole aligned vectors, with no such offsets to work out. Of other rows those of up to 256 elements take one element
// per thread (65536 x 9: gradient 37 us, 43 by vectors and edges).
template <typename T>
__device__ __forceinline__ int row_head(const T* row, int D) {       // elements before the first 16-byte boundary
  return min(D, (int)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(row) & 15u)) & 15u) / sizeof(T)));
}
//
// WIDE: three vectors of a row are asked for before the first is used; one at a time left the memory waiting for the
// exponentials. From 8 vectors per thread on. us, one at a time and three: 4096 x 32000 bf16 57.8, 52.1, 100 x 32000 6.7, 4.7,
// 4096 x 8192 fp32 27.2, 24.6; below the line 4096 x 10001 bf16 21.7, 23.0, 16384 x 1000 20.1, 23.2.
template <typename T, bool WHOLE, bool WIDE>
__global__ void __launch_bounds__(256) lse_pick_fwd_kernel(const T* __restrict__ logits,
                                                          const long long* __restrict__ tgt, float* __restrict__ lse_out,
                                                          float* __restrict__ picked, int rows, int D) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS || D > 4096, logits, tgt);
  __shared__ float sh[8];
  const int row = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, row, rows)) return;   // debug build: one block per row
  const T* xr = logits + (size_t)row * D;
  // the maximum starts at the lowest finite value: elements of -inf then add exp(-inf) = 0 without a test
  float m = -FLT_MAX, s = 0.f;
  constexpr int V = Vec<T>::N;
  const int head = WHOLE ? 0 : D <= 256 ? D : row_head(xr, D), body = WHOLE ? D : (D - head) / V * V, tail = head + body;
  const int edge = threadIdx.x < head ? (int)threadIdx.x : tail + (int)threadIdx.x - head;     // one edge element per thread
  if (!WHOLE && edge < D) {
    const float v = to_f<T>(xr[edge]);
    m = fmaxf(m, v);
    s = __expf(v - m);                                         // NaN stays in s
  }
  int c = head + threadIdx.x * V;
  if constexpr (WIDE) {
    const int step = blockDim.x * V;
    for (; c + 2 * step < tail; c += 3 * step) {
      float v[3][V];
#pragma unroll
      for (int i = 0; i < 3; ++i) load_vec<T>(xr + c + i * step, v[i]);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        float lm = v[i][0];
#pragma unroll
        for (int j = 1; j < V; ++j) lm = fmaxf(lm, v[i][j]);
        if (lm > m) { s = s * __expf(m - lm); m = lm; }
#pragma unroll
        for (int j = 0; j < V; ++j) s += __expf(v[i][j] - m);
      }
    }
  }
  for (; c < tail; c += blockDim.x * V) {
    float v[V];
    load_vec<T>(xr + c, v);
    float lm = v[0];
#pragma unroll
    for (int j = 1; j < V; ++j) lm = fmaxf(lm, v[j]);
    if (lm > m) { s = s * __expf(m - lm); m = lm; }
#pragma unroll
    for (int j = 0; j < V; ++j) s += __expf(v[j] - m);
  }
  const float gm = block_max<8>(m, sh);
  s *= __expf(m - gm);
  const float gs = block_sum<8>(s, sh);
  if (threadIdx.x == 0) {
    const long long t = tgt[row];
    lse_out[row] = gm + logf(gs);
    picked[row] = (t >= 0 && t < D) ? to_f<T>(xr[t]) : 0.f;
  }
}
// dlogits = exp(logits - lse) * g_lse[row] + onehot(target) * g_pick[row]
template <typename T, bool WHOLE>
__global__ void __launch_bounds__(256) lse_pick_bwd_kernel(const T* __restrict__ logits,
                                                          const long long* __restrict__ tgt,
                                                          const float* __restrict__ lse, const float* __restrict__ g_lse,
                                                          const float* __restrict__ g_pick, T* __restrict__ dlogits,
                                                          int rows, int D) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS || D > 4096, logits, tgt, lse, g_lse, g_pick);
  const int row = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, row, rows)) return;   // debug build: one block per row
  const T* xr = logits + (size_t)row * D;
  T* dr = dlogits + (size_t)row * D;
  const float l = lse[row];
  const long long t = tgt[row];
  const float gl = g_lse ? g_lse[row] : 0.f;
  const float gp = g_pick ? g_pick[row] : 0.f;
  constexpr int V = Vec<T>::N;
  auto grad = [&](float v, int c) { return __expf(v - l) * gl + (c == t ? gp : 0.f); };
  if (!WHOLE && D <= 256) {
    const int c = threadIdx.x;
    if (c < D) dr[c] = from_f<T>(grad(to_f<T>(xr[c]), c));
    return;
  }
  // both rows have the same offset from a 16-byte boundary unless a caller's base pointers differ in it
  const int head = WHOLE ? 0 : row_head(xr, D) == row_head(dr, D) ? row_head(xr, D) : D;
  const int body = WHOLE ? D : (D - head) / V * V, tail = head + body;
  for (int e = threadIdx.x; !WHOLE && e < D - body; e += blockDim.x) {
    const int c = e < head ? e : body + e;
    dr[c] = from_f<T>(grad(to_f<T>(xr[c]), c));
  }
  for (int c = head + threadIdx.x * V; c < tail; c += blockDim.x * V) {
    float v[V], o[V];
    load_vec<T>(xr + c, v);
#pragma unroll
    for (int j = 0; j < V; ++j) o[j] = grad(v[j], c + j);
    store_vec<T>(dr + c, o);
  }
}

// ============================================================== optimizers
// AdamW with decoupled weight decay; P/G may be bf16 or fp32, moments fp32.
// step-dependent bias corrections are passed as bc1 = 1 - b1^t, bc2 = 1 - b2^t via device scalars
// when `hyper` is non-null: hyper = {lr, bc1, bc2, grad_scale}.
template <typename T>
__device__ __forceinline__ void load8(const T* p, float* out);
template <>
__device__ __forceinline__ void load8<bf16>(const bf16* p, float* out) { load_vec<bf16>(p, out); }
template <>
__device__ __forceinline__ void load8<float>(const float* p, float* out) {
  load_vec<float>(p, out);
  load_vec<float>(p + 4, out + 4);
}
template <typename T>
__device__ __forceinline__ void store8(T* p, const float* in);
template <>
__device__ __forceinline__ void store8<bf16>(bf16* p, const float* in) { store_vec<bf16>(p, in); }
template <>
__device__ __forceinline__ void store8<float>(float* p, const float* in) {
  store_vec<float>(p, in);
  store_vec<float>(p + 4, in + 4);
}

struct AdamHyper { float lr, b1, b2, eps, wd, bc1, bc2, grad_scale; };

// Elements [i, i + 8) of one tensor with 16-byte accesses (all tensors come from the caching allocator and
// are at least 16-byte aligned); the ragged tail is handled element-wise.
template <typename TP, typename TG>
__device__ __forceinline__ void adamw_update8(const TP* __restrict__ p, const TG* __restrict__ g, const float* __restrict__ m,
                                              const float* __restrict__ v, TP* __restrict__ p_out, float* __restrict__ m_out,
                                              float* __restrict__ v_out, size_t i, size_t n, const AdamHyper& h, float ibc1,
                                              float ibc2) {
  float pv[8], gv[8], mv[8], vv[8];
  const bool full = i + 8 <= n;
  if (full) {
    load8<TP>(p + i, pv);
    load8<TG>(g + i, gv);
    load8<float>(m + i, mv);
    load8<float>(v + i, vv);
  } else {
    for (int j = 0; j < 8; ++j) {
      const bool ok = i + j < n;
      pv[j] = ok ? to_f<TP>(p[i + j]) : 0.f;
      gv[j] = ok ? to_f<TG>(g[i + j]) : 0.f;
      mv[j] = ok ? m[i + j] : 0.f;
      vv[j] = ok ? v[i + j] : 0.f;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float gr = gv[j] * h.grad_scale;
    mv[j] = h.b1 * mv[j] + (1.f - h.b1) * gr;
    vv[j] = h.b2 * vv[j] + (1.f - h.b2) * gr * gr;
    const float upd = (mv[j] * ibc1) / (sqrtf(vv[j] * ibc2) + h.eps) + h.wd * pv[j];
    pv[j] -= h.lr * upd;
  }
  if (full) {
    store8<TP>(p_out + i, pv);
    store8<float>(m_out + i, mv);
    store8<float>(v_out + i, vv);
  } else {
    for (int j = 0; j < 8; ++j)
      if (i + j < n) {
        p_out[i + j] = from_f<TP>(pv[j]);
        m_out[i + j] = mv[j];
        v_out[i + j] = vv[j];
      }
  }
}
__device__ __forceinline__ void adamw_device_hyper(AdamHyper& h, const float* __restrict__ hyper) {
  if (hyper) { h.lr = hyper[0]; h.bc1 = hyper[1]; h.bc2 = hyper[2]; h.grad_scale = hyper[3]; }
}
template <typename TP, typename TG>
__global__ void __launch_bounds__(256) adamw_kernel(const TP* __restrict__ p, const TG* __restrict__ g,
                                                   const float* __restrict__ m, const float* __restrict__ v,
                                                   TP* __restrict__ p_out, float* __restrict__ m_out,
                                                   float* __restrict__ v_out, size_t n, AdamHyper h,
                                                   const float* __restrict__ hyper) {
  nb::follow_grid(p, g, m, v, hyper);
  adamw_device_hyper(h, hyper);
  const float ibc1 = 1.f / h.bc1, ibc2 = 1.f / h.bc2;
  const size_t i0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const size_t stride = (size_t)gridDim.x * blockDim.x * 8;
  for (size_t i = i0; i < n; i += stride) adamw_update8<TP, TG>(p, g, m, v, p_out, m_out, v_out, i, n, h, ibc1, ibc2);
}
// The same update of many small tensors in one launch, 2048 elements per block. A launch of one of them is 2.5 to 4 us
// whatever its size: the eight of a 64-256-256-256-1 MLP took 24 us of a 165 us step, 4.2 together.
constexpr int ADAM_GROUP = 48, ADAM_GROUP_MAX = 1 << 20;     // tensors of a launch, elements of one
struct AdamGroup {
  struct Leaf {
    const void *p, *g;
    const float *m, *v;
    void* p_out;
    float *m_out, *v_out;
    unsigned n, block0;                              // elements; first block of the leaf
  } leaf[ADAM_GROUP];
  int count;
};
template <typename TP, typename TG>
__global__ void __launch_bounds__(256) adamw_group_kernel(const __grid_constant__ AdamGroup c, AdamHyper h,
                                                         const float* __restrict__ hyper) {
  nb::follow_grid(hyper);
  adamw_device_hyper(h, hyper);
  int l = 0;
  while (l + 1 < c.count && blockIdx.x >= c.leaf[l + 1].block0) ++l;
  const AdamGroup::Leaf& t = c.leaf[l];
  const unsigned i = ((blockIdx.x - t.block0) * 256 + threadIdx.x) * 8;
  if (i >= t.n || !NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, i, t.n)) return;
  adamw_update8<TP, TG>((const TP*)t.p, (const TG*)t.g, t.m, t.v, (TP*)t.p_out, t.m_out, t.v_out, i, t.n, h, 1.f / h.bc1, 1.f / h.bc2);
}
// hyper = {lr, 1 - b1^t, 1 - b2^t, 1} for a step count t that lives on the device (in 64 bits: 1 - b2^t of the
// first steps cancels). One thread; the same four numbers took ten launches of elementwise kernels, as much
// as the updates of a small model (13 us of a 180 us training step; 2.8 now). `plus`: t is the sum of two counts, kept in `total`.
__global__ void adam_hyper_kernel(const float* __restrict__ step, const float* __restrict__ plus, float* __restrict__ total,
                                  float* __restrict__ hyper, float lr, double b1, double b2) {
  nb::follow_grid(step, plus);
  const float sum = plus != nullptr ? step[0] + plus[0] : step[0];
  if (total != nullptr) total[0] = sum;
  const double t = (double)sum;
  hyper[0] = lr;
  hyper[1] = (float)(1.0 - pow(b1, t));
  hyper[2] = (float)(1.0 - pow(b2, t));
  hyper[3] = 1.f;
}
// d = a - b (rounded to T) and the sum of d, or of d * d, over all n elements / count: the mean of a cross-entropy's rows or of a squared
// error together with the difference that its gradient is made of. One block, or the eight of a cluster, whose sums meet in
// distributed shared memory; latency bounds it. As sub, mul, a sum per axis and a division it was four or five launches of 1.2 to
// 2.5 us and three roundings of the sum; 512 x 1 bf16 8.2 -> 2.1 us, the mean of 256 rows of a cross-entropy 5.5 -> 2.4.
constexpr int MEAN_THREADS = 1024;
template <typename T, int C>
__global__ void __launch_bounds__(MEAN_THREADS) __cluster_dims__(C, 1, 1)
    mean_diff_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ d, T* __restrict__ out, int n, int square,
                     const T* __restrict__ count_at, float count) {
  nb::follow_grid(a, b, count_at);
  __shared__ float sh[MEAN_THREADS / 32], tot;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float s = 0.f;
#pragma unroll 4
  for (int i = rank * MEAN_THREADS + threadIdx.x; i < n; i += C * MEAN_THREADS) {
    const T v = from_f<T>(to_f<T>(a[i]) - to_f<T>(b[i]));
    d[i] = v;
    const float f = to_f<T>(v);
    s += square ? f * f : f;
  }
  s = warp_sum(s);
  if (lane == 0) sh[w] = s;
  __syncthreads();
  if (w == 0) {
    s = warp_sum(sh[lane]);
    if (lane == 0) tot = s;
  }
  if (C > 1) cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    float p[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) p[k] = k < C ? (C > 1 ? *cluster.map_shared_rank(&tot, k) : s) : 0.f;
    out[0] = from_f<T>(sum8(p) / (count_at != nullptr ? to_f<T>(count_at[0]) : count));
  }
  if (C > 1) cluster.sync();                         // a block's shared memory is read until here
}
template <typename TP, typename TG>
__global__ void __launch_bounds__(256) sgd_kernel(const TP* __restrict__ p, const TG* __restrict__ g,
                                                 const float* __restrict__ buf, TP* __restrict__ p_out,
                                                 float* __restrict__ buf_out, size_t n, float lr, float momentum,
                                                 float wd, float grad_scale) {
  nb::follow_grid(p, g, buf);
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t k = i0; k < n; k += stride) {
    const float pm = to_f<TP>(p[k]);
    float gr = to_f<TG>(g[k]) * grad_scale + wd * pm;
    if (buf) {
      gr = momentum * buf[k] + gr;
      buf_out[k] = gr;
    }
    p_out[k] = from_f<TP>(pm - lr * gr);
  }
}

// ============================================================== embedding
// out[i] = table[ids[i]] (+ add[i % period]: a position embedding, or one row for all). Ids outside the table give zeros.
// Bound by the write of `out` and the table's rows. 16384 ids, 32000 x 2048 bf16, 2048 positions: gather 16 us and the
// add behind it 30, 20 together.
template <typename T, bool ADD>
__global__ void __launch_bounds__(128) embedding_gather_kernel(const T* __restrict__ table,
                                                              const long long* __restrict__ ids, const T* __restrict__ add,
                                                              T* __restrict__ out, int n_ids, int D, int vocab, int period) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS, table, ids, add);
  constexpr int V = Vec<T>::N;
  const int i = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, i, n_ids)) return;   // debug build: one block per id
  long long id = ids[i];
  const bool ok = id >= 0 && id < vocab;
  const T* src = table + (size_t)(ok ? id : 0) * D;
  const T* pos = ADD ? add + (size_t)(i % period) * D : nullptr;
  T* dst = out + (size_t)i * D;
  if ((D % V) == 0) {
    for (int c = threadIdx.x * V; c < D; c += blockDim.x * V) {
      uint4 raw = ok ? *reinterpret_cast<const uint4*>(src + c) : make_uint4(0, 0, 0, 0);
      if constexpr (ADD) {
        float x[V], p[V];
        load_vec<T>(pos + c, p);
        unpack_vec<T>(raw, x);
#pragma unroll
        for (int j = 0; j < V; ++j) x[j] += p[j];
        store_vec<T>(dst + c, x);
      } else {
        *reinterpret_cast<uint4*>(dst + c) = raw;
      }
    }
  } else {
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
      const T x = ok ? src[c] : from_f<T>(0.f);
      dst[c] = ADD ? from_f<T>(to_f<T>(x) + to_f<T>(pos[c])) : x;
    }
  }
}
// out = base + scatter_add(ids, upd): the gradient of an embedding.
// Large tables: the ids are bucketed by row (three short launches over the integers), and one launch writes every
// row of the table once: rows that occur as the fp32 sum of their updates in registers, the others as zeros or as the
// base's row. No fp32 table that is zeroed, added to with atomics and converted, and, but for crowded tables, no fill of `out`.
// A row with at most SCAT_LIGHT entries is one warp's work (its loads are a list entry and then the rows, two
// latencies in a chain, so what counts is how many rows the chip has on its way: 4 KB rows by a block each were 1.4 TB/s);
// a row with more takes the whole block, in segments of SCAT_SEG entries whose fp32 partial rows are added up in two
// steps where there are several: the last block of every SCAT_GROUP segments adds those, the last group of a row the
// groups. One block per row would leave the most frequent id, some 1000 of 16384 tokens (ids of text fall off about as
// 1 / rank), to one block, and joining them in one step the padding id of a batch (29700 of 33000 ids into 4097 x 2048
// fp32: 881 us in one step, 128 in two).
// 16384 ids of text into 32000 x 2048 bf16, bucketing included: fill and rows 68 us, 54 so (131 MB written, 67 read: 30 us at the
// copy rate); onto a base table 92, 79.
constexpr int SCAT_SEG = 32, SCAT_GROUP = 32, SCAT_LIGHT = 4;
struct ScatWs {
  int *counts, *done, *total, *nseg, *nheavy, *nlight;   // zeroed by the launcher
  int light;                                    // most entries of a row that one warp adds: SCAT_LIGHT, or 0
  int* gdone;                                   // likewise zeroed: finished segments of a group, at its first partial row
  int *start, *rank, *list;                     // first list slot per row; place of an entry in its row; entries by row
  int4* seg;                                    // (row, first list slot, entries, partial row or -1): the rows of at most
                                                // SCAT_LIGHT entries from the end backwards, the others from the start on
};
// Segment q of a row of `c` entries from list slot `at` on; h: its first partial row, or -1.
__device__ __forceinline__ int4 scatter_segment(int v, int c, int at, int h, int q) {
  return make_int4(v, at + q * SCAT_SEG, min(SCAT_SEG, c - q * SCAT_SEG), h < 0 ? -1 : h + q);
}
// Lanes of a warp with the same id share one atomic; returns the entry's place among those of its row.
__device__ __forceinline__ int scatter_rank(int* counts, long long id, bool ok) {
  const unsigned same = __match_any_sync(0xffffffffu, ok ? (int)id : -1);
  const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
  int base = 0;
  if (ok && lane == leader) base = atomicAdd(counts + id, __popc(same));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(same & ((1u << lane) - 1u));
}
// Inclusive scan over the block, two numbers packed in the halves of 64 bits.
template <int NW>
__device__ __forceinline__ unsigned long long scatter_scan(unsigned long long x, unsigned long long* wsum,
                                                           unsigned long long& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  unsigned long long before = 0, all = 0;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    if (i < w) before += wsum[i];
    all += wsum[i];
  }
  total = all;
  return x + before;
}

__global__ void __launch_bounds__(256) scatter_count_kernel(const long long* __restrict__ ids, ScatWs ws, int n_ids, int vocab) {
  nb::follow_grid(ids);
  const int i = blockIdx.x * 256 + threadIdx.x;
  const long long id = i < n_ids ? ids[i] : -1;
  const bool ok = id >= 0 && id < vocab;
  const int rank = scatter_rank(ws.counts, id, ok);
  if (ok && NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, rank, n_ids)) ws.rank[i] = rank;
}
// List slots and segments of every row; the rows of a block come in order, the blocks in any. A row of many
// segments is written by the whole block.
__global__ void __launch_bounds__(256) scatter_slots_kernel(ScatWs ws, int n_ids, int vocab) {
  nb::follow_grid();
  constexpr int FEW = 4;
  struct Row { int v, c, at, sg, h; };
  __shared__ unsigned long long wsum[8], wsum2[8];
  __shared__ int base_at, base_lt, base_sg, nmany;
  __shared__ Row many[256];
  if (threadIdx.x == 0) nmany = 0;                   // (the scan below has the barrier)
  const int v = blockIdx.x * 256 + threadIdx.x;
  const int c = v < vocab ? ws.counts[v] : 0;
  const bool light = c <= ws.light;
  const int k = light ? 0 : (c + SCAT_SEG - 1) / SCAT_SEG;
  const unsigned long long t = (unsigned long long)(c > 0 && light) << 32 | (unsigned)c;     // (light rows, entries)
  unsigned long long total, heavy = 0;
  const unsigned long long at0 = scatter_scan<8>(t, wsum, total) - t;
  if (total == 0) return;                            // the same in every thread
  const unsigned long long sg0 = scatter_scan<8>((unsigned)k, wsum2, heavy) - (unsigned)k;
  if (threadIdx.x == 0) {
    base_at = atomicAdd(ws.total, (int)(unsigned)total);
    base_lt = total >> 32 ? atomicAdd(ws.nlight, (int)(total >> 32)) : 0;
    base_sg = heavy ? atomicAdd(ws.nseg, (int)heavy) : 0;
  }
  __syncthreads();
  if (c && NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, base_at + (int)(unsigned)at0 + c - 1, n_ids)) {      // as many segments at most
    const int at = base_at + (int)(unsigned)at0, sg = base_sg + (int)sg0;
    ws.start[v] = at;
    const int h = k > 1 ? atomicAdd(ws.nheavy, k) : -1;
    if (light) {
      ws.seg[n_ids - 1 - (base_lt + (int)(at0 >> 32))] = make_int4(v, at, c, -1);
    } else if (k <= FEW) {
      for (int q = 0; q < k; ++q) ws.seg[sg + q] = scatter_segment(v, c, at, h, q);
    } else {
      many[atomicAdd(&nmany, 1)] = Row{v, c, at, sg, h};
    }
  }
  __syncthreads();
  for (int r = 0; r < nmany; ++r) {
    const Row w = many[r];
    for (int q = threadIdx.x; q < (w.c + SCAT_SEG - 1) / SCAT_SEG; q += 256) ws.seg[w.sg + q] = scatter_segment(w.v, w.c, w.at, w.h, q);
  }
}
__global__ void __launch_bounds__(256) scatter_place_kernel(const long long* __restrict__ ids, ScatWs ws, int n_ids, int vocab) {
  nb::follow_grid(ids);
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n_ids) return;
  const long long id = ids[i];
  if (id < 0 || id >= vocab) return;
  const int slot = ws.start[id] + ws.rank[i];
  if (NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, slot, n_ids)) ws.list[slot] = i;
}

// Columns [c, c + VN) of the fp32 sum of `n` rows of upd. SCAT_U rows are in flight: the rows lie anywhere, so
// each is a full memory latency.
constexpr int SCAT_U = 8;
template <typename T, int VN>
__device__ __forceinline__ void scatter_sum(const T* __restrict__ upd, const int* __restrict__ list, int n, size_t D, int c,
                                            int n_ids, float (&acc)[VN]) {
#pragma unroll
  for (int j = 0; j < VN; ++j) acc[j] = 0.f;
  for (int k = 0; k < n; k += SCAT_U) {
    uint4 raw[SCAT_U];
    T one[SCAT_U];
#pragma unroll
    for (int u = 0; u < SCAT_U; ++u) {
      if (k + u < n) {
        const int i = list[k + u];
        if (!NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, i, n_ids)) return;
        if (VN > 1) raw[u] = *reinterpret_cast<const uint4*>(upd + i * D + c);
        else one[u] = upd[i * D + c];
      }
    }
#pragma unroll
    for (int u = 0; u < SCAT_U; ++u) {
      if (k + u < n) {
        float v[VN];
        if constexpr (VN > 1) unpack_vec<T>(raw[u], v);
        else v[0] = to_f<T>(one[u]);
#pragma unroll
        for (int j = 0; j < VN; ++j) acc[j] += v[j];
      }
    }
  }
}
template <typename T, int VN>
__device__ __forceinline__ void scatter_write(const T* __restrict__ base, T* __restrict__ out, size_t at, float (&acc)[VN]) {
  if (base != nullptr) {
    float b[VN];
    if (VN > 1) load_vec<T>(base + at, b);
    else b[0] = to_f<T>(base[at]);
#pragma unroll
    for (int j = 0; j < VN; ++j) acc[j] += b[j];
  }
  if (VN > 1) store_vec<T>(out + at, acc);
  else out[at] = from_f<T>(acc[0]);
}
// Columns [c, c + VN) of the sum of `n` fp32 partial rows, `step` rows apart, from p on.
template <int VN>
__device__ __forceinline__ void scatter_join(const float* p, int n, size_t step, int c, float (&acc)[VN]) {
#pragma unroll
  for (int j = 0; j < VN; ++j) acc[j] = 0.f;
  constexpr int U = 8;                               // rows in flight
  int q = 0;
  if constexpr (VN > 1) {                            // rows are 16-byte aligned
    for (; q + U <= n; q += U) {
      float4 r[U][VN / 4];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < VN / 4; ++j) r[u][j] = __ldcg(reinterpret_cast<const float4*>(p + (q + u) * step + c) + j);
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < VN / 4; ++j) {
          acc[4 * j] += r[u][j].x; acc[4 * j + 1] += r[u][j].y; acc[4 * j + 2] += r[u][j].z; acc[4 * j + 3] += r[u][j].w;
        }
    }
  }
#pragma unroll 8
  for (; q < n; ++q)
#pragma unroll
    for (int j = 0; j < VN; ++j) acc[j] += __ldcg(p + q * step + c + j);
}
// A row of `n` <= R entries by one warp: R rows times SCAT_U / R vectors of each on their way per lane.
template <typename T, int VN, int R>
__device__ __forceinline__ void scatter_light(const T* __restrict__ upd, const T* __restrict__ base, T* __restrict__ out,
                                              const int* __restrict__ list, int n, size_t v, int D, int n_ids, int lane) {
  constexpr int CU = SCAT_U / R;
  const T* row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = list[r < n ? r : 0];
    if (!NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, i, n_ids)) return;
    row[r] = upd + (size_t)i * D;
  }
#pragma unroll 1
  for (int c0 = lane * VN; c0 < D; c0 += 32 * VN * CU) {
    uint4 raw[CU][R];
#pragma unroll
    for (int u = 0; u < CU; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int c = c0 + u * 32 * VN;
        raw[u][r] = make_uint4(0, 0, 0, 0);
        if (r < n && c < D) {
          if (VN > 1) raw[u][r] = *reinterpret_cast<const uint4*>(row[r] + c);
          else raw[u][r].x = __float_as_uint(to_f<T>(row[r][c]));
        }
      }
#pragma unroll
    for (int u = 0; u < CU; ++u) {
      const int c = c0 + u * 32 * VN;
      float acc[VN];
#pragma unroll
      for (int j = 0; j < VN; ++j) acc[j] = 0.f;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float x[VN];
        if constexpr (VN > 1) unpack_vec<T>(raw[u][r], x);
        else x[0] = __uint_as_float(raw[u][r].x);
#pragma unroll
        for (int j = 0; j < VN; ++j) acc[j] += x[j];
      }
      if (c < D) scatter_write<T, VN>(base, out, v * D + c, acc);
    }
  }
}
// Rows without an entry, one warp per SCAT_IDLE rows: zeros, or the base's row.
constexpr int SCAT_IDLE = 8;
template <typename T, int VN>
__device__ __forceinline__ void scatter_idle(const T* __restrict__ base, T* __restrict__ out, const int* __restrict__ counts,
                                             int vocab, size_t D, int warp, int nwarps, int lane) {
  for (int v0 = warp * SCAT_IDLE; v0 < vocab; v0 += nwarps * SCAT_IDLE) {
    const bool idle = lane < SCAT_IDLE && v0 + lane < vocab && counts[v0 + lane] == 0;
    for (unsigned m = __ballot_sync(0xffffffffu, idle); m; m &= m - 1) {
      const size_t at = (size_t)(v0 + __ffs(m) - 1) * D;
      if (base != nullptr) {
        constexpr int U = 8;                         // loads on their way per lane
        for (size_t c = lane * VN; c < D; c += 32 * VN * U) {
          if constexpr (VN > 1) {
            uint4 r[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (c + u * 32 * VN < D) r[u] = *reinterpret_cast<const uint4*>(base + at + c + u * 32 * VN);
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (c + u * 32 * VN < D) *reinterpret_cast<uint4*>(out + at + c + u * 32 * VN) = r[u];
          } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (c + u * 32 < D) out[at + c + u * 32] = base[at + c + u * 32];
          }
        }
      } else {
        for (size_t c = lane * VN; c < D; c += 32 * VN) {
          if (VN > 1) *reinterpret_cast<uint4*>(out + at + c) = make_uint4(0, 0, 0, 0);
          else out[at + c] = from_f<T>(0.f);
        }
      }
    }
    if (v0 > vocab - nwarps * SCAT_IDLE) break;      // (the next v0 may not fit an int)
  }
}
// ALL: every row of the table, once. The blocks walk the segments of crowded rows, the next descriptor on its way while one is
// worked on; then their warps the rows of few entries. Every other block writes its rows without an entry first, the rest
// last, so that stores and dependent loads run side by side. Else only the rows that occur, all of them by blocks, over a table that
// holds the base: what the other form does besides costs this one registers. VN: elements per access (16 bytes, or 1 where rows are
// not 16-byte aligned).
template <typename T, int VN, bool ALL>
__global__ void __launch_bounds__(256, VN == 8 ? 3 : 4) scatter_rows_kernel(const T* __restrict__ upd, const T* __restrict__ base,
                                                          T* __restrict__ out, ScatWs ws, float* __restrict__ part, int n_ids,
                                                          int D, int vocab) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS, upd, base, part);
  __shared__ int last;
  const int total = *ws.nseg, lights = ALL ? *ws.nlight : 0;
  const int lane = threadIdx.x & 31, nwarps = gridDim.x * (blockDim.x >> 5), warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lwarp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;         // few rows: spread over the blocks
  if (ALL && (blockIdx.x & 1)) scatter_idle<T, VN>(base, out, ws.counts, vocab, D, warp, nwarps, lane);
  int4 next = make_int4(0, 0, 0, -1);
  if ((int)blockIdx.x < total) next = ws.seg[blockIdx.x];
  for (int s = blockIdx.x; s < total; s += gridDim.x) {
    const int4 sg = next;
    if (s + (int)gridDim.x < total) next = ws.seg[s + gridDim.x];
    const int v = sg.x;
    if (!NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, sg.w < 0 ? 0 : sg.w, 2 * (n_ids / SCAT_SEG) + 1)) continue;   // partial row
    for (int c = threadIdx.x * VN; c < D; c += blockDim.x * VN) {
      float acc[VN];
      scatter_sum<T, VN>(upd, ws.list + sg.y, sg.z, D, c, n_ids, acc);
      if (sg.w < 0) {
        scatter_write<T, VN>(base, out, (size_t)v * D + c, acc);
      } else {
#pragma unroll
        for (int j = 0; j < VN; ++j) part[(size_t)sg.w * D + c + j] = acc[j];
      }
    }
    if (sg.w < 0) continue;
    const int nseg = (ws.counts[v] + SCAT_SEG - 1) / SCAT_SEG, ngroups = (nseg + SCAT_GROUP - 1) / SCAT_GROUP;
    const int q = (sg.y - ws.start[v]) / SCAT_SEG, h0 = sg.w - q, g0 = h0 + q / SCAT_GROUP * SCAT_GROUP;
    const int gsize = min(SCAT_GROUP, h0 + nseg - g0);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ws.gdone + g0, 1) == gsize - 1;
    __syncthreads();
    if (!last) continue;                             // the same in every thread
    __threadfence();
    float* grow = part + (size_t)g0 * D;
    for (int c = threadIdx.x * VN; c < D; c += blockDim.x * VN) {
      float acc[VN];
      scatter_join<VN>(grow, gsize, D, c, acc);
      if (ngroups == 1) {
        scatter_write<T, VN>(base, out, (size_t)v * D + c, acc);
      } else {
#pragma unroll
        for (int j = 0; j < VN; ++j) grow[c + j] = acc[j];       // this thread alone reads and writes these columns
      }
    }
    if (ngroups == 1) continue;
    __threadfence();
    __syncthreads();                                 // also: every thread has read `last`
    if (threadIdx.x == 0) last = atomicAdd(ws.done + v, 1) == ngroups - 1;
    __syncthreads();
    if (!last) continue;
    __threadfence();
    for (int c = threadIdx.x * VN; c < D; c += blockDim.x * VN) {
      float acc[VN];
      scatter_join<VN>(part + (size_t)h0 * D, ngroups, (size_t)SCAT_GROUP * D, c, acc);
      scatter_write<T, VN>(base, out, (size_t)v * D + c, acc);
    }
  }
  if (!ALL) return;
  const int4* lseg = ws.seg + n_ids - 1;
  int4 lnext = make_int4(0, 0, 0, -1);
  if (lwarp < lights) lnext = lseg[-lwarp];
  for (int s = lwarp; s < lights; s += nwarps) {
    const int4 sg = lnext;
    if (nwarps < lights - s) lnext = lseg[-(s + nwarps)];
    const int* list = ws.list + sg.y;
    if (sg.z == 1) scatter_light<T, VN, 1>(upd, base, out, list, 1, sg.x, D, n_ids, lane);
    else scatter_light<T, VN, SCAT_LIGHT>(upd, base, out, list, sg.z, sg.x, D, n_ids, lane);
    if (nwarps >= lights - s) break;
  }
  if (!(blockIdx.x & 1)) scatter_idle<T, VN>(base, out, ws.counts, vocab, D, warp, nwarps, lane);
}
// Small tables: acc[ids[i]] += upd[i] in an fp32 table that stays in L2, four columns per atomic (VEC).
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) embedding_scatter_add_kernel(float* __restrict__ acc, const long long* __restrict__ ids,
                                                                   const T* __restrict__ upd, int n_ids, int D, int vocab) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS, acc, ids, upd);
  const int i = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, i, n_ids)) return;   // debug build: one block per id
  const long long id = ids[i];
  if (id < 0 || id >= vocab) return;
  float* dst = acc + (size_t)id * D;
  const T* src = upd + (size_t)i * D;
  if constexpr (VEC) {
    for (int c = threadIdx.x * 4; c < D; c += blockDim.x * 4) {
      float4 v;
      if constexpr (sizeof(T) == 4) {
        v = *reinterpret_cast<const float4*>(src + c);
      } else {
        const uint2 w = *reinterpret_cast<const uint2*>(src + c);
        v = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                        __uint_as_float(w.y & 0xffff0000u));
      }
      atomicAdd(reinterpret_cast<float4*>(dst + c), v);
    }
  } else {
    for (int c = threadIdx.x; c < D; c += blockDim.x) atomicAdd(dst + c, to_f<T>(src[c]));
  }
}
// The same sum without atomics, for runs that must repeat bit for bit: the ids come sorted (stable,
// `perm[k]` = position of the k-th sorted id in the original order); the block at the head of each
// run of equal ids adds the run's rows in that order and writes base + sum.
template <typename T>
__global__ void __launch_bounds__(128) embedding_scatter_sorted_kernel(const long long* __restrict__ sorted_ids,
                                                                      const long long* __restrict__ perm,
                                                                      const T* __restrict__ upd, const T* __restrict__ base,
                                                                      T* __restrict__ out, int n_ids, int D, int vocab) {
  nb::follow_grid_when(gridDim.x <= nb::MANY_BLOCKS, sorted_ids, perm, upd, base);
  const int i = blockIdx.x;
  if (!NB_IN_BOUNDS(NB_SITE_ROW_INDEX, i, n_ids)) return;
  const long long id = sorted_ids[i];
  if (id < 0 || id >= vocab) return;
  if (i > 0 && sorted_ids[i - 1] == id) return;   // not the head of its run
  int end = i + 1;
  while (end < n_ids && sorted_ids[end] == id) ++end;
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    float acc = 0.f;
    for (int k = i; k < end; ++k) {
      const long long src = perm[k];
      if (!NB_IN_BOUNDS(NB_SITE_EMB_SCATTER_ID, src, n_ids)) continue;
      acc += to_f<T>(upd[(size_t)src * D + c]);
    }
    out[(size_t)id * D + c] = from_f<T>(to_f<T>(base[(size_t)id * D + c]) + acc);
  }
}
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) cast_kernel(const TI* __restrict__ in, TO* __restrict__ out, size_t n,
                                                  const TO* __restrict__ add_to) {
  nb::follow_grid(in, add_to);
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t k = i0; k < n; k += stride) {
    float v = to_f<TI>(in[k]);
    if (add_to) v += to_f<TO>(add_to[k]);
    out[k] = from_f<TO>(v);
  }
}

// ============================================================== activations
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_tanh_f(float x) {
  return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ float dgelu_f(float x) {
  return 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}
__device__ __forceinline__ float dgelu_tanh_f(float x) {
  const float x2 = x * x, u = 0.7978845608028654f * (x + 0.044715f * x * x2), t = tanhf(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * 0.7978845608028654f * (1.f + 3.f * 0.044715f * x2);
}
// mode: 0 relu, 1 gelu(erf), 2 gelu(tanh), 3 silu ; bwd: out = dy * act'(z)
template <typename T, bool BWD>
__global__ void __launch_bounds__(256) act_kernel(const T* __restrict__ z, const T* __restrict__ dy, T* __restrict__ out,
                                                 size_t n, int mode) {
  nb::follow_grid(z, dy);
  constexpr int V = Vec<T>::N;
  const size_t i0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * V;
  const size_t stride = (size_t)gridDim.x * blockDim.x * V;
  for (size_t i = i0; i < n; i += stride) {
    float zv[V], dv[V], o[V];
    if (i + V <= n) {
      load_vec<T>(z + i, zv);
      if (BWD) load_vec<T>(dy + i, dv);
    } else {
      for (int j = 0; j < V; ++j) {
        zv[j] = (i + j < n) ? to_f<T>(z[i + j]) : 0.f;
        dv[j] = (BWD && i + j < n) ? to_f<T>(dy[i + j]) : 0.f;
      }
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float x = zv[j];
      float r;
      if (!BWD) {
        r = mode == 0 ? fmaxf(x, 0.f) : mode == 1 ? gelu_f(x) : mode == 2 ? gelu_tanh_f(x) : x / (1.f + __expf(-x));
      } else {
        float d;
        if (mode == 0) d = x > 0.f ? 1.f : 0.f;
        else if (mode == 1) d = dgelu_f(x);
        else if (mode == 2) d = dgelu_tanh_f(x);
        else { const float sg = 1.f / (1.f + __expf(-x)); d = sg * (1.f + x * (1.f - sg)); }
        r = dv[j] * d;
      }
      o[j] = r;
    }
    if (i + V <= n) store_vec<T>(out + i, o);
    else for (int j = 0; j < V; ++j) if (i + j < n) out[i + j] = from_f<T>(o[j]);
  }
}

// ============================================================== Philox4x32-10 RNG
struct Philox {
  uint32_t key[2];
  uint32_t ctr[4];
  __device__ Philox(uint64_t seed, uint64_t subseq, uint64_t offset) {
    key[0] = (uint32_t)seed; key[1] = (uint32_t)(seed >> 32);
    ctr[0] = (uint32_t)offset; ctr[1] = (uint32_t)(offset >> 32);
    ctr[2] = (uint32_t)subseq; ctr[3] = (uint32_t)(subseq >> 32);
  }
  __device__ uint4 next() {
    uint32_t c0 = ctr[0], c1 = ctr[1], c2 = ctr[2], c3 = ctr[3], k0 = key[0], k1 = key[1];
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
      const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
      const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
      c0 = n0; c1 = n1; c2 = n2; c3 = n3;
      k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    if (++ctr[0] == 0) ++ctr[1];
    return make_uint4(c0, c1, c2, c3);
  }
};
__device__ __forceinline__ float u01(uint32_t x) { return ((x >> 8) + 0.5f) * (1.0f / 16777216.0f); }

// Random streams. With `state` (device memory: [0] seed, [1] number of draws made so far on this
// device) the Philox key and offset come from there and `seed` is only a salt that tells the shards
// of one tensor apart; the launcher advances state[1] with a one-thread kernel afterwards. Because
// the kernel reads the state when it RUNS, a launch replayed from a CUDA graph draws fresh numbers
// every time (reference: the seed threaded graph-in -> graph-out, nabla/core/graph/engine.py:80-88).
__device__ __forceinline__ void rng_resolve(const unsigned long long* state, uint64_t& seed, uint64_t& offset) {
  if (state != nullptr) {
    seed = state[0] * 1000003ull + seed;
    offset = state[1] << 32;
  }
}
__global__ void rng_bump_kernel(unsigned long long* state) {
  nb::follow_grid(state); state[1] += 1ull; }

// mode 0: uniform in [a, b); mode 1: gaussian mean a std b
template <typename T>
__global__ void __launch_bounds__(256) rng_kernel(T* __restrict__ out, size_t n, uint64_t seed, uint64_t offset,
                                                 int mode, float a, float b, const unsigned long long* state) {
  nb::follow_grid(state);
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nthreads = (size_t)gridDim.x * blockDim.x;
  rng_resolve(state, seed, offset);
  Philox ph(seed, tid, offset);
  for (size_t i = tid * 4; i < n; i += nthreads * 4) {
    const uint4 r = ph.next();
    float f[4];
    if (mode == 0) {
      f[0] = a + (b - a) * u01(r.x); f[1] = a + (b - a) * u01(r.y);
      f[2] = a + (b - a) * u01(r.z); f[3] = a + (b - a) * u01(r.w);
    } else {
      const float r1 = sqrtf(-2.f * logf(u01(r.x))), t1 = 6.283185307179586f * u01(r.y);
      const float r2 = sqrtf(-2.f * logf(u01(r.z))), t2 = 6.283185307179586f * u01(r.w);
      f[0] = a + b * r1 * cosf(t1); f[1] = a + b * r1 * sinf(t1);
      f[2] = a + b * r2 * cosf(t2); f[3] = a + b * r2 * sinf(t2);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) if (i + j < n) out[i + j] = from_f<T>(f[j]);
  }
}
// y = x * mask / (1-p); mask (uint8) kept for the backward
template <typename T>
__global__ void __launch_bounds__(256) dropout_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                     uint8_t* __restrict__ mask, size_t n, float p, uint64_t seed,
                                                     uint64_t offset, const unsigned long long* state) {
  nb::follow_grid(x, state);
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nthreads = (size_t)gridDim.x * blockDim.x;
  rng_resolve(state, seed, offset);
  Philox ph(seed, tid, offset);
  const float keep_scale = 1.f / (1.f - p);
  for (size_t i = tid * 4; i < n; i += nthreads * 4) {
    const uint4 r = ph.next();
    const float u[4] = {u01(r.x), u01(r.y), u01(r.z), u01(r.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i + j < n) {
        const bool keep = u[j] >= p;
        mask[i + j] = keep ? 1 : 0;
        y[i + j] = from_f<T>(keep ? to_f<T>(x[i + j]) * keep_scale : 0.f);
      }
    }
  }
}

// ============================================================== NF4 dequantisation
// packed: 2 codes per byte (high nibble first); absmax per block of `block` elements.
__constant__ float NF4_CODE[16] = {-1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f,
                                   -0.28444138169288635f, -0.18477343022823334f, -0.09105003625154495f, 0.0f,
                                   0.07958029955625534f, 0.16093020141124725f, 0.24611230194568634f,
                                   0.33791524171829224f, 0.44070982933044434f, 0.5626170039176941f,
                                   0.7229568362236023f, 1.0f};
template <typename T>
__global__ void __launch_bounds__(256) nf4_dequant_kernel(const uint8_t* __restrict__ packed,
                                                         const float* __restrict__ absmax, T* __restrict__ out,
                                                         size_t n, int block) {
  nb::follow_grid(packed, absmax);
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t b = i0; b * 2 < n; b += stride) {
    const uint8_t byte = packed[b];
    const size_t e0 = b * 2;
    out[e0] = from_f<T>(NF4_CODE[byte >> 4] * absmax[e0 / block]);
    if (e0 + 1 < n) out[e0 + 1] = from_f<T>(NF4_CODE[byte & 15] * absmax[(e0 + 1) / block]);
  }
}

// One code per byte (the layout of the QLoRA weight dict: `indices` uint8 [padded_numel], `scales`
// fp32 per block) and the 16-entry codebook passed by the caller. 16 codes per thread: one 16-byte load of
// codes and, where the scale blocks are whole multiples of 16 codes (WHOLE), one scale; the results leave as
// 16-byte stores. A 64-bit division and a 2- or 4-byte store per element, as it was before, bound the kernel
// by instructions instead of the 1 + sizeof(T) bytes per weight that it has to move: 2048 x 6144 to bf16 in blocks
// of 64 took 74 us, now 9 (4.3 TB/s).
template <typename T, bool WHOLE>
__global__ void __launch_bounds__(256) nf4_dequant_codes_kernel(const uint8_t* __restrict__ codes,
                                                               const float* __restrict__ absmax,
                                                               const float* __restrict__ codebook, T* __restrict__ out,
                                                               size_t n, int block) {
  nb::follow_grid(codes, absmax, codebook);
  __shared__ float cb[16];
  if (threadIdx.x < 16) cb[threadIdx.x] = codebook[threadIdx.x];
  __syncthreads();
  const size_t stride = (size_t)gridDim.x * blockDim.x * 16;
  for (size_t i0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 16; i0 < n; i0 += stride) {
    if (WHOLE && i0 + 16 <= n) {
      const uint4 raw = *reinterpret_cast<const uint4*>(codes + i0);
      const float scale = absmax[i0 <= 0xffffffffull ? (size_t)((unsigned)i0 / (unsigned)block) : i0 / block];
      const unsigned w[4] = {raw.x, raw.y, raw.z, raw.w};
      float o[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] = cb[(w[j >> 2] >> (8 * (j & 3))) & 15] * scale;
#pragma unroll
      for (int j = 0; j < 16; j += Vec<T>::N) store_vec<T>(out + i0 + j, o + j);
    } else if constexpr (WHOLE) {                    // the last codes
      for (int j = 0; j < 16; ++j)
        if (i0 + j < n) out[i0 + j] = from_f<T>(cb[codes[i0 + j] & 15] * absmax[(i0 + j) / block]);
    } else {
      // any block size and alignment: one division per thread, then the scale moves on where a block ends
      size_t b = i0 / block;
      int left = block - (int)(i0 - b * block);
      float scale = absmax[b];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (i0 + j < n) {
          if (left == 0) {
            if (!NB_IN_BOUNDS(NB_SITE_NF4_BLOCK, b + 1, (n + block - 1) / block)) return;
            scale = absmax[++b];
            left = block;
          }
          out[i0 + j] = from_f<T>(cb[codes[i0 + j] & 15] * scale);
          --left;
        }
      }
    }
  }
}

// ============================================================== pooling (NHWC)
// mode 0 avg, 1 max. Backward: avg spreads dy/(kh*kw); max routes to the first arg-max.
template <typename T>
__global__ void __launch_bounds__(256) pool2d_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int N, int H, int W,
                                                        int C, int OH, int OW, int kh, int kw, int sh, int sw, int ph,
                                                        int pw, int mode) {
  nb::follow_grid(x);
  const size_t total = (size_t)N * OH * OW * C;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    size_t r = i / C;
    const int ow = r % OW; r /= OW;
    const int oh = r % OH;
    const int n = r / OH;
    float acc = mode == 0 ? 0.f : -INFINITY;
    for (int a = 0; a < kh; ++a)
      for (int b = 0; b < kw; ++b) {
        const int ih = oh * sh - ph + a, iw = ow * sw - pw + b;
        float v = mode == 0 ? 0.f : -INFINITY;
        if (ih >= 0 && ih < H && iw >= 0 && iw < W) v = to_f<T>(x[(((size_t)n * H + ih) * W + iw) * C + c]);
        acc = mode == 0 ? acc + v : fmaxf(acc, v);
      }
    y[i] = from_f<T>(mode == 0 ? acc / (kh * kw) : acc);
  }
}
// Pooling whose windows do not overlap and lie in the image (kernel <= stride, no padding: the usual 2 x 2), C a
// multiple of the 16-byte vector: one thread per vector of channels of a stride x stride cell. Forward: the
// window's elements are read once. Backward: so are x and dy, and the cell's dx is written whole, zeros where
// no window reaches (the gather form below finds every window's arg-max again for each of its pixels, with
// six 64-bit divisions per element). Same values, first arg-max included. 2 x 2 over 256 x 28 x 28 x 16 fp32:
// forward 10 -> 3.6 us, backward 52 -> 5.4 us. A thread walks its cell alone, so large cells leave few threads.
// Forward and max backward are faster all the same (the gather forms walk the window too, the latter once per
// pixel: 8 x 56 x 56 x 64 in one window fp32 1.25 -> 0.45 ms and 6.2 -> 0.94 ms), but average backward has only one
// load per pixel to do there and keeps the gather form where cells of more than 9 pixels times channels are below
// 8192: that image 20 us by pixels, 108 by cells (512 cells); 1 x 256 x 256 x 16 in 16 x 16 18 and 23 (4096); 64 x 14 x 14 x
// 256 in one window each 35 and 19 (16384).
struct CellGeom {
  int N, H, W, CV, OH, OW, kh, kw, sh, sw, cells_h, cells_w;
};
template <typename T, bool MAX>
__global__ void __launch_bounds__(256) pool2d_cell_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, const CellGeom g, unsigned total) {
  nb::follow_grid(x);
  constexpr int V = Vec<T>::N;
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= total) return;
  const unsigned c = i % g.CV, p = i / g.CV, ow = p % g.OW, q = p / g.OW, oh = q % g.OH, n = q / g.OH;
  const size_t at = (((size_t)n * g.H + oh * g.sh) * g.W + ow * g.sw) * g.CV * V + c * V;
  if (!NB_IN_BOUNDS(NB_SITE_POOL_INPUT, at + ((size_t)(g.kh - 1) * g.W + g.kw - 1) * g.CV * V + V - 1, (size_t)g.N * g.H * g.W * g.CV * V))
    return;
  const T* xp = x + at;
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = MAX ? -INFINITY : 0.f;
  for (int a = 0; a < g.kh; ++a)
    for (int b = 0; b < g.kw; ++b) {
      float v[V];
      load_vec<T>(xp + ((size_t)a * g.W + b) * g.CV * V, v);
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] = MAX ? fmaxf(acc[j], v[j]) : acc[j] + v[j];
    }
  if (!MAX) {
#pragma unroll
    for (int j = 0; j < V; ++j) acc[j] /= g.kh * g.kw;
  }
  store_vec<T>(y + (size_t)i * V, acc);
}
// RELU: x came out of a relu, and its derivative is applied too (what reaches a maximum of 0 or less is multiplied by 0). As a pass of its
// own it read and wrote all of x's size: 256 x 28 x 28 x 16 fp32 5.4 + 4.7 us, 5.7 so.
template <typename T, bool MAX, bool RELU = false>
__global__ void __launch_bounds__(256) pool2d_cell_bwd_kernel(const T* __restrict__ x, const T* __restrict__ dy, T* __restrict__ dx,
                                                             const CellGeom g, unsigned total) {
  nb::follow_grid(x, dy);
  constexpr int V = Vec<T>::N;
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= total) return;
  const unsigned c = i % g.CV, p = i / g.CV, cw = p % g.cells_w, q = p / g.cells_w, ch = q % g.cells_h, n = q / g.cells_h;
  const size_t at = (((size_t)n * g.H + ch * g.sh) * g.W + cw * g.sw) * g.CV * V + c * V, down = (size_t)g.W * g.CV * V;
  const bool window = (int)ch < g.OH && (int)cw < g.OW;
  const int hh = min(g.sh, g.H - (int)ch * g.sh), ww = min(g.sw, g.W - (int)cw * g.sw);      // the cell's part of the image
  if (!NB_IN_BOUNDS(NB_SITE_POOL_INPUT, at + (hh - 1) * down + (size_t)(ww - 1) * g.CV * V + V - 1, (size_t)g.N * g.H * g.W * g.CV * V) ||
      (window && !NB_IN_BOUNDS(NB_SITE_POOL_INPUT, ((((size_t)n * g.OH + ch) * g.OW + cw) * g.CV + c) * V + V - 1,
                               (size_t)g.N * g.OH * g.OW * g.CV * V)))
    return;
  float d[V], best[V];
  int where[V];                                      // position of the first maximum in the window, -1: none
#pragma unroll
  for (int j = 0; j < V; ++j) { d[j] = 0.f; best[j] = -INFINITY; where[j] = -1; }
  if (window) {
    load_vec<T>(dy + (((size_t)n * g.OH + ch) * g.OW + cw) * g.CV * V + c * V, d);
    if (MAX) {
      for (int a = 0; a < g.kh; ++a)
        for (int b = 0; b < g.kw; ++b) {
          float v[V];
          load_vec<T>(x + at + a * down + (size_t)b * g.CV * V, v);
#pragma unroll
          for (int j = 0; j < V; ++j)
            if (v[j] > best[j]) { best[j] = v[j]; where[j] = a * g.kw + b; }
        }
    }
  }
  if (RELU) {
#pragma unroll
    for (int j = 0; j < V; ++j) d[j] *= best[j] > 0.f ? 1.f : 0.f;
  }
  const float inv = 1.f / (g.kh * g.kw);
  for (int a = 0; a < hh; ++a)
    for (int b = 0; b < ww; ++b) {
      const bool in = window && a < g.kh && b < g.kw;
      float o[V];
#pragma unroll
      for (int j = 0; j < V; ++j) o[j] = !in ? 0.f : MAX ? (where[j] == a * g.kw + b ? d[j] : 0.f) : d[j] * inv;
      store_vec<T>(dx + at + a * down + (size_t)b * g.CV * V, o);
    }
}
// Whether the two kernels above can take a problem.
static inline bool pool_cells(const void* x, const void* y, const void* z, int N, int H, int W, int C, int OH, int OW, int kh, int kw,
                              int sh, int sw, int ph, int pw, int V, CellGeom& g) {
  g = CellGeom{N, H, W, C / V, OH, OW, kh, kw, sh, sw, (H + sh - 1) / sh, (W + sw - 1) / sw};
  return ph == 0 && pw == 0 && kh <= sh && kw <= sw && C % V == 0 && (long long)N * g.cells_h * g.cells_w * g.CV < 0x7fffff00ll &&
         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z)) & 15) == 0;
}
static inline bool pool_cells_avg_bwd(int N, int C, const CellGeom& g) {
  return (long long)(g.sh < g.H ? g.sh : g.H) * (g.sw < g.W ? g.sw : g.W) <= 9 || (long long)N * g.cells_h * g.cells_w * C >= 8192;
}

// out[window] = t[first arg-max of x over the window] (0 for a window that lies in the padding): the
// forward-mode derivative of max pooling, and the transpose of its backward routing.
template <typename T>
__global__ void __launch_bounds__(256) pool2d_select_kernel(const T* __restrict__ x, const T* __restrict__ t,
                                                           T* __restrict__ y, int N, int H, int W, int C, int OH, int OW,
                                                           int kh, int kw, int sh, int sw, int ph, int pw) {
  nb::follow_grid(x, t);
  const size_t total = (size_t)N * OH * OW * C;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    size_t r = i / C;
    const int ow = r % OW; r /= OW;
    const int oh = r % OH;
    const int n = r / OH;
    float best = -INFINITY;
    size_t at = 0;
    bool found = false;
    for (int a = 0; a < kh; ++a)
      for (int b = 0; b < kw; ++b) {
        const int ih = oh * sh - ph + a, iw = ow * sw - pw + b;
        if (ih >= 0 && ih < H && iw >= 0 && iw < W) {
          const size_t off = (((size_t)n * H + ih) * W + iw) * C + c;
          const float v = to_f<T>(x[off]);
          if (v > best || !found) { best = v; at = off; found = true; }
        }
      }
    y[i] = found ? t[at] : from_f<T>(0.f);
  }
}

// Backward in gather form: one thread per input pixel sums over the windows that cover it (for max
// pooling it finds each window's first arg-max again and takes the gradient when that is this
// pixel). No atomics, so the result does not depend on the order in which blocks run, and dx needs
// no zero fill and no fp32 staging.
template <typename T>
__global__ void __launch_bounds__(256) pool2d_bwd_kernel(const T* __restrict__ x, const T* __restrict__ dy,
                                                        T* __restrict__ dx, int N, int H, int W, int C, int OH,
                                                        int OW, int kh, int kw, int sh, int sw, int ph, int pw, int mode, int relu) {
  nb::follow_grid(x, dy);
  const size_t total = (size_t)N * H * W * C;
  const float inv = 1.f / (kh * kw);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int c = i % C;
    size_t r = i / C;
    const int iw = r % W; r /= W;
    const int ih = r % H;
    const int n = r / H;
    // windows (oh, ow) with oh*sh - ph <= ih < oh*sh - ph + kh, likewise for the width
    const int th = ih + ph - kh + 1, tw = iw + pw - kw + 1;
    const int oh_lo = th > 0 ? (th + sh - 1) / sh : 0, oh_hi = min(OH - 1, (ih + ph) / sh);
    const int ow_lo = tw > 0 ? (tw + sw - 1) / sw : 0, ow_hi = min(OW - 1, (iw + pw) / sw);
    float acc = 0.f;
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        const size_t yo = (((size_t)n * OH + oh) * OW + ow) * C + c;
        if (!NB_IN_BOUNDS(NB_SITE_POOL_INPUT, yo, (size_t)N * OH * OW * C)) continue;
        const float g = to_f<T>(dy[yo]);
        if (mode == 0) {
          acc += g * inv;
        } else {
          float best = -INFINITY;
          int bh = -1, bw = -1;
          for (int a = 0; a < kh; ++a)
            for (int b = 0; b < kw; ++b) {
              const int jh = oh * sh - ph + a, jw = ow * sw - pw + b;
              if (jh >= 0 && jh < H && jw >= 0 && jw < W) {
                const float v = to_f<T>(x[(((size_t)n * H + jh) * W + jw) * C + c]);
                if (v > best) { best = v; bh = jh; bw = jw; }
              }
            }
          if (bh == ih && bw == iw) acc += g;
        }
      }
    dx[i] = from_f<T>(relu ? acc * (to_f<T>(x[i]) > 0.f ? 1.f : 0.f) : acc);
  }
}

// ============================================================== direct conv2d NHWC x RSCF (small C)
// y[n,oh,ow,f] = sum_{r,s,c} x[n, oh*sh - pt + r, ow*sw - pl + s, c] * w[r,s,c,f] (+ bias[f])
//
// An implicit matrix product over k = (r, s, c) in fp32 FMAs: a block owns 2 * PG output positions and
// 4 * FG channels, each thread a 2 x 4 tile of them. CONV_KC values of k are staged at a time (the gathered
// input and the filter rows, as floats), so a thread does 8 FMAs for two shared loads; one thread per
// output value with both operands from global memory was bound by its two loads per FMA. (A 4 x 4 tile
// leaves too few warps: 50,000 threads for 256 images of 14 x 14 x 16.)
// Measured (fp32, 3x3): 256 x 28 x 28 x 1 -> 16 83 -> 19 us, 256 x 14 x 14 x 16 -> 32 133 -> 38 us; still some
// five times its FMAs' time, which goes to staging the gathered input.
// The terms are added in the same order (bias, then k ascending), so fp32 results are unchanged.
// A padded position counts as absent, not as 0 * w: where the staged filter holds an infinity or a NaN
// the block falls back to conv_point, which skips such positions.
struct ConvGeom {
  int N, H, W, C, R, S, F, OH, OW, sh, sw, pt, pl;
};

// The filter of an input gradient: out[r][s][f][c] = w[R - 1 - r][S - 1 - s][c][f].
template <typename T>
__global__ void __launch_bounds__(256) conv_flip_kernel(const T* __restrict__ w, T* __restrict__ out, int taps, int C, int F, unsigned n) {
  nb::follow_grid(w);
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= n || !NB_IN_BOUNDS(NB_SITE_FLAT_INDEX, i, n)) return;
  const unsigned c = i % C, q = i / C, f = q % F, t = q / F;
  out[i] = w[((size_t)(taps - 1 - t) * C + c) * F + f];
}

template <typename T>
__device__ __noinline__ float conv_point(const T* __restrict__ x, const T* __restrict__ w, float acc, const ConvGeom g,
                                         long long m, int f) {
  const int ow = (int)(m % g.OW);
  const long long q = m / g.OW;
  const int oh = (int)(q % g.OH), n = (int)(q / g.OH);
  for (int r = 0; r < g.R; ++r) {
    const int ih = oh * g.sh - g.pt + r;
    if (ih < 0 || ih >= g.H) continue;
    for (int s = 0; s < g.S; ++s) {
      const int iw = ow * g.sw - g.pl + s;
      if (iw < 0 || iw >= g.W) continue;
      if (!NB_IN_BOUNDS(NB_SITE_CONV_INPUT, (((size_t)n * g.H + ih) * g.W + iw) * g.C, (size_t)g.N * g.H * g.W * g.C)) continue;
      const T* xp = x + (((size_t)n * g.H + ih) * g.W + iw) * g.C;
      const T* wp = w + ((size_t)(r * g.S + s) * g.C) * g.F + f;
      for (int c = 0; c < g.C; ++c) acc = fmaf(to_f<T>(xp[c]), to_f<T>(wp[(size_t)c * g.F]), acc);
    }
  }
  return acc;
}

// Four consecutive elements (16 bytes of fp32, 8 of bf16).
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 r = *reinterpret_cast<const float4*>(p);
  v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 r = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xffff0000u);
  v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xffff0000u);
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(bf16* p, const float (&v)[4]) {
  const __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
  *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(h);
}

constexpr int CONV_KC = 32;      // values of k staged at a time

// Filter tap k = (r, s, c) and its offset from the first pixel of a window, 16 bytes. The offset is
// 64 bits wide: r * W * C may pass 2^31 where the image is large, or low but padded to a tall filter.
struct __align__(16) ConvTap {
  int r, s;
  long long off;
};
__device__ __forceinline__ ConvTap conv_tap(int k, const ConvGeom& g) {
  const int rs = k / g.C, r = rs / g.S, s = rs - r * g.S;
  return ConvTap{r, s, ((long long)r * g.W + s) * g.C + (k - rs * g.C)};
}

// relu: below 0 becomes 0, NaN stays.
template <typename T, int FG, bool VEC>
__global__ void __launch_bounds__(128) conv2d_direct_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                           const T* __restrict__ bias, T* __restrict__ y, const ConvGeom g, int relu) {
  nb::follow_grid(x, w, bias);
  constexpr int PG = 128 / FG, MT = 2 * PG, FT = 4 * FG, PER = (MT + 127) / 128, KSTEP = MT < 128 ? 128 / MT : 1;
  __shared__ __align__(16) float xs[CONV_KC][MT + 4];
  __shared__ __align__(16) float ws[CONV_KC][FT];
  __shared__ ConvTap taps[CONV_KC];
  const int tid = threadIdx.x;
  const long long positions = (long long)g.N * g.OH * g.OW;
  const long long m0 = (long long)blockIdx.x * MT;
  // channel tile; a grid holds 65535 in y, more go on in z
  if ((blockIdx.z * 65535ll + blockIdx.y) * FT >= g.F) return;
  const int f0 = (blockIdx.z * 65535 + blockIdx.y) * FT;
  const int K = g.R * g.S * g.C;
  // the positions whose input this thread stages
  int ih0[PER], iw0[PER];
  long long base[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const long long m = m0 + (tid % (MT < 128 ? MT : 128)) + j * 128;
    ih0[j] = -0x40000000;                            // a position past the end: every row of its window is out of range
    iw0[j] = 0;
    base[j] = 0;
    if (m < positions) {
      const int ow = (int)(m % g.OW);
      const long long q = m / g.OW;
      const int oh = (int)(q % g.OH);
      ih0[j] = oh * g.sh - g.pt;
      iw0[j] = ow * g.sw - g.pl;
      base[j] = (((q / g.OH) * g.H + ih0[j]) * g.W + iw0[j]) * g.C;
    }
  }
  const int fg = tid % FG, pg = tid / FG;
  float acc[2][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int f = f0 + fg * 4 + j;
    const float b = bias && f < g.F ? to_f<T>(bias[f]) : 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) acc[i][j] = b;
  }
  int odd = 0;                                       // a filter value that is not finite was staged
  for (int k0 = 0; k0 < K; k0 += CONV_KC) {
    const int kn = min(CONV_KC, K - k0);
    __syncthreads();
    if (tid < kn) taps[tid] = conv_tap(k0 + tid, g);
    for (int e = tid; e < kn * FT; e += 128) {
      const int k = e / FT, f = f0 + e % FT;
      const float v = f < g.F ? to_f<T>(w[(size_t)(k0 + k) * g.F + f]) : 0.f;
      odd |= !isfinite(v);
      ws[k][e % FT] = v;
    }
    __syncthreads();
    constexpr int KV = VEC ? 4 : 1;                  // VEC (C % 4 == 0): four channels of one pixel per load
#pragma unroll 8
    for (int k = (MT < 128 ? tid / MT : 0) * KV; k < kn; k += KSTEP * KV) {
      const ConvTap tap = taps[k];
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int ih = ih0[j] + tap.r, iw = iw0[j] + tap.s;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W &&
            NB_IN_BOUNDS(NB_SITE_CONV_INPUT, base[j] + tap.off + KV - 1, (long long)g.N * g.H * g.W * g.C)) {
          if (VEC) load4(x + base[j] + tap.off, v);
          else v[0] = to_f<T>(x[base[j] + tap.off]);
        }
#pragma unroll
        for (int i = 0; i < KV; ++i) xs[k + i][(tid % (MT < 128 ? MT : 128)) + j * 128] = v[i];
      }
    }
    __syncthreads();
    auto step = [&](int k) {
      const float2 a = *reinterpret_cast<const float2*>(&xs[k][pg * 2]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[k][fg * 4]);
      const float av[2] = {a.x, a.y}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    };
    if (kn == CONV_KC) {
#pragma unroll 8
      for (int k = 0; k < CONV_KC; ++k) step(k);
    } else {
      for (int k = 0; k < kn; ++k) step(k);
    }
  }
  odd = __syncthreads_or(odd);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const long long m = m0 + pg * 2 + i;
    if (m >= positions) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int f = f0 + fg * 4 + j;
      if (f >= g.F) break;
      if (odd) acc[i][j] = conv_point<T>(x, w, bias ? to_f<T>(bias[f]) : 0.f, g, m, f);
      if (relu && acc[i][j] < 0.f) acc[i][j] = 0.f;
      y[m * g.F + f] = from_f<T>(acc[i][j]);
    }
  }
}

// Input patch of `rows` x pw pixels whose first is (ih0, iw0) of an image, nq groups of KV channels from group q0 on, to xs as
// [nq][rows][pw] of KV floats; zeros outside the image. The coordinates of a thread's next pixel follow from those of the last (two divisions per value took as long
// as the loads).
template <typename T, bool VEC>
__device__ __forceinline__ void stage_patch(const T* __restrict__ image, float* __restrict__ xs, const ConvGeom& g, int n, int ih0,
                                            int iw0, int rows, int pw, int q0, int nq) {
  constexpr int KV = VEC ? 4 : 1;
  const int plane = rows * pw, step = 128 / nq, dq = 128 - step * nq, dr = step / pw, dc = step - dr * pw;
  int pix = threadIdx.x / nq, q = threadIdx.x - pix * nq, pr = pix / pw, pc = pix - pr * pw;
#pragma unroll 4
  while (pix < plane) {
    const int ih = ih0 + pr, iw = iw0 + pc;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W && NB_IN_BOUNDS(NB_SITE_CONV_INPUT, n, g.N)) {
      const T* p = image + ((size_t)ih * g.W + iw) * g.C + (q0 + q) * KV;
      if (VEC) load4(p, v);
      else v[0] = to_f<T>(*p);
    }
    if (VEC) *reinterpret_cast<float4*>(xs + (q * plane + pix) * 4) = make_float4(v[0], v[1], v[2], v[3]);
    else xs[q * plane + pix] = v[0];
    const int carry = q + dq >= nq;
    q += dq - carry * nq;
    pix += step + carry;
    pc += dc + carry;
    pr += dr;
    if (pc >= pw) { pc -= pw; ++pr; }
  }
}

// The same sums from a patch: a block stages the input of TH rows of one image's output once, with its halo, and the whole
// filter tile, and walks (r, s, c) by addresses, where the kernel above stages every input value once per filter tap. A
// thread has PX positions and 4 channels, the FG channel groups of a position in neighbouring lanes: a warp's loads of input are then
// few distinct 16-byte pieces, its stores whole rows, and PX + 4 wavefronts serve 16 PX FMAs (with consecutive positions in
// neighbouring lanes 2 PX + 4 and half-used sectors: 71 % of the shared-memory pipe). The FMAs go two channels at a time. VEC: four
// input channels per shared load, kept as float4 planes. The additions are those of the kernel above, in its order: the same bits.
// Bound by the staging, which all blocks do at the same time, and then by issue; 128 registers, so that 512 blocks run at once. us, tiled,
// from patches with positions in neighbouring lanes, and so, fp32, 3 x 3: 256 x 14 x 14 x 16 -> 32 28.8, 23.7, 20.9; 256 x 14 x 14 x 32 -> 16
// (an input gradient) 40.2, 25.5, 22.5; 256 x 28 x 28 x 1 -> 16 14.0, 13.1, 11.2.
template <typename T, int FG, int PX, bool VEC>
__global__ void __launch_bounds__(128, 4) conv2d_patch_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                          const T* __restrict__ bias, T* __restrict__ y, const ConvGeom g,
                                                          int TH, int bands, int wvec, int yvec, int relu) {
  nb::follow_grid(x, w, bias);
  constexpr int PG = 128 / FG, FT = 4 * FG, KV = VEC ? 4 : 1;
  extern __shared__ __align__(16) float conv_smem[];
  const int tid = threadIdx.x, K = g.R * g.S * g.C, CQ = g.C / KV;
  const int pw = (g.OW - 1) * g.sw + g.S, ph = (TH - 1) * g.sh + g.R, plane = pw * ph;
  float* ws = conv_smem;                             // [K][FT]
  float* xs = conv_smem + K * FT;                    // [CQ][ph][pw] of KV floats
  const int n = blockIdx.x / bands, oh0 = (blockIdx.x - n * bands) * TH, f0 = blockIdx.y * FT;
  int odd = 0;                                       // a filter value that is not finite was staged
  if (wvec) {
#pragma unroll 4
    for (int e = tid; e < K * (FT / 4); e += 128) {
      const int f = f0 + e % (FT / 4) * 4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (f < g.F) load4(w + (size_t)(e / (FT / 4)) * g.F + f, v);
      odd |= !isfinite(v[0]) | !isfinite(v[1]) | !isfinite(v[2]) | !isfinite(v[3]);
      *reinterpret_cast<float4*>(ws + e * 4) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
#pragma unroll 4
    for (int e = tid; e < K * FT; e += 128) {
      const int f = f0 + e % FT;
      const float v = f < g.F ? to_f<T>(w[(size_t)(e / FT) * g.F + f]) : 0.f;
      odd |= !isfinite(v);
      ws[e] = v;
    }
  }
  stage_patch<T, VEC>(x + (size_t)n * g.H * g.W * g.C, xs, g, n, oh0 * g.sh - g.pt, -g.pl, ph, pw, 0, CQ);
  const int fg = tid % FG, pg = tid / FG;
  int at[PX];
  float2 acc[PX][2];                                 // four channels in two pairs
#pragma unroll
  for (int i = 0; i < PX; ++i) {
    const int p = pg + i * PG, r = p / g.OW, c = p - r * g.OW;
    at[i] = r < TH ? r * g.sh * pw + c * g.sw : 0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int f = f0 + fg * 4 + 2 * j;
      acc[i][j] = make_float2(bias && f < g.F ? to_f<T>(bias[f]) : 0.f, bias && f + 1 < g.F ? to_f<T>(bias[f + 1]) : 0.f);
    }
  }
  __syncthreads();
  const float* wp = ws + fg * 4;
  for (int r = 0; r < g.R; ++r)
    for (int s = 0; s < g.S; ++s)
      for (int q = 0; q < CQ; ++q) {
        const float* xp = xs + (q * plane + r * pw + s) * KV;
        float a[PX][KV];
#pragma unroll
        for (int i = 0; i < PX; ++i) {
          if constexpr (VEC) {
            const float4 t = *reinterpret_cast<const float4*>(xp + at[i] * 4);
            a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w;
          } else {
            a[i][0] = xp[at[i]];
          }
        }
#pragma unroll
        for (int k = 0; k < KV; ++k) {
          const float4 b = *reinterpret_cast<const float4*>(wp);
          wp += FT;
#pragma unroll
          for (int i = 0; i < PX; ++i) {
            const float2 t = make_float2(a[i][k], a[i][k]);
            acc[i][0] = __ffma2_rn(t, make_float2(b.x, b.y), acc[i][0]);
            acc[i][1] = __ffma2_rn(t, make_float2(b.z, b.w), acc[i][1]);
          }
        }
      }
  odd = __syncthreads_or(odd);
#pragma unroll
  for (int i = 0; i < PX; ++i) {
    const int p = pg + i * PG, r = p / g.OW, c = p - r * g.OW, oh = oh0 + r, f = f0 + fg * 4;
    if (r >= TH || oh >= g.OH || f >= g.F) continue;
    const long long m = ((long long)n * g.OH + oh) * g.OW + c;
    float v[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
    if (odd) {
      for (int j = 0; j < 4 && f + j < g.F; ++j) v[j] = conv_point<T>(x, w, bias ? to_f<T>(bias[f + j]) : 0.f, g, m, f + j);
    }
    if (relu) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v[j] < 0.f) v[j] = 0.f;
    }
    T* o = y + m * g.F + f;
    if (yvec) {
      store4(o, v);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (f + j < g.F) o[j] = from_f<T>(v[j]);
    }
  }
}

// Filter gradient of the direct convolution (small channel counts, fp32 or bf16):
//   dw[r,s,c,f] = sum_{n,oh,ow} x[n, oh*sh - pt + r, ow*sw - pl + s, c] * dy[n,oh,ow,f]
// The same implicit product with the output positions as the summed index, which is long (N * OH * OW)
// while the result is tiny: the positions are split over gridDim.z blocks, each writing its fp32 partial
// sums to part[z][k][f], and fold_slices_kernel adds those in a fixed order (no atomics:
// deterministic). Inside a block the 128 threads are SL slices of KG x FG threads; each thread owns
// 4 x 4 values of (k, f) and its slice takes every SL-th position. One block per (r, s, c), as it was
// before, left 9 blocks walking 200,000 positions for a 3x3 filter over one plane. Measured with the sizes
// above: 15.8 ms -> 38 us and 3.5 ms -> 42 us.
// Padded positions are absent (see above): a chunk whose dy holds an infinity or a NaN is added by the
// branch that tests every term.
constexpr int WG_MC = 64;        // positions staged at a time

template <typename T, int KG, int FG, bool VEC>
__global__ void __launch_bounds__(128, 4) conv2d_wgrad_direct_kernel(const T* __restrict__ x, const T* __restrict__ dy,
                                                                 float* __restrict__ part, const ConvGeom g,
                                                                 long long per_block) {
  nb::follow_grid(x, dy);
  constexpr int SL = 128 / (KG * FG), KT = 4 * KG, FT = 4 * FG;
  constexpr int RED = SL > 1 ? 128 * 16 : 4, STAGE = WG_MC * (KT + FT);
  __shared__ __align__(16) float sm[RED > STAGE ? RED : STAGE];
  constexpr int KV = VEC ? 4 : 1;                    // VEC (C % 4 == 0): four channels of one pixel per load
  __shared__ int tap_r[KT / KV], tap_s[KT / KV];
  __shared__ int mh[WG_MC], mw[WG_MC];
  __shared__ long long mb[WG_MC];
  float (*xs)[KT] = reinterpret_cast<float (*)[KT]>(sm);
  float (*ds)[FT] = reinterpret_cast<float (*)[FT]>(sm + WG_MC * KT);
  const int tid = threadIdx.x;
  const int K = g.R * g.S * g.C, k0 = blockIdx.x * KT, f0 = blockIdx.y * FT;
  const long long positions = (long long)g.N * g.OH * g.OW;
  const long long p0 = blockIdx.z * per_block, p1 = min(positions, p0 + per_block);
  // the tap that this thread stages, of every (128 KV / KT)-th position
  const int kq = tid % (KT / KV), kt = k0 + kq * KV;
  const ConvTap tap = conv_tap(min(kt, K - KV), g);
  if (tid < KT / KV) {
    tap_r[tid] = tap.r;
    tap_s[tid] = tap.s;
  }
  const int fg = tid % FG, kg = (tid / FG) % KG, sl = tid / (FG * KG);
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (long long pc = p0; pc < p1; pc += WG_MC) {
    const int mn = (int)min((long long)WG_MC, p1 - pc);
    __syncthreads();
    if (tid < WG_MC) {
      const long long m = pc + min(tid, mn - 1);
      const int ow = (int)(m % g.OW);
      const long long q = m / g.OW;
      const int oh = (int)(q % g.OH);
      mh[tid] = oh * g.sh - g.pt;
      mw[tid] = ow * g.sw - g.pl;
      mb[tid] = (((q / g.OH) * g.H + mh[tid]) * g.W + mw[tid]) * g.C;
    }
    int odd = 0;
#pragma unroll 8
    for (int e = tid; e < WG_MC * FT; e += 128) {
      const int m = e / FT, f = f0 + e % FT;
      const float v = m < mn && f < g.F ? to_f<T>(dy[(pc + m) * g.F + f]) : 0.f;
      odd |= !isfinite(v);
      ds[m][e % FT] = v;
    }
    odd = __syncthreads_or(odd);
#pragma unroll 8
    for (int m = tid / (KT / KV); m < WG_MC; m += 128 / (KT / KV)) {
      const int ih = mh[m] + tap.r, iw = mw[m] + tap.s;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (m < mn && kt < K && ih >= 0 && ih < g.H && iw >= 0 && iw < g.W &&
          NB_IN_BOUNDS(NB_SITE_CONV_INPUT, mb[m] + tap.off + KV - 1, (long long)g.N * g.H * g.W * g.C)) {
        if (VEC) load4(x + mb[m] + tap.off, v);
        else v[0] = to_f<T>(x[mb[m] + tap.off]);
      }
      if (VEC) *reinterpret_cast<float4*>(&xs[m][kq * KV]) = make_float4(v[0], v[1], v[2], v[3]);
      else xs[m][kq * KV] = v[0];
    }
    __syncthreads();
    if (!odd) {
#pragma unroll 8
      for (int m = sl; m < WG_MC; m += SL) {
        const float4 a = *reinterpret_cast<const float4*>(&xs[m][kg * 4]);
        const float4 b = *reinterpret_cast<const float4*>(&ds[m][fg * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    } else {
      for (int m = sl; m < mn; m += SL)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ih = mh[m] + tap_r[(kg * 4 + i) / KV], iw = mw[m] + tap_s[(kg * 4 + i) / KV];
          if (ih < 0 || ih >= g.H || iw < 0 || iw >= g.W) continue;
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[m][kg * 4 + i], ds[m][fg * 4 + j], acc[i][j]);
        }
    }
  }
  if (SL > 1) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sm[(i * 4 + j) * 128 + tid] = acc[i][j];
    __syncthreads();
    if (sl != 0) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < SL; ++q) t += sm[(i * 4 + j) * 128 + q * (KG * FG) + tid];
        acc[i][j] = t;
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = k0 + kg * 4 + i;
    if (k >= K) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int f = f0 + fg * 4 + j;
      if (f < g.F) part[((size_t)blockIdx.z * K + k) * g.F + f] = acc[i][j];
    }
  }
}

// The same partial sums from patches, as the forward has them: a block walks bands of TH output rows of one image, stages
// their dy and the input under them once (the kernel above gathers every input value once per tap, in three steps with a
// barrier each per 64 positions, which is what bounds it) and reads each tap at its offset. A block's (r, s, c) are all taps
// of some channels, so that it stages no others: in the order of the filter each block staged every channel, and 256 x 14 x 14
// x 32 -> 16 took 49.5 us. offs: the patch address of a position. us with the sum of the slices, gathered and from patches,
// fp32, 3 x 3: 256 x 28 x 28 x 1 -> 16 22.0, 17.7; 64 x 32 x 32 x 3 -> 32 22.7, 14.5; 100 x 16 x 16 x 8 -> 16 18.3, 13.3;
// 32 x 28 x 28 x 64 -> 64 86.7, 74.4; 256 x 14 x 14 x 16 -> 32 31.0, 31.2; 7 x 7 of stride 2, 16 x 112 x 112 x 3 -> 64 92.7, 67.3.
template <typename T, int KG, int FG, bool VEC>
__global__ void __launch_bounds__(128, 4) conv2d_wgrad_patch_kernel(const T* __restrict__ x, const T* __restrict__ dy,
                                                                float* __restrict__ part, const ConvGeom g, int TH,
                                                                int bands, int total, int dvec) {
  nb::follow_grid(x, dy);
  constexpr int SL = 128 / (KG * FG), KT = 4 * KG, FT = 4 * FG, KV = VEC ? 4 : 1;
  extern __shared__ __align__(16) float conv_smem[];
  const int tid = threadIdx.x;
  const int RS = g.R * g.S, K = RS * g.C, f0 = blockIdx.y * FT;
  const int u0 = blockIdx.x * (KT / KV), units = K / KV;                   // (channel group, r, s) in this order
  const int q0 = u0 / RS, nq = (min(u0 + KT / KV, units) - 1) / RS - q0 + 1;
  const int pw = (g.OW - 1) * g.sw + g.S, plane = pw * ((TH - 1) * g.sh + g.R);
  float* xs = conv_smem;                               // [nq][ph][pw] of KV floats
  float* ds = xs + (plane * nq * KV + 3) / 4 * 4;      // [TH * OW][FT]
  int* offs = reinterpret_cast<int*>(ds + TH * g.OW * FT);
  for (int m = tid; m < TH * g.OW; m += 128) offs[m] = ((m / g.OW) * g.sh * pw + (m % g.OW) * g.sw) * KV;
  const int fg = tid % FG, kg = (tid / FG) % KG, sl = tid / (FG * KG);
  int at[4], tr[4], ts[4], kk[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int u = min(u0 + (VEC ? kg : kg * 4 + i), units - 1), q = u / RS, rs = u - q * RS;
    tr[i] = rs / g.S;
    ts[i] = rs - tr[i] * g.S;
    at[i] = ((q - q0) * plane + tr[i] * pw + ts[i]) * KV + (VEC ? i : 0);   // VEC: at[0] is of the first of four channels
    kk[i] = u0 + (VEC ? kg : kg * 4 + i) < units ? rs * g.C + q * KV + (VEC ? i : 0) : -1;
  }
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int b = blockIdx.z; b < total; b += gridDim.z) {
    const int n = b / bands, oh0 = (b - n * bands) * TH, count = min(TH, g.OH - oh0) * g.OW;
    __syncthreads();
    stage_patch<T, VEC>(x + (size_t)n * g.H * g.W * g.C, xs, g, n, oh0 * g.sh - g.pt, -g.pl, (TH - 1) * g.sh + g.R, pw, q0, nq);
    const T* d = dy + ((size_t)n * g.OH + oh0) * g.OW * g.F;
    int odd = 0;
    if (dvec) {
#pragma unroll 4
      for (int e = tid; e < count * (FT / 4); e += 128) {
        const int f = f0 + e % (FT / 4) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (f < g.F) load4(d + (size_t)(e / (FT / 4)) * g.F + f, v);
        odd |= !isfinite(v[0]) | !isfinite(v[1]) | !isfinite(v[2]) | !isfinite(v[3]);
        *reinterpret_cast<float4*>(ds + e * 4) = make_float4(v[0], v[1], v[2], v[3]);
      }
    } else {
#pragma unroll 4
      for (int e = tid; e < count * FT; e += 128) {
        const int f = f0 + e % FT;
        const float v = f < g.F ? to_f<T>(d[(size_t)(e / FT) * g.F + f]) : 0.f;
        odd |= !isfinite(v);
        ds[e] = v;
      }
    }
    odd = __syncthreads_or(odd);
    if (!odd) {
#pragma unroll 4
      for (int m = sl; m < count; m += SL) {
        const float* xp = xs + offs[m];
        float av[4];
        if constexpr (VEC) {
          const float4 a = *reinterpret_cast<const float4*>(xp + at[0]);
          av[0] = a.x; av[1] = a.y; av[2] = a.z; av[3] = a.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) av[i] = xp[at[i]];
        }
        const float4 t = *reinterpret_cast<const float4*>(ds + m * FT + fg * 4);
        const float bv[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    } else {                                           // dy holds an infinity or a NaN: padded positions are absent
      for (int m = sl; m < count; m += SL)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int ih = (oh0 + m / g.OW) * g.sh - g.pt + tr[i], iw = m % g.OW * g.sw - g.pl + ts[i];
          if (ih < 0 || ih >= g.H || iw < 0 || iw >= g.W) continue;
          const float a = xs[offs[m] + at[i]];
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a, ds[m * FT + fg * 4 + j], acc[i][j]);
        }
    }
  }
  if (SL > 1) {
    float* sm = conv_smem;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sm[(i * 4 + j) * 128 + tid] = acc[i][j];
    __syncthreads();
    if (sl != 0) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < SL; ++q) t += sm[(i * 4 + j) * 128 + q * (KG * FG) + tid];
        acc[i][j] = t;
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = kk[i];
    if (k < 0) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int f = f0 + fg * 4 + j;
      if (f < g.F) part[((size_t)blockIdx.z * K + k) * g.F + f] = acc[i][j];
    }
  }
}
// out[i] = sum_j part[j][i] for `slices` fp32 slices of n elements (n % 4 == 0): the second half of
// a split-K GEMM, whose partial products are written as fp32 by the tensor-core kernel.
template <typename T>
__global__ void __launch_bounds__(256) sum_slices_kernel(const float* __restrict__ part, T* __restrict__ out, size_t n,
                                                        int slices) {
  nb::follow_grid(part);
  const size_t nv = n / 4;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += (size_t)gridDim.x * blockDim.x) {
    float4 acc = reinterpret_cast<const float4*>(part)[i];
    for (int j = 1; j < slices; ++j) {
      const float4 v = reinterpret_cast<const float4*>(part + (size_t)j * n)[i];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    out[4 * i] = from_f<T>(acc.x); out[4 * i + 1] = from_f<T>(acc.y);
    out[4 * i + 2] = from_f<T>(acc.z); out[4 * i + 3] = from_f<T>(acc.w);
  }
}

// ============================================================== many copies, one launch
// The inputs of a captured step are copied into the graph's buffers and its results out of them: dozens of
// tensors of a few KB, for which a launch each is the whole cost. Up to COPY_MAX copies ride in one launch's
// parameters; a block moves one COPY_CHUNK of one of them, found by bisection over the chunk counts. 27 copies in and
// 27 out of a small training step: 2.4 + 2.8 us; the step went from 443 to 233 us.
constexpr int COPY_MAX = 128, COPY_CHUNK = 32 * 1024;
struct CopyBatch {
  void* dst[COPY_MAX];
  const void* src[COPY_MAX];
  unsigned long long bytes[COPY_MAX];
  unsigned first[COPY_MAX + 1];        // first block of every copy; first[n] = blocks
  int n;
};
template <typename W>
__device__ __forceinline__ void copy_words(void* dst, const void* src, unsigned bytes) {
  const unsigned words = bytes / sizeof(W);
  W* d = reinterpret_cast<W*>(dst);
  const W* s = reinterpret_cast<const W*>(src);
  unsigned i = threadIdx.x;
  for (; i + 3 * 256 < words; i += 4 * 256) {
    W v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = s[i + u * 256];
#pragma unroll
    for (int u = 0; u < 4; ++u) d[i + u * 256] = v[u];
  }
  for (; i < words; i += 256) d[i] = s[i];
  for (unsigned b = words * sizeof(W) + threadIdx.x; b < bytes; b += 256)
    reinterpret_cast<uint8_t*>(dst)[b] = reinterpret_cast<const uint8_t*>(src)[b];
}
__global__ void __launch_bounds__(256) copy_batch_kernel(const __grid_constant__ CopyBatch c) {
  nb::follow_grid();
  int lo = 0, hi = c.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (c.first[mid] <= blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const unsigned long long at = (unsigned long long)(blockIdx.x - c.first[lo]) * COPY_CHUNK, total = c.bytes[lo];
  if (at >= total) return;
  char* dst = static_cast<char*>(c.dst[lo]) + at;
  const char* src = static_cast<const char*>(c.src[lo]) + at;
  const unsigned n = (unsigned)(total - at < COPY_CHUNK ? total - at : COPY_CHUNK);
  const unsigned align = (unsigned)((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u);
  if (align == 0) copy_words<uint4>(dst, src, n);
  else if ((align & 3u) == 0) copy_words<unsigned>(dst, src, n);
  else if ((align & 1u) == 0) copy_words<unsigned short>(dst, src, n);
  else copy_words<uint8_t>(dst, src, n);
}

static inline int grid_for(size_t n, int per_block, int cap = 148 * 16) {
  size_t g = (n + per_block - 1) / per_block;
  if (g < 1) g = 1;
  return (int)(g > (size_t)cap ? cap : g);
}

}  // namespace nbk

using namespace nbk;
#define STREAM reinterpret_cast<cudaStream_t>(stream)
#define CHECK_LAUNCH() (cudaGetLastError() == cudaSuccess ? 0 : -1)

// dtype codes: 0 = fp32, 1 = bf16
extern "C" {

int nb_layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows,
                     int D, float eps, int dtype, void* stream) {
  if (rows <= 0) return 0;
  const int V = dtype ? 8 : 4;
  if (D % V) return -2;
  const int vpl = (D / V + 31) / 32;
  dim3 grid((rows + 3) / 4), block(128);
#define LN_FWD(T, VPL) nb::launch_following(layernorm_fwd_kernel<T, VPL>, grid, block, 0, STREAM, (const T*)x, (const T*)gamma, (const T*)beta, (T*)y, mean, rstd, rows, D, eps)
  if (dtype) {
    if (vpl <= 1) LN_FWD(bf16, 1); else if (vpl <= 2) LN_FWD(bf16, 2); else if (vpl <= 4) LN_FWD(bf16, 4);
    else if (vpl <= 8) LN_FWD(bf16, 8); else if (vpl <= 16) LN_FWD(bf16, 16); else return -3;
  } else {
    if (vpl <= 1) LN_FWD(float, 1); else if (vpl <= 2) LN_FWD(float, 2); else if (vpl <= 4) LN_FWD(float, 4);
    else if (vpl <= 8) LN_FWD(float, 8); else if (vpl <= 16) LN_FWD(float, 16); else return -3;
  }
  return CHECK_LAUNCH();
}

// Number of rows of the `partial` scratch buffer (each 2*D floats) that nb_layernorm_bwd writes for
// this problem: the grid of the one-pass kernels, or the number of row slabs of the two-kernel path.
static int ln_bwd_vpl(int D, int dtype) { const int V = dtype ? 8 : 4; return (D / V + 31) / 32; }
static int g_ln_bwd_two_kernels = 0;
// 1: always take the two-kernel path (dx, then dgamma / dbeta). For comparisons only: no row needs it.
void nb_layernorm_bwd_two_kernels(int on) { g_ln_bwd_two_kernels = on; }
int nb_layernorm_bwd_nblocks(int rows, int D, int dtype) {
  const int vpl = ln_bwd_vpl(D, dtype);              // = warps that share a row in layernorm_bwd_rows_kernel
  int nb, cap;
  if (g_ln_bwd_two_kernels || vpl > LN_MAX_WARPS) {
    nb = (rows + 255) / 256;
    cap = 128;
  } else if (vpl == 1) {
    nb = (rows + 3) / 4;
    cap = 148 * 4;
  } else {                                           // 32 warps per SM, two rows per slot and iteration
    const int rb = vpl < 8 ? 8 / vpl : 1;
    nb = (rows + 2 * rb - 1) / (2 * rb);
    cap = 148 * (32 / (vpl * rb));
  }
  if (nb > cap) nb = cap;
  return nb < 1 ? 1 : nb;
}

// Dynamic shared memory that lets no SM take more than its share of the `nb` blocks of `warps` warps, where registers (64 and 56 a thread) would:
// blocks begin in the room that the launch ahead leaves, and pile up where it leaves it first. us in chains, before launches followed each other, piled up
// and so: 100 x 4096 bf16 8.7, 10.7, 8.0; 4096 x 1536 fp32 22.1, 20.1, 16.4. Where all that fit are there the share is no help and shared memory
// is lost to the L1: 16384 x 2048 with its forward pass 74.8 us, 75.9 so.
static int ln_share(int nb, int warps, int dtype) {
  const int share = (nb + 147) / 148, fit = 65536 / ((dtype ? 64 : 56) * 32 * warps);
  return share < fit ? 227 * 1024 / (share + 1) + 1024 : 0;
}

int nb_layernorm_bwd(const void* dy, const void* x, const void* gamma, const float* mean, const float* rstd, const void* add, void* dx,
                     void* dgamma, void* dbeta, float* partial, int rows, int D, int dtype, void* stream) {
  if (rows <= 0) return 0;
  const int V = dtype ? 8 : 4;
  if (D % V) return -2;
  const int vpl = ln_bwd_vpl(D, dtype);
  if (vpl > LN_MAX_WARPS) return -3;
  if (add != nullptr && (g_ln_bwd_two_kernels || (reinterpret_cast<uintptr_t>(add) & 15))) return -4;
  const int nb = nb_layernorm_bwd_nblocks(rows, D, dtype);
  const int rpb = (rows + nb - 1) / nb;
  dim3 grid_dx((rows + 3) / 4);
  dim3 grid_gb((D + 32 * V - 1) / (32 * V), nb);
#define LN_BWD(T, VPL)                                                                                                \
  {                                                                                                                   \
    nb::launch_following(layernorm_bwd_dx_kernel<T, VPL>, grid_dx, 128, 0, STREAM, (const T*)dy, (const T*)x, (const T*)gamma, mean,    \
                                                                  rstd, (T*)dx, rows, D);                            \
    nb::launch_following(layernorm_bwd_dgb_kernel<T>, grid_gb, 256, 0, STREAM, (const T*)dy, (const T*)x, mean, rstd, partial, rows, D, \
                                                              rpb);                                                   \
  }
#define LN_BWD_ONE_PASS(T, ADD)                                                                                       \
  {                                                                                                                   \
    if (vpl == 1)                                                                                                     \
      nb::launch_following(layernorm_bwd_fused_kernel<T, ADD>, nb, 128, 0, STREAM, (const T*)dy, (const T*)x, (const T*)gamma, mean, rstd, \
                                                                 (const T*)add, (T*)dx, partial, rows, D);            \
    else {                                                                                                            \
      const int rb = vpl < 8 ? 8 / vpl : 1, ring = 32 * vpl * rb * 16 * 2 * 2 * (ADD ? 3 : 2);                        \
      const int share = ln_share(nb, vpl * rb, dtype), smem = ring > share ? ring : share;                                             \
      const auto kernel = layernorm_bwd_rows_kernel<T, ADD>;                                                          \
      if (smem > 40 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);          \
      nb::launch_following(kernel, nb, 32 * vpl * rb, smem, STREAM, (const T*)dy, (const T*)x, (const T*)gamma, mean, rstd, (const T*)add, (T*)dx, \
                                                  partial, rows, D, vpl, rb);                                         \
    }                                                                                                                 \
  }
  if (!g_ln_bwd_two_kernels) {
    if (dtype) { if (add) LN_BWD_ONE_PASS(bf16, true) else LN_BWD_ONE_PASS(bf16, false) }
    else { if (add) LN_BWD_ONE_PASS(float, true) else LN_BWD_ONE_PASS(float, false) }
  } else if (dtype) {
    if (vpl <= 1) LN_BWD(bf16, 1) else if (vpl <= 2) LN_BWD(bf16, 2) else if (vpl <= 4) LN_BWD(bf16, 4)
    else if (vpl <= 8) LN_BWD(bf16, 8) else LN_BWD(bf16, 16)
  } else {
    if (vpl <= 1) LN_BWD(float, 1) else if (vpl <= 2) LN_BWD(float, 2) else if (vpl <= 4) LN_BWD(float, 4)
    else if (vpl <= 8) LN_BWD(float, 8) else LN_BWD(float, 16)
  }
#undef LN_BWD
#undef LN_BWD_ONE_PASS
  const dim3 grid_fold((D + 31) / 32, 2);
  if (dtype) nb::launch_following(colsum_partials_kernel<bf16>, grid_fold, 1024, 0, STREAM, partial, (bf16*)dgamma, (bf16*)dbeta, nb, D);
  else nb::launch_following(colsum_partials_kernel<float>, grid_fold, 1024, 0, STREAM, partial, (float*)dgamma, (float*)dbeta, nb, D);
  return CHECK_LAUNCH();
}

// Narrow: fewer vectors per row than a warp has lanes, and rows enough for many blocks (256 rows each at least).
static bool colsum_narrow(int rows, int N, int V) { return N / V < 32 && rows >= 4096; }
// Row slabs. Otherwise 512 rows each and at most 64 slabs, but no fewer than give every SM two blocks while a
// warp still has eight rows: at 2002 x 512 four slabs of two column tiles were 8 blocks, each warp of which
// read 64 rows one after the other. 2002 x 512 to 2002 x 2048 bf16: 8.3 us and 1.6 for the final sum, now 2.8 and 2.5;
// 16384 x 8192, where the slabs stay as they were, 62 us both ways.
int nb_colsum_nparts(int rows, int N, int in_dtype) {
  const int V = in_dtype ? 8 : 4, tiles = (N + 32 * V - 1) / (32 * V);
  int np = (rows + 511) / 512, most = 64;
  if (colsum_narrow(rows, N, V)) {
    np = (rows + 255) / 256;
    most = 148 * 4;
  } else {
    int fill = (2 * 148 + tiles - 1) / tiles;
    if (fill > (rows + 63) / 64) fill = (rows + 63) / 64;
    if (np < fill) np = fill;
  }
  if (np > most) np = most;
  return np < 1 ? 1 : np;
}
// partial: fp32 scratch of nb_colsum_nparts(rows, N, in_dtype) * N elements.
int nb_colsum(const void* x, void* out, float* partial, int rows, int N, int in_dtype, int out_dtype, void* stream) {
  const int V = in_dtype ? 8 : 4;
  if (N % V) return -2;
  const int np = nb_colsum_nparts(rows, N, in_dtype);
  const int rpb = (rows + np - 1) / np;
  if (colsum_narrow(rows, N, V)) {
    if (in_dtype) nb::launch_following(colsum_narrow_kernel<bf16>, np, 256, 0, STREAM, (const bf16*)x, partial, rows, N, rpb);
    else nb::launch_following(colsum_narrow_kernel<float>, np, 256, 0, STREAM, (const float*)x, partial, rows, N, rpb);
  } else {
    const dim3 grid((N + 32 * V - 1) / (32 * V), np);
    if (in_dtype) nb::launch_following(colsum_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, partial, rows, N, rpb);
    else nb::launch_following(colsum_kernel<float>, grid, 256, 0, STREAM, (const float*)x, partial, rows, N, rpb);
  }
  if (out_dtype) fold_slices<bf16>(partial, out, (size_t)N, np, STREAM);
  else fold_slices<float>(partial, out, (size_t)N, np, STREAM);
  return CHECK_LAUNCH();
}

// Column sums of `count` matrices of one type (host arrays of device pointers and sizes) in as few launches as their table
// has room for; `wide`: tiles of 32 vectors of columns instead of 8. Returns the number of launches, or a negative code.
int nb_colsum_group(const void* const* x, void* const* out, const int* rows, const int* N, const int* out_dtype, int count, int in_dtype,
                    int wide, void* stream) {
  const int V = in_dtype ? 8 : 4, L = wide ? 32 : 8;
  int launches = 0;
  for (int k = 0; k < count;) {
    ColsumGroup g;
    unsigned tiles = 0;
    g.count = 0;
    for (; k < count && g.count < COLSUM_GROUP; ++k) {
      if (N[k] <= 0) continue;
      const int vec = N[k] % V == 0 && (reinterpret_cast<uintptr_t>(x[k]) & 15) == 0, width = vec ? L * V : L;
      g.leaf[g.count++] = ColsumGroup::Leaf{x[k], out[k], rows[k], N[k], tiles, vec, out_dtype[k]};
      tiles += (N[k] + width - 1) / width;
    }
    if (g.count == 0) break;
    const dim3 grid(tiles, COLSUM_CLUSTER);
    if (in_dtype) {
      if (wide) nb::launch_following(colsum_group_kernel<bf16, 32>, grid, 256, 0, STREAM, g); else nb::launch_following(colsum_group_kernel<bf16, 8>, grid, 256, 0, STREAM, g);
    } else {
      if (wide) nb::launch_following(colsum_group_kernel<float, 32>, grid, 256, 0, STREAM, g); else nb::launch_following(colsum_group_kernel<float, 8>, grid, 256, 0, STREAM, g);
    }
    ++launches;
  }
  return cudaGetLastError() == cudaSuccess ? launches : -1;
}

// Rows by a block each: some hundred long ones, three to seven for an SM, begin when all ahead has ended, evenly spread (see launch_when). us in chains,
// before launches followed each other, following and so: softmax of 627 x 10001 fp32 21.4, 23.7, 21.5; cross-entropy's log-sum-exp 6.5, 6.9, 6.6 and
// gradient 8.2, 9.4, 8.4; 763 x 32000 bf16 13.9, 14.6, 13.9 and 21.6, 23.8, 22.0. Fewer, or a whole wave of them, are better off following (300 x 32000
// fp32 8.9, 9.6 behind; 1183 x 10001 8.1, 8.8).
static bool rows_follow(int rows, int D) { return D < 8192 || rows < 400 || rows > 1100; }

int nb_softmax(const void* x, void* y, int rows, int D, int log, int dtype, void* stream) {
  if (rows <= 0) return 0;
  if (dtype) {
    if (log) nb::launch_when(rows_follow(rows, D), softmax_kernel<bf16, true>, rows, 256, 0, STREAM, (const bf16*)x, (bf16*)y, rows, D);
    else nb::launch_when(rows_follow(rows, D), softmax_kernel<bf16, false>, rows, 256, 0, STREAM, (const bf16*)x, (bf16*)y, rows, D);
  } else {
    if (log) nb::launch_when(rows_follow(rows, D), softmax_kernel<float, true>, rows, 256, 0, STREAM, (const float*)x, (float*)y, rows, D);
    else nb::launch_when(rows_follow(rows, D), softmax_kernel<float, false>, rows, 256, 0, STREAM, (const float*)x, (float*)y, rows, D);
  }
  return CHECK_LAUNCH();
}

int nb_lse_pick_fwd(const void* logits, const long long* tgt, float* lse, float* picked, int rows, int D, int dtype,
                    void* stream) {
  if (rows <= 0) return 0;
  const bool whole = D % (dtype ? 8 : 4) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  const bool wide = D >= 8 * 256 * (dtype ? 8 : 4);
#define LSE_V(T, W, WIDE) nb::launch_when(rows_follow(rows, D), lse_pick_fwd_kernel<T, W, WIDE>, rows, 256, 0, STREAM, (const T*)logits, tgt, lse, picked, rows, D)
#define LSE(T, W) do { if (wide) LSE_V(T, W, true); else LSE_V(T, W, false); } while (0)
  if (dtype) { if (whole) LSE(bf16, true); else LSE(bf16, false); }
  else { if (whole) LSE(float, true); else LSE(float, false); }
#undef LSE
#undef LSE_V
  return CHECK_LAUNCH();
}
int nb_lse_pick_bwd(const void* logits, const long long* tgt, const float* lse, const float* g_lse, const float* g_pick,
                    void* dlogits, int rows, int D, int dtype, void* stream) {
  if (rows <= 0) return 0;
  const bool whole = D % (dtype ? 8 : 4) == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0;
#define LSE(T, W) nb::launch_when(rows_follow(rows, D), lse_pick_bwd_kernel<T, W>, rows, 256, 0, STREAM, (const T*)logits, tgt, lse, g_lse, g_pick, (T*)dlogits, rows, D)
  if (dtype) { if (whole) LSE(bf16, true); else LSE(bf16, false); }
  else { if (whole) LSE(float, true); else LSE(float, false); }
#undef LSE
  return CHECK_LAUNCH();
}

int nb_adamw(const void* p, const void* g, const float* m, const float* v, void* p_out, float* m_out, float* v_out,
             long long n, float lr, float b1, float b2, float eps, float wd, float bc1, float bc2, float grad_scale,
             const float* hyper, int p_dtype, int g_dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)n, 256 * 8, 148 * 8);
  const AdamHyper h{lr, b1, b2, eps, wd, bc1, bc2, grad_scale};
#define ADAMW(TP, TG) nb::launch_following(adamw_kernel<TP, TG>, grid, 256, 0, STREAM, (const TP*)p, (const TG*)g, m, v, (TP*)p_out, m_out, v_out, (size_t)n, h, hyper)
  if (p_dtype) { if (g_dtype) ADAMW(bf16, bf16); else ADAMW(bf16, float); }
  else { if (g_dtype) ADAMW(float, bf16); else ADAMW(float, float); }
#undef ADAMW
  return CHECK_LAUNCH();
}
// The updates of `count` tensors (host arrays of device pointers and element counts) with one set of hyperparameters. -2, and
// nothing updated, where one is not 16-byte aligned or has more than ADAM_GROUP_MAX elements.
int nb_adamw_group(const void* const* p, const void* const* g, const float* const* m, const float* const* v, void* const* p_out,
                   float* const* m_out, float* const* v_out, const int* n, int count, float lr, float b1, float b2, float eps,
                   float wd, float bc1, float bc2, float grad_scale, const float* hyper, int p_dtype, int g_dtype, void* stream) {
  const AdamHyper h{lr, b1, b2, eps, wd, bc1, bc2, grad_scale};
  for (int k = 0; k < count; ++k)                      // all of them, before the first launch updates any
    if (n[k] > 0 && (((reinterpret_cast<uintptr_t>(p[k]) | reinterpret_cast<uintptr_t>(g[k]) | reinterpret_cast<uintptr_t>(m[k]) |
                       reinterpret_cast<uintptr_t>(v[k]) | reinterpret_cast<uintptr_t>(p_out[k]) | reinterpret_cast<uintptr_t>(m_out[k]) |
                       reinterpret_cast<uintptr_t>(v_out[k])) & 15) || n[k] > ADAM_GROUP_MAX))
      return -2;
  for (int k = 0; k < count;) {
    AdamGroup c;
    unsigned blocks = 0;
    c.count = 0;
    for (; k < count && c.count < ADAM_GROUP; ++k) {
      if (n[k] <= 0) continue;
      c.leaf[c.count++] = AdamGroup::Leaf{p[k], g[k], m[k], v[k], p_out[k], m_out[k], v_out[k], (unsigned)n[k], blocks};
      blocks += ((unsigned)n[k] + 2047) / 2048;
    }
    if (c.count == 0) break;
#define ADAMW(TP, TG) nb::launch_following(adamw_group_kernel<TP, TG>, blocks, 256, 0, STREAM, c, h, hyper)
    if (p_dtype) { if (g_dtype) ADAMW(bf16, bf16); else ADAMW(bf16, float); }
    else { if (g_dtype) ADAMW(float, bf16); else ADAMW(float, float); }
#undef ADAMW
  }
  return CHECK_LAUNCH();
}
int nb_adam_hyper(const float* step, const float* plus, float* total, float* hyper, float lr, double b1, double b2, void* stream) {
  nb::launch_following(adam_hyper_kernel, 1, 1, 0, STREAM, step, plus, total, hyper, lr, b1, b2);
  return CHECK_LAUNCH();
}
int nb_mean_diff(const void* a, const void* b, void* d, void* out, long long n, int square, const void* count_at, float count, int dtype,
                 void* stream) {
  if (n <= 0 || n > (1 << 20)) return -2;
#define MEAN(T, C) nb::launch_following(mean_diff_kernel<T, C>, C, MEAN_THREADS, 0, STREAM, (const T*)a, (const T*)b, (T*)d, (T*)out, (int)n, square, (const T*)count_at, count)
  if (n <= 4 * MEAN_THREADS) { if (dtype) MEAN(bf16, 1); else MEAN(float, 1); }
  else { if (dtype) MEAN(bf16, 8); else MEAN(float, 8); }
#undef MEAN
  return CHECK_LAUNCH();
}
int nb_sgd(const void* p, const void* g, const float* buf, void* p_out, float* buf_out, long long n, float lr,
           float momentum, float wd, float grad_scale, int p_dtype, int g_dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)n, 256);
#define SGD(TP, TG) nb::launch_following(sgd_kernel<TP, TG>, grid, 256, 0, STREAM, (const TP*)p, (const TG*)g, buf, (TP*)p_out, buf_out, (size_t)n, lr, momentum, wd, grad_scale)
  if (p_dtype && g_dtype) SGD(bf16, bf16);
  else if (p_dtype) SGD(bf16, float);
  else if (g_dtype) SGD(float, bf16);
  else SGD(float, float);
  return CHECK_LAUNCH();
}

int nb_embedding_gather(const void* table, const long long* ids, const void* add, void* out, int n_ids, int D, int vocab,
                        int period, int dtype, void* stream) {
  if (n_ids <= 0) return 0;
  if (add != nullptr && period <= 0) return -2;
#define GATHER(T, ADD) nb::launch_following(embedding_gather_kernel<T, ADD>, n_ids, 128, 0, STREAM, (const T*)table, ids, (const T*)add, (T*)out, n_ids, D, vocab, period)
  if (dtype) { if (add) GATHER(bf16, true); else GATHER(bf16, false); }
  else { if (add) GATHER(float, true); else GATHER(float, false); }
#undef GATHER
  return CHECK_LAUNCH();
}
// out = base + scatter_add(ids, upd); base null: zeros. `work`: nb_embedding_scatter_work(...) 32-bit words of
// 16-byte aligned scratch.
static long long scat_max_heavy(long long n_ids) { return 2 * (n_ids / SCAT_SEG); }   // segments of rows with > SCAT_SEG entries
static long long scat_ints(long long n_ids, long long vocab) { return (3 * vocab + 4 + scat_max_heavy(n_ids) + 2 * n_ids + 3) / 4 * 4; }
// Atomics into an fp32 table, or bucketed ids, by times over tables of 2 .. 32000 rows of 8 .. 2048, 100 .. 100000 ids,
// spread or crowded on one row. The bucketing is 25 to 35 us of short launches: it wins where the table is more than the
// L2 keeps (32000 x 2048 bf16, 16384 ids: 263 us with atomics, 136), where much is added to few rows (1000 x
// 2048, 16384 ids: 83 and 46, all on one row 189 and 58; 2 x 256, 100000 ids: 433 and 56), and for many ids, each of
// which is a block of the atomics' grid (1000 x 64, 100000 ids: 64 and 46), not for small sums (16 x 8, 1000 ids: 11 and
// 31; 100 x 256, 10000 ids: 19 and 39; 100 x 64, 100000 ids: 64 and 71). Rows that are not whole vectors are read by
// elements, where it wins only with few ids in a large table (32000 x 1001: 1000 ids 110 and 62, 100000 ids 312 and 355).
static bool scat_atomics(long long n_ids, long long D, long long vocab, int dtype) {
  if (D % (dtype ? 8 : 4) != 0) return vocab * D <= (16ll << 20) || n_ids > vocab;
  return vocab * D <= (8ll << 20) && n_ids * D <= (24ll << 20) && (n_ids <= 49152 || (vocab <= 256 && n_ids * D <= (8ll << 20)));
}
long long nb_embedding_scatter_work(int n_ids, int D, int vocab, int dtype) {
  if (scat_atomics(n_ids, D, vocab, dtype)) return (long long)vocab * D;
  return scat_ints(n_ids, vocab) + 4ll * n_ids + scat_max_heavy(n_ids) * D;
}
int nb_embedding_scatter_add(int* work, const long long* ids, const void* upd, const void* base, void* out, int n_ids, int D,
                             int vocab, int dtype, void* stream) {
  if (vocab <= 0 || D <= 0) return 0;
  if (n_ids < 0) return -2;
  if (n_ids > 0 && scat_atomics(n_ids, D, vocab, dtype)) {
    const size_t n = (size_t)vocab * D;
    const bool direct = !dtype && base == nullptr;   // the sum is the result
    float* acc = direct ? (float*)out : reinterpret_cast<float*>(work);
    if (cudaMemsetAsync(acc, 0, n * sizeof(float), STREAM) != cudaSuccess) return -1;
    const bool vec = D % 4 == 0 && ((reinterpret_cast<uintptr_t>(upd) | reinterpret_cast<uintptr_t>(acc)) & 15) == 0;
#define SCAT(T, VEC) nb::launch_following(embedding_scatter_add_kernel<T, VEC>, n_ids, 128, 0, STREAM, acc, ids, (const T*)upd, n_ids, D, vocab)
    if (dtype) { if (vec) SCAT(bf16, true); else SCAT(bf16, false); }
    else { if (vec) SCAT(float, true); else SCAT(float, false); }
#undef SCAT
    const int grid = grid_for(n, 256);
    if (dtype) nb::launch_following(cast_kernel<float, bf16>, grid, 256, 0, STREAM, acc, (bf16*)out, n, (const bf16*)base);
    else if (!direct) nb::launch_following(cast_kernel<float, float>, grid, 256, 0, STREAM, acc, (float*)out, n, (const float*)base);
    return CHECK_LAUNCH();
  }
  // Crowded tables: rows of few entries are few, and the time is that of the long ones. us, all rows in one launch and a copied base
  // (or zeros) under the rows that occur: 16384 ids into 1000 x 2048 fp32 62, 52, bf16 36.5, 36.6; 33000 with 90 % padding into
  // 4097 x 2048 fp32 101, 95, bf16 30000 into 4096 58, 60; 65536 into 2000 x 1024 bf16 52, 50; below the line 60000 into 5000 x 1024 60, 67,
  // 65536 into 32000 x 1024 67, 90, with a base 82, 105.
  const bool crowded = n_ids >= (dtype == 0 && D >= 1024 ? 4ll : 24ll) * vocab;
  if (n_ids == 0 || crowded) {
    const size_t bytes = (size_t)vocab * D * (dtype ? 2 : 4);
    if ((base != nullptr ? cudaMemcpyAsync(out, base, bytes, cudaMemcpyDeviceToDevice, STREAM)
                         : cudaMemsetAsync(out, 0, bytes, STREAM)) != cudaSuccess)
      return -1;
    if (n_ids == 0) return 0;
  }
  ScatWs ws;
  ws.light = crowded ? 0 : SCAT_LIGHT;
  ws.counts = work;
  ws.done = ws.counts + vocab;
  ws.total = ws.done + vocab;
  ws.nseg = ws.total + 1;
  ws.nheavy = ws.nseg + 1;
  ws.nlight = ws.nheavy + 1;
  ws.gdone = ws.nlight + 1;
  ws.start = ws.gdone + scat_max_heavy(n_ids);
  ws.rank = ws.start + vocab;
  ws.list = ws.rank + n_ids;
  ws.seg = reinterpret_cast<int4*>(work + scat_ints(n_ids, vocab));
  float* part = reinterpret_cast<float*>(ws.seg + n_ids);
  const int idb = (n_ids + 255) / 256;
  if (cudaMemsetAsync(work, 0, (2 * (size_t)vocab + 4 + scat_max_heavy(n_ids)) * sizeof(int), STREAM) != cudaSuccess) return -1;
  nb::launch_following(scatter_count_kernel, idb, 256, 0, STREAM, ids, ws, n_ids, vocab);
  nb::launch_following(scatter_slots_kernel, (vocab + 255) / 256, 256, 0, STREAM, ws, n_ids, vocab);
  nb::launch_following(scatter_place_kernel, idb, 256, 0, STREAM, ids, ws, n_ids, vocab);
  const int V = dtype ? 8 : 4;
  const bool vec = D % V == 0 && ((reinterpret_cast<uintptr_t>(upd) | reinterpret_cast<uintptr_t>(base) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  int threads = 32;                                  // the power of two that covers a row in one pass, at most 256
  while (threads < 256 && threads * (vec ? V : 1) < D) threads *= 2;
  // blocks: four times what the chip holds, so that those of short segments make room (one time left the last of the long ones alone:
  // 16384 ids of text into 32000 x 2048 bf16 62 us, 54 so), or as many as there are entries and groups of SCAT_IDLE rows for their warps
  const long long held = 148ll * (crowded ? 2048 : 4 * (vec && dtype ? 768 : 1024)) / threads;
  const long long want = crowded ? n_ids : ((long long)vocab / SCAT_IDLE + 1) * 32 / threads + 1;
  const int grid = (int)(held < n_ids || held < want ? held : n_ids > want ? n_ids : want);
#define SCAT_R(T, VN, ALL) nb::launch_following(scatter_rows_kernel<T, VN, ALL>, grid, threads, 0, STREAM, (const T*)upd, (const T*)base, (T*)out, ws, part, n_ids, D, vocab)
#define SCAT(T, VN) do { if (crowded) SCAT_R(T, VN, false); else SCAT_R(T, VN, true); } while (0)
  if (dtype) { if (vec) SCAT(bf16, 8); else SCAT(bf16, 1); }
  else { if (vec) SCAT(float, 4); else SCAT(float, 1); }
#undef SCAT_R
#undef SCAT
  return CHECK_LAUNCH();
}

// out = base + scatter_add(ids, upd) from stably sorted ids; `out` already holds a copy of `base`.
int nb_embedding_scatter_sorted(const long long* sorted_ids, const long long* perm, const void* upd, const void* base,
                                void* out, int n_ids, int D, int vocab, int dtype, void* stream) {
  if (n_ids <= 0) return 0;
  if (dtype) nb::launch_following(embedding_scatter_sorted_kernel<bf16>, n_ids, 128, 0, STREAM, sorted_ids, perm, (const bf16*)upd, (const bf16*)base, (bf16*)out, n_ids, D, vocab);
  else nb::launch_following(embedding_scatter_sorted_kernel<float>, n_ids, 128, 0, STREAM, sorted_ids, perm, (const float*)upd, (const float*)base, (float*)out, n_ids, D, vocab);
  return CHECK_LAUNCH();
}

// n copies of bytes[i] bytes from src[i] to dst[i] (host arrays; the ranges do not overlap), as few launches as
// the parameter space allows. Returns the number of launches, or a negative code.
int nb_copy_batch(void* const* dst, const void* const* src, const unsigned long long* bytes, int n, void* stream) {
  int launches = 0;
  for (int i = 0; i < n;) {
    CopyBatch c;
    unsigned long long blocks = 0;
    c.n = 0;
    for (; i < n && c.n < COPY_MAX; ++i) {
      const unsigned long long k = (bytes[i] + COPY_CHUNK - 1) / COPY_CHUNK;
      if (k == 0) continue;
      if (blocks + k > 0x7fffffffull) {
        if (c.n == 0) return -4;
        break;
      }
      c.dst[c.n] = dst[i];
      c.src[c.n] = src[i];
      c.bytes[c.n] = bytes[i];
      c.first[c.n++] = (unsigned)blocks;
      blocks += k;
    }
    if (c.n == 0) break;
    c.first[c.n] = (unsigned)blocks;
    nb::launch_following(copy_batch_kernel, (unsigned)blocks, 256, 0, STREAM, c);
    ++launches;
  }
  return cudaGetLastError() == cudaSuccess ? launches : -1;
}

int nb_cast(const void* in, void* out, long long n, int in_dtype, int out_dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)n, 256);
  if (in_dtype && !out_dtype) nb::launch_following(cast_kernel<bf16, float>, grid, 256, 0, STREAM, (const bf16*)in, (float*)out, (size_t)n, nullptr);
  else if (!in_dtype && out_dtype) nb::launch_following(cast_kernel<float, bf16>, grid, 256, 0, STREAM, (const float*)in, (bf16*)out, (size_t)n, nullptr);
  else return -2;
  return CHECK_LAUNCH();
}

int nb_activation(const void* z, const void* dy, void* out, long long n, int mode, int bwd, int dtype, void* stream) {
  if (n <= 0) return 0;
  const int V = dtype ? 8 : 4;
  const int grid = grid_for((size_t)n, 256 * V);
  if (dtype) {
    if (bwd) nb::launch_following(act_kernel<bf16, true>, grid, 256, 0, STREAM, (const bf16*)z, (const bf16*)dy, (bf16*)out, (size_t)n, mode);
    else nb::launch_following(act_kernel<bf16, false>, grid, 256, 0, STREAM, (const bf16*)z, nullptr, (bf16*)out, (size_t)n, mode);
  } else {
    if (bwd) nb::launch_following(act_kernel<float, true>, grid, 256, 0, STREAM, (const float*)z, (const float*)dy, (float*)out, (size_t)n, mode);
    else nb::launch_following(act_kernel<float, false>, grid, 256, 0, STREAM, (const float*)z, nullptr, (float*)out, (size_t)n, mode);
  }
  return CHECK_LAUNCH();
}

int nb_rng(void* out, long long n, unsigned long long seed, unsigned long long offset, int mode, float a, float b,
           int dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)n, 256 * 4, 148 * 8);
  if (dtype) nb::launch_following(rng_kernel<bf16>, grid, 256, 0, STREAM, (bf16*)out, (size_t)n, seed, offset, mode, a, b, nullptr);
  else nb::launch_following(rng_kernel<float>, grid, 256, 0, STREAM, (float*)out, (size_t)n, seed, offset, mode, a, b, nullptr);
  return CHECK_LAUNCH();
}
int nb_dropout(const void* x, void* y, unsigned char* mask, long long n, float p, unsigned long long seed,
               unsigned long long offset, int dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)n, 256 * 4, 148 * 8);
  if (dtype) nb::launch_following(dropout_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, (bf16*)y, mask, (size_t)n, p, seed, offset, nullptr);
  else nb::launch_following(dropout_kernel<float>, grid, 256, 0, STREAM, (const float*)x, (float*)y, mask, (size_t)n, p, seed, offset, nullptr);
  return CHECK_LAUNCH();
}
// Variants whose stream position lives on the device: `state` = [seed, draws so far] (two 64-bit
// words of device memory), `salt` distinguishes the shards of one tensor. The draw counter is
// advanced here, after the kernel, by a one-thread launch on the same stream.
int nb_rng_dev(void* out, long long n, unsigned long long* state, unsigned long long salt, int mode, float a, float b,
               int dtype, void* stream) {
  if (n > 0) {
    const int grid = grid_for((size_t)n, 256 * 4, 148 * 8);
    if (dtype) nb::launch_following(rng_kernel<bf16>, grid, 256, 0, STREAM, (bf16*)out, (size_t)n, salt, 0, mode, a, b, state);
    else nb::launch_following(rng_kernel<float>, grid, 256, 0, STREAM, (float*)out, (size_t)n, salt, 0, mode, a, b, state);
  }
  nb::launch_following(rng_bump_kernel, 1, 1, 0, STREAM, state);
  return CHECK_LAUNCH();
}
int nb_dropout_dev(const void* x, void* y, unsigned char* mask, long long n, float p, unsigned long long* state,
                   unsigned long long salt, int dtype, void* stream) {
  if (n > 0) {
    const int grid = grid_for((size_t)n, 256 * 4, 148 * 8);
    if (dtype) nb::launch_following(dropout_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, (bf16*)y, mask, (size_t)n, p, salt, 0, state);
    else nb::launch_following(dropout_kernel<float>, grid, 256, 0, STREAM, (const float*)x, (float*)y, mask, (size_t)n, p, salt, 0, state);
  }
  nb::launch_following(rng_bump_kernel, 1, 1, 0, STREAM, state);
  return CHECK_LAUNCH();
}

int nb_nf4_dequant(const unsigned char* packed, const float* absmax, void* out, long long n, int block, int dtype,
                   void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)(n + 1) / 2, 256);
  if (dtype) nb::launch_following(nf4_dequant_kernel<bf16>, grid, 256, 0, STREAM, packed, absmax, (bf16*)out, (size_t)n, block);
  else nb::launch_following(nf4_dequant_kernel<float>, grid, 256, 0, STREAM, packed, absmax, (float*)out, (size_t)n, block);
  return CHECK_LAUNCH();
}

int nb_nf4_dequant_codes(const unsigned char* codes, const float* absmax, const float* codebook, void* out, long long n,
                         int block, int dtype, void* stream) {
  if (n <= 0) return 0;
  const int grid = grid_for((size_t)(n + 15) / 16, 256);
  const bool whole = block % 16 == 0 && ((reinterpret_cast<uintptr_t>(codes) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
#define NF4(T, W) nb::launch_following(nf4_dequant_codes_kernel<T, W>, grid, 256, 0, STREAM, codes, absmax, codebook, (T*)out, (size_t)n, block)
  if (dtype) { if (whole) NF4(bf16, true); else NF4(bf16, false); }
  else { if (whole) NF4(float, true); else NF4(float, false); }
#undef NF4
  return CHECK_LAUNCH();
}

int nb_pool2d_fwd(const void* x, void* y, int N, int H, int W, int C, int OH, int OW, int kh, int kw, int sh, int sw,
                  int ph, int pw, int mode, int dtype, void* stream) {
  const size_t total = (size_t)N * OH * OW * C;
  if (!total) return 0;
  const int V = dtype ? 8 : 4;
  CellGeom g;
  if (pool_cells(x, y, nullptr, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, V, g)) {
    const unsigned n = (unsigned)(total / V);
#define POOL(T, MAX) nb::launch_following(pool2d_cell_fwd_kernel<T, MAX>, (n + 255) / 256, 256, 0, STREAM, (const T*)x, (T*)y, g, n)
    if (dtype) { if (mode) POOL(bf16, true); else POOL(bf16, false); }
    else { if (mode) POOL(float, true); else POOL(float, false); }
#undef POOL
    return CHECK_LAUNCH();
  }
  const int grid = grid_for(total, 256);
  if (dtype) nb::launch_following(pool2d_fwd_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, (bf16*)y, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, mode);
  else nb::launch_following(pool2d_fwd_kernel<float>, grid, 256, 0, STREAM, (const float*)x, (float*)y, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, mode);
  return CHECK_LAUNCH();
}
int nb_pool2d_bwd(const void* x, const void* dy, void* dx, int N, int H, int W, int C, int OH, int OW, int kh, int kw,
                  int sh, int sw, int ph, int pw, int mode, int relu, int dtype, void* stream) {
  const size_t total = (size_t)N * H * W * C;
  if (!total) return 0;
  if (relu && mode != 1) return -2;
  const int V = dtype ? 8 : 4;
  CellGeom g;
  if (pool_cells(x, dy, dx, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, V, g) && (mode == 1 || pool_cells_avg_bwd(N, C, g))) {
    const unsigned n = (unsigned)((size_t)N * g.cells_h * g.cells_w * g.CV);
#define POOL(T, ...) nb::launch_following(pool2d_cell_bwd_kernel<T, __VA_ARGS__>, (n + 255) / 256, 256, 0, STREAM, (const T*)x, (const T*)dy, (T*)dx, g, n)
    if (dtype) { if (relu) POOL(bf16, true, true); else if (mode) POOL(bf16, true); else POOL(bf16, false); }
    else { if (relu) POOL(float, true, true); else if (mode) POOL(float, true); else POOL(float, false); }
#undef POOL
    return CHECK_LAUNCH();
  }
  const int grid = grid_for(total, 256);
  if (dtype) nb::launch_following(pool2d_bwd_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, (const bf16*)dy, (bf16*)dx, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, mode, relu);
  else nb::launch_following(pool2d_bwd_kernel<float>, grid, 256, 0, STREAM, (const float*)x, (const float*)dy, (float*)dx, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, mode, relu);
  return CHECK_LAUNCH();
}

int nb_pool2d_select(const void* x, const void* t, void* y, int N, int H, int W, int C, int OH, int OW, int kh, int kw,
                     int sh, int sw, int ph, int pw, int dtype, void* stream) {
  const size_t total = (size_t)N * OH * OW * C;
  if (!total) return 0;
  const int grid = grid_for(total, 256);
  if (dtype) nb::launch_following(pool2d_select_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)x, (const bf16*)t, (bf16*)y, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw);
  else nb::launch_following(pool2d_select_kernel<float>, grid, 256, 0, STREAM, (const float*)x, (const float*)t, (float*)y, N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw);
  return CHECK_LAUNCH();
}

// Forward from patches: positions per thread (0: not taken), output rows of a band, and the filter tiles of 4 `fg` channels. Where the patch and
// the filter tile fit 48 KB, positions fill the threads to 60 % (rows of one image only) and there are blocks enough, but not
// one channel at a time with a stride (bank conflicts: 16 x 112 x 112 x 3 -> 64, 7 x 7 of stride 2, 59.5 us tiled, 67.2 from patches): 8 positions
// per thread from two blocks per SM on, 4 from 48 blocks on (148 where a sum has few terms or strides widen the patches: 1 x 224 x 224
// x 3 -> 16 of stride 2 5.6 us, 7.7 from 112 patches). Of 260 sizes in either type that these lines take the patches were slower in 74, down
// to 0.66 of the tiled kernel's speed; with the following in 6, at 0.87 and more (us, tiled and from patches):
//  - channels in fours: whole output vectors and a value staged for at least 1.75 terms, or one tap (64 x 24 x 24 x 32 -> 1, 1 x 1, 4.7,
//    7.1; 100 x 32 x 32 x 32 -> 32, 1 x 1 of stride 2, 7.2, 9.0; 100 x 40 x 40 x 12 -> 16, 2 x 2 of stride 2, 8.0, 9.6); results one by one only where
//    sums are longer than 64 terms (256 x 12 x 12 x 8 -> 33, 2 x 2, 14.3, 18.1; 256 x 32 x 32 x 12 -> 33, 3 x 3, 175, 122);
//  - one channel at a time: whole vectors, one tap or at least 5 terms per value, 56 positions and a tile mostly of channels that exist
//    (16 x 40 x 40 x 1 -> 32 6.0, 7.7; 100 x 12 x 12 x 1 -> 64 6.0, 7.6; 32 x 112 x 112 x 5 -> 20 80, 92; 128 x 64 x 64 x 1 -> 8 18.6, 14.0), or sums
//    of 200 terms and more (100 x 64 x 64 x 5 -> 7, 7 x 7, 132, 100).
struct ConvPatches {
  int px, th, bands, fg;
  long long f_tiles;
};
static ConvPatches conv_patches(const ConvGeom& g, bool vec, bool fvec) {
  const int fg = g.F <= 8 ? 2 : g.F <= 16 ? 4 : 8;
  const long long f_tiles = (g.F + 4 * fg - 1) / (4 * fg), K = (long long)g.R * g.S * g.C;
  ConvPatches p{0, 0, 0, fg, f_tiles};
  for (int c = 8; c >= 4 && !p.px && K > 0 && (vec || g.sw == 1); c -= 4) {   // (an empty sum stays tiled)
    const int mt = 128 / fg * c;
    if (g.OW > mt) continue;
    const int nb = (g.OH + mt / g.OW - 1) / (mt / g.OW), rows = (g.OH + nb - 1) / nb, bands = (g.OH + rows - 1) / rows;
    const long long patch = ((long long)(rows - 1) * g.sh + g.R) * ((long long)(g.OW - 1) * g.sw + g.S) * g.C, count = (long long)rows * g.OW;
    if (5ll * g.OH * g.OW < 3ll * nb * mt || 4ll * K * 4 * fg + 4 * patch > 48 * 1024 ||
        (long long)g.N * nb * f_tiles < (c == 8 ? 2 * 148 : K >= 32 && g.sh * g.sw == 1 ? 48 : 148))
      continue;
    // terms per staged value: K count / patch
    const bool tap = g.R * g.S == 1 && g.sh * g.sw == 1;
    const bool pays = vec ? (fvec ? tap || 4 * K * count >= 7 * patch : K > 64 && 2 * K * count >= 5 * patch)
                          : K >= 200 || (fvec && (tap || (K * count >= 5 * patch && count >= 56 && 10ll * g.F >= 7 * f_tiles * 4 * fg)));
    if (!pays || (long long)g.N * bands >= 0x7fffffffll || f_tiles > 65535) break;
    p = ConvPatches{c, rows, bands, fg, f_tiles};
  }
  return p;
}
// For tests: positions per thread where nb_conv2d_direct takes patches (all operands aligned), 0 where it does not.
int nb_conv2d_patches(int N, int H, int W, int C, int R, int S, int F, int OH, int OW, int sh, int sw) {
  if (OH <= 0 || OW <= 0) return 0;
  return conv_patches(ConvGeom{N, H, W, C, R, S, F, OH, OW, sh, sw, 0, 0}, C % 4 == 0, F % 4 == 0).px;
}

int nb_conv_flip(const void* w, void* out, int R, int S, int C, int F, int dtype, void* stream) {
  const long long n = (long long)R * S * C * F;
  if (n <= 0) return 0;
  if (n > 0x7fffffffll) return -2;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (dtype) nb::launch_following(conv_flip_kernel<bf16>, grid, 256, 0, STREAM, (const bf16*)w, (bf16*)out, R * S, C, F, (unsigned)n);
  else nb::launch_following(conv_flip_kernel<float>, grid, 256, 0, STREAM, (const float*)w, (float*)out, R * S, C, F, (unsigned)n);
  return CHECK_LAUNCH();
}
int nb_conv2d_direct(const void* x, const void* w, const void* bias, void* y, int N, int H, int W, int C, int R, int S,
                     int F, int OH, int OW, int sh, int sw, int pt, int pl, int relu, int dtype, void* stream) {
  const size_t positions = (size_t)N * OH * OW;
  if (!positions || !F) return 0;
  const ConvGeom g{N, H, W, C, R, S, F, OH, OW, sh, sw, pt, pl};
  // the narrowest channel tile that holds F, so that lanes of absent channels are few
  const bool vec = C % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & (dtype ? 7 : 15)) == 0;
  const auto grid = [&](int fg) {
    const unsigned tiles = (unsigned)((F + 4ll * fg - 1) / (4 * fg));
    return dim3((unsigned)((positions + 256 / fg - 1) / (256 / fg)), tiles < 65535u ? tiles : 65535u, (tiles + 65534u) / 65535u);
  };
  const int low = dtype ? 7 : 15, wvec = F % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & low) == 0, yvec = F % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & low) == 0;
  const ConvPatches pp = conv_patches(g, vec, wvec && yvec);
  // (as for the filter gradient: from 3e8 multiply-adds on following gains 0.4 % in the mean and may cost a quarter, 256 x 28 x 28 x 16 -> 16, 5 x 5 of
  // stride 2, 55.4 and 70.7 us; a classifier's 256 x 14 x 14 x 16 -> 32, of 2.3e8, gains 1.5 us a launch in its step)
  const bool following = (double)positions * F * R * S * C < 3e8;
  if (pp.px) {
    const int px = pp.px, th = pp.th, bands = pp.bands, fg_w = pp.fg;
    const size_t smem = 4 * ((size_t)R * S * C * 4 * fg_w + (size_t)((th - 1) * sh + R) * ((OW - 1) * sw + S) * C);
    const dim3 pgrid((unsigned)(N * bands), (unsigned)pp.f_tiles);
#define PATCH_V(T, FG, PX, VEC) nb::launch_when(following, conv2d_patch_kernel<T, FG, PX, VEC>, pgrid, 128, smem, STREAM, (const T*)x, (const T*)w, (const T*)bias, (T*)y, g, th, bands, wvec, yvec, relu)
#define PATCH_P(T, FG, PX) do { if (vec) PATCH_V(T, FG, PX, true); else PATCH_V(T, FG, PX, false); } while (0)
#define PATCH(T, FG) do { if (px == 8) PATCH_P(T, FG, 8); else PATCH_P(T, FG, 4); } while (0)
    if (dtype) { if (fg_w == 2) PATCH(bf16, 2); else if (fg_w == 4) PATCH(bf16, 4); else PATCH(bf16, 8); }
    else { if (fg_w == 2) PATCH(float, 2); else if (fg_w == 4) PATCH(float, 4); else PATCH(float, 8); }
#undef PATCH
#undef PATCH_P
#undef PATCH_V
    return CHECK_LAUNCH();
  }
#define CONV_V(T, FG, VEC) nb::launch_when(following, conv2d_direct_kernel<T, FG, VEC>, grid(FG), 128, 0, STREAM, (const T*)x, (const T*)w, (const T*)bias, (T*)y, g, relu)
#define CONV(T, FG) do { if (vec) CONV_V(T, FG, true); else CONV_V(T, FG, false); } while (0)
  if (dtype) { if (F <= 8) CONV(bf16, 2); else if (F <= 16) CONV(bf16, 4); else CONV(bf16, 8); }
  else { if (F <= 8) CONV(float, 2); else if (F <= 16) CONV(float, 4); else CONV(float, 8); }
#undef CONV
#undef CONV_V
  return CHECK_LAUNCH();
}

// Slices of K for sgemm_kernel: as many as bring the grid to 300 blocks, of at least 64 steps.
int nb_sgemm_slices(int M, int N, int K) {
  const long long tiles = (long long)((M + SG - 1) / SG) * ((N + SG - 1) / SG);
  long long z = 300 / (tiles < 1 ? 1 : tiles);
  if (z > K / 64) z = K / 64;
  if (z > 32) z = 32;
  return z < 1 ? 1 : (int)z;
}
// partial: fp32 scratch of nb_sgemm_slices(M, N, K) * M * N elements, unused for one slice. Strides in elements.
int nb_sgemm(const float* a, const float* b, const float* bias, float* out, float* partial, int M, int N, int K, long long a_m,
             long long a_k, long long b_k, long long b_n, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || (M + SG - 1) / SG > 65535 || (long long)M * N > 0x7fffffffll) return -2;
  int z = nb_sgemm_slices(M, N, K);
  const int per = ((K + z - 1) / z + SG - 1) / SG * SG;
  z = (K + per - 1) / per;
  const SgemmArgs g{a, b, bias, z > 1 ? partial : out, M, N, K, per, a_m, a_k, b_k, b_n};
  nb::launch_following(sgemm_kernel, dim3((N + SG - 1) / SG, (M + SG - 1) / SG, z), 256, 0, STREAM, g);
  if (z > 1) nb::launch_following(sgemm_fold_kernel, (M * N + 31) / 32, 256, 0, STREAM, partial, bias, out, M * N, N, z);
  return CHECK_LAUNCH();
}

int nb_sum_slices(const float* part, void* out, long long n, int slices, int dtype, void* stream) {
  if (n <= 0 || slices <= 0) return 0;
  if (n & 3) return -2;
  const int grid = grid_for((size_t)n / 4, 256, 148 * 8);
  if (dtype) nb::launch_following(sum_slices_kernel<bf16>, grid, 256, 0, STREAM, part, (bf16*)out, (size_t)n, slices);
  else nb::launch_following(sum_slices_kernel<float>, grid, 256, 0, STREAM, part, (float*)out, (size_t)n, slices);
  return CHECK_LAUNCH();
}

// Position slices of the filter gradient: four blocks per SM and no more, since a few blocks above that would
// be a wave of their own (8 x 224 x 224 x 3 -> 64, 7 x 7: 594 blocks 310 us, 588 blocks 218); at least 256 positions each.
int nb_conv2d_wgrad_slices(long long positions, int K, int F) {
  const int kt = K <= 16 ? 16 : K <= 32 ? 32 : 64, ft = F <= 16 ? 16 : 32;
  const long long tiles = (long long)((K + kt - 1) / kt) * ((F + ft - 1) / ft);
  long long z = 148 * 4 / tiles;
  if (z > (positions + 255) / 256) z = (positions + 255) / 256;
  return (int)(z < 1 ? 1 : z);
}
// Bands of output rows for the filter gradient from patches, and whether to take it: where a band of some 96 positions (whole
// rows of one image) fits 48 KB and there are taps to share it (one tap: 256 x 14 x 14 x 16 -> 32 13.0 us without, 15.0 with), and
// the patches pay. Over 320 sizes in both types (4 to 224 pixels a side, 1 to 64 channels, filters of 2 to 7) they were 0.34 to 1.75
// times as fast as the gathering kernel, 109 times slower by 3 % or more; with these lines 7 times, by 9 % at most:
//  - bands of few positions are barriers (us, gathered and from patches: 100 x 4 x 4 x 24 -> 17 of stride 2, 4 positions, 17, 52;
//    256 x 5 x 5 x 16 -> 32 19.0, 23.2; 64 x 7 x 7 x 16 -> 16, 49 positions, 15.3, 13.2; one channel at a time, where gathering is slow,
//    64 x 6 x 6 x 5 -> 4 pays from 24 on);
//  - a slice has to stage less than it would gather, whole bands and halo included (64 x 28 x 28 x 16 -> 32, 2 x 2 of stride 2, every
//    value once, 19.7, 25.8; 1 x 224 x 224 x 3 -> 16 of stride 2 bf16 20.3, 21.9, fp32 22.5, 20.4), by half where dy comes one value at
//    a time beside whole pixels (1 x 112 x 112 x 24 -> 17, 5 x 5, 32, 37.5), and with no part of a band too much there for two
//    filter tiles (16 x 28 x 28 x 16 -> 17 20.2, 22.0);
//  - on a full chip (z fills it, of which whole bands take less) by no more than a fifth (64 x 28 x 28 x 16 -> 32 31.4, 34.4).
struct WgradPatches {
  int th, bands, slices;
  long long smem;
  bool take;
};
static WgradPatches wgrad_patches(const ConvGeom& g, int z, bool vec, bool dvec, int dtype) {
  const int K = g.R * g.S * g.C, kt = K <= 16 ? 16 : K <= 32 ? 32 : 64, ft = g.F <= 16 ? 16 : 32, kv = vec ? 4 : 1;
  const long long image = (long long)g.OH * g.OW, per = ((long long)g.N * image + z - 1) / z;
  const int nb = image >= 2 * 96 ? (int)min((long long)g.OH, image / 96) : 1, th = g.OH > 0 ? (g.OH + nb - 1) / nb : 1, bands = (g.OH + th - 1) / th;
  const long long total = (long long)g.N * bands, rounds = (total + z - 1) / z, count = (long long)th * g.OW;
  const long long spanned = ((long long)kt / kv + g.R * g.S - 2) / (g.R * g.S) + 1, channels = min(spanned * kv, (long long)g.C);
  const long long staged = ((long long)(th - 1) * g.sh + g.R) * ((long long)(g.OW - 1) * g.sw + g.S) * channels;
  WgradPatches p{th, bands, z, 4ll * ((staged + 3) / 4 * 4 + count * (ft + 1)), false};
  if (g.R * g.S <= 1 || p.smem > 48 * 1024 || total <= 0 || total >= 0x7fffffffll) return p;
  p.slices = (int)((total + rounds - 1) / rounds);           // no more than `part` has
  const bool scalar_dy = vec && !dvec;
  const long long tiles = (long long)((K + kt - 1) / kt) * ((g.F + ft - 1) / ft);
  p.take = count >= (vec || K <= 16 ? 40 : 24) && 100 * per * min(kt, K) >= rounds * staged * (scalar_dy ? 200 : !vec && dtype ? 125 : 110) &&
           !(scalar_dy && g.F > 16 && 10 * rounds * count > 11 * per) && !(vec && K > 64 && tiles * z >= 444 && 5 * rounds * count > 6 * per);
  return p;
}
// For tests: does nb_conv2d_wgrad_direct take patches (x and dy aligned)?
int nb_conv2d_wgrad_patches(int N, int H, int W, int C, int R, int S, int F, int OH, int OW, int sh, int sw, int dtype) {
  const ConvGeom g{N, H, W, C, R, S, F, OH, OW, sh, sw, 0, 0};
  return wgrad_patches(g, nb_conv2d_wgrad_slices((long long)N * OH * OW, R * S * C, F), C % 4 == 0, F % 4 == 0, dtype).take;
}
// part: fp32 scratch of nb_conv2d_wgrad_slices(N * OH * OW, R * S * C, F) * R * S * C * F elements.
int nb_conv2d_wgrad_direct(const void* x, const void* dy, void* dw, float* part, int N, int H, int W, int C, int R, int S, int F,
                           int OH, int OW, int sh, int sw, int pt, int pl, int dtype, void* stream) {
  const size_t n = (size_t)R * S * C * F;
  if (n == 0) return 0;
  const int K = R * S * C;
  const long long positions = (long long)N * OH * OW;
  const int z = nb_conv2d_wgrad_slices(positions, K, F);
  const long long per = (positions + z - 1) / z;
  const ConvGeom g{N, H, W, C, R, S, F, OH, OW, sh, sw, pt, pl};
  const bool vec = C % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & (dtype ? 7 : 15)) == 0;
  const int dvec = F % 4 == 0 && (reinterpret_cast<uintptr_t>(dy) & (dtype ? 7 : 15)) == 0;
  const WgradPatches pp = wgrad_patches(g, z, vec, dvec, dtype);
  const bool patch = pp.take;
  const int zp = patch ? pp.slices : z, th = pp.th, bands = pp.bands;
  const long long total = (long long)N * bands, smem = pp.smem;
  const size_t dyn = smem < 8192 ? 8192 : (size_t)smem;    // (the sum of the position slices of a block takes 8 KB)
  // Long ones start evenly spread (see launch_when). 220 sizes in chains, behind the launch ahead and following it: below 1e7 multiply-adds 1.07 times the
  // time, from 4e7 on 0.95 (64 x 56 x 56 x 32 -> 32, 3 x 3, 163 and 181 us; 256 x 16 x 16 x 4 -> 64, 5 x 5 of stride 2, 20.5 and 29.0; 100 x 16 x 16 x
  // 4 -> 64 17.4 and 21.0).
  const bool following = (double)positions * K * F < 4e7;
#define WGRAD_V(T, KG, FG, VEC)                                                                                                          \
  do {                                                                                                                                   \
    if (patch) nb::launch_when(following, conv2d_wgrad_patch_kernel<T, KG, FG, VEC>, dim3((K + 4 * KG - 1) / (4 * KG), (F + 4 * FG - 1) / (4 * FG), zp), 128, dyn, STREAM, (const T*)x, (const T*)dy, part, g, th, bands, (int)total, dvec); \
    else nb::launch_when(following, conv2d_wgrad_direct_kernel<T, KG, FG, VEC>, dim3((K + 4 * KG - 1) / (4 * KG), (F + 4 * FG - 1) / (4 * FG), z), 128, 0, STREAM, (const T*)x, (const T*)dy, part, g, per);  \
  } while (0)
#define WGRAD(T, KG, FG) do { if (vec) WGRAD_V(T, KG, FG, true); else WGRAD_V(T, KG, FG, false); } while (0)
#define WGRAD_T(T)                                                                            \
  do {                                                                                        \
    if (K <= 16) { if (F <= 16) WGRAD(T, 4, 4); else WGRAD(T, 4, 8); }                        \
    else if (K <= 32) { if (F <= 16) WGRAD(T, 8, 4); else WGRAD(T, 8, 8); }                   \
    else { if (F <= 16) WGRAD(T, 16, 4); else WGRAD(T, 16, 8); }                              \
    fold_slices<T>(part, dw, n, zp, STREAM);                                                  \
  } while (0)
  if (dtype) WGRAD_T(bf16);
  else WGRAD_T(float);
#undef WGRAD_T
#undef WGRAD
#undef WGRAD_V
  return CHECK_LAUNCH();
}

}  // extern "C"

NB_DEBUG_DEFINE(fused)

// Kernels of the portable Qwen2 executor on a GPU: fp32 / fp16 / bf16 activations, any head size.  They
// stand where that executor ran chains of torch operators (a norm was 8 launches, attention without
// its products 18, rotary positions 12): its step is bound by the host that launches them, 2000 launches
// and 36 ms for 4 layers of 512, two micro-steps, of which the GPU worked 6 ms.  One launch each here.
// Every value is rounded where the operators rounded it (sums in fp32, probabilities in fp32 until they
// enter a product), and this file is compiled without fast math: fp32 runs use it too.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "api.h"
#include "common.cuh"

namespace stb {

namespace {

template <class T> __device__ __forceinline__ float wide(T v);
template <> __device__ __forceinline__ float wide(float v) { return v; }
template <> __device__ __forceinline__ float wide(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float wide(__nv_bfloat16 v) { return __bfloat162float(v); }
template <class T> __device__ __forceinline__ T narrow(float v);
template <> __device__ __forceinline__ float narrow(float v) { return v; }
template <> __device__ __forceinline__ __half narrow(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 narrow(float v) { return __float2bfloat16_rn(v); }

constexpr int kThreads = 128;

// Sum (or maximum) over the CTA; every thread receives it.
template <bool MAX>
__device__ __forceinline__ float cta_reduce(float v) {
  __shared__ float part[kThreads / 32];
  auto join = [](float a, float b) { return MAX ? fmaxf(a, b) : a + b; };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = join(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();                                   // the last call's readers are done
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = part[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) v = join(v, part[w]);
  return v;
}

// ------------------------------------------------------------------ RMSNorm (fp32 rows), a CTA per row
__global__ void __launch_bounds__(kThreads)
portable_norm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ out,
                         float* __restrict__ inv_out, int cols, float eps) {
  const float* xr = x + static_cast<int64_t>(blockIdx.x) * cols;
  float ss = 0.f;
  for (int c = threadIdx.x; c < cols; c += kThreads) ss += xr[c] * xr[c];
  const float inv = rsqrtf(cta_reduce<false>(ss) / cols + eps);
  if (threadIdx.x == 0) inv_out[blockIdx.x] = inv;
  for (int c = threadIdx.x; c < cols; c += kThreads)
    out[static_cast<int64_t>(blockIdx.x) * cols + c] = xr[c] * inv * w[c];
}

// dx = inv (g w - x inv^2 mean(g w x)); partial[CTA, c] = sum over its rows of g (x inv)
__global__ void __launch_bounds__(kThreads)
portable_norm_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x,
                         const float* __restrict__ inv, const float* __restrict__ w, float* __restrict__ dx,
                         float* __restrict__ partial, int rows, int cols) {
  extern __shared__ float dw[];                      // thread t owns columns t, t + kThreads, ...
  for (int c = threadIdx.x; c < cols; c += kThreads) dw[c] = 0.f;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const int64_t at = static_cast<int64_t>(row) * cols;
    float dot = 0.f;
    for (int c = threadIdx.x; c < cols; c += kThreads) dot += g[at + c] * w[c] * x[at + c];
    dot = cta_reduce<false>(dot) / cols;
    const float iv = inv[row];
    for (int c = threadIdx.x; c < cols; c += kThreads) {
      const float gv = g[at + c], xv = x[at + c];
      dx[at + c] = iv * (gv * w[c] - xv * (iv * iv) * dot);
      dw[c] += gv * (xv * iv);
    }
  }
  for (int c = threadIdx.x; c < cols; c += kThreads)
    partial[static_cast<int64_t>(blockIdx.x) * cols + c] = dw[c];
}

// ------------------------------------------------------------------ rotary positions, heads to the front
// Linear outputs [B, S, heads * d] -> [B, heads, S, d]; q and k rotated in fp32 and rounded once, v moved.
// blockIdx.x = token, threads over its (hq + 2 hkv) * d elements.
template <class T, bool BACK>
__global__ void __launch_bounds__(kThreads)
portable_rotate_kernel(HeadTensors in, HeadTensors out, const float* __restrict__ cos,
                       const float* __restrict__ sin, int batch_tables, int seq, int hq, int hkv, int d) {
  const int b = blockIdx.x / seq, s = blockIdx.x - b * seq;
  const int64_t table = (static_cast<int64_t>(batch_tables > 1 ? b : 0) * seq + s) * d;
  const int half = d / 2, total = (hq + 2 * hkv) * d;
  for (int e = threadIdx.x; e < total; e += kThreads) {
    const int head = e / d, c = e - head * d;
    const int which = head < hq ? 0 : head < hq + hkv ? 1 : 2;
    const int h = which == 0 ? head : which == 1 ? head - hq : head - hq - hkv;
    const int n = which == 0 ? hq : hkv;
    const int64_t rows = (static_cast<int64_t>(b) * seq + s) * n * d + h * d;           // [B, S, n, d]
    const int64_t heads = ((static_cast<int64_t>(b) * n + h) * seq + s) * d;            // [B, n, S, d]
    const T* src = reinterpret_cast<const T*>(in.p[which]) + (BACK ? heads : rows);
    T* dst = reinterpret_cast<T*>(out.p[which]) + (BACK ? rows : heads);
    const float v = wide(src[c]);
    if (which == 2) {
      dst[c] = src[c];
    } else {
      const int o = c < half ? c + half : c - half;
      const float pair = wide(src[o]);
      // forward: x cos + rotate_half(x) sin; backward: g cos + the transpose of rotate_half on (g sin)
      const float turned = BACK ? (c < half ? __fmul_rn(pair, sin[table + o]) : -__fmul_rn(pair, sin[table + o]))
                                : __fmul_rn(c < half ? -pair : pair, sin[table + c]);
      dst[c] = narrow<T>(__fadd_rn(__fmul_rn(v, cos[table + c]), turned));
    }
  }
}

// ------------------------------------------------------------------ masked softmax, a CTA per row
// scores [B, hkv, g * S, S] (before the scale); a key is visible when it is not after the query and its
// mask byte is not zero.  Probabilities of a row without a visible key are zero.  `stats`: the row's
// maximum and sum, from which the backward forms the same fp32 probabilities again.
// What is not finite travels as in softmax(masked_fill(-inf)): an invisible key has e^-inf = 0 over the sum.
template <class T>
__global__ void __launch_bounds__(kThreads)
portable_softmax_fwd_kernel(const T* __restrict__ scores, const uint8_t* __restrict__ mask,
                            T* __restrict__ probs, float2* __restrict__ stats, int rows_per_batch, int seq,
                            float scale) {
  const int64_t row = blockIdx.x;
  const int i = static_cast<int>(row % seq);
  const uint8_t* km = mask != nullptr ? mask + row / rows_per_batch * seq : nullptr;
  const T* src = scores + row * seq;
  auto score = [&](int j) { return __fmul_rn(wide(src[j]), scale); };   // rounded, as the scaled scores were
  float top = -INFINITY;
  int seen = 0;
  for (int j = threadIdx.x; j <= i; j += kThreads)
    if (km == nullptr || km[j]) {
      top = fmaxf(top, score(j));
      seen = 1;
    }
  top = cta_reduce<true>(top);
  if (!__syncthreads_or(seen)) {
    for (int j = threadIdx.x; j < seq; j += kThreads) probs[row * seq + j] = narrow<T>(0.f);
    if (threadIdx.x == 0) stats[row] = make_float2(0.f, 0.f);       // (a sum of zero marks the row)
    return;
  }
  float sum = 0.f;
  for (int j = threadIdx.x; j <= i; j += kThreads)
    if (km == nullptr || km[j]) sum += expf(score(j) - top);
  sum = cta_reduce<false>(sum);
  if (threadIdx.x == 0) stats[row] = make_float2(top, sum);
  for (int j = threadIdx.x; j < seq; j += kThreads) {
    const bool visible = j <= i && (km == nullptr || km[j]);
    probs[row * seq + j] = narrow<T>((visible ? expf(score(j) - top) : 0.f) / sum);
  }
}

template <class T>
__global__ void __launch_bounds__(kThreads)
portable_softmax_bwd_kernel(const T* __restrict__ scores, const uint8_t* __restrict__ mask,
                            const float2* __restrict__ stats, const T* __restrict__ dprobs,
                            T* __restrict__ dscores, int rows_per_batch, int seq, float scale) {
  const int64_t row = blockIdx.x;
  const int i = static_cast<int>(row % seq);
  const uint8_t* km = mask != nullptr ? mask + row / rows_per_batch * seq : nullptr;
  const float2 st = stats[row];
  if (st.y == 0.f) {
    for (int j = threadIdx.x; j < seq; j += kThreads) dscores[row * seq + j] = narrow<T>(0.f);
    return;
  }
  const T* src = scores + row * seq;
  const T* dp = dprobs + row * seq;
  auto visible = [&](int j) { return j <= i && (km == nullptr || km[j]); };
  auto prob = [&](int j) { return (visible(j) ? expf(__fmul_rn(wide(src[j]), scale) - st.x) : 0.f) / st.y; };
  float dot = 0.f;
  for (int j = threadIdx.x; j < seq; j += kThreads) dot += prob(j) * wide(dp[j]);
  dot = cta_reduce<false>(dot);
  for (int j = threadIdx.x; j < seq; j += kThreads) {
    const float p = prob(j);
    dscores[row * seq + j] = narrow<T>(visible(j) ? (p * wide(dp[j]) - p * dot) * scale : 0.f);
  }
}

// ------------------------------------------------------------------ SwiGLU
// silu(gate) is rounded before the product, as the operator's output was
template <class T>
__global__ void portable_swiglu_fwd_kernel(const T* __restrict__ gate, const T* __restrict__ up,
                                           T* __restrict__ out, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float x = wide(gate[i]);
    out[i] = narrow<T>(wide(narrow<T>(x / (1.f + expf(-x)))) * wide(up[i]));
  }
}
template <class T>
__global__ void portable_swiglu_bwd_kernel(const T* __restrict__ grad, const T* __restrict__ gate,
                                           const T* __restrict__ up, T* __restrict__ dgate,
                                           T* __restrict__ dup, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float x = wide(gate[i]), g = wide(grad[i]);
    dup[i] = narrow<T>(g * wide(narrow<T>(x / (1.f + expf(-x)))));
    const float ds = wide(narrow<T>(g * wide(up[i])));
    const float sig = 1.f / (1.f + expf(-x));
    dgate[i] = narrow<T>(ds * sig * (1.f + x * (1.f - sig)));
  }
}

// out = a (+ b (+ c)) in fp32, in that order
template <class T>
__global__ void portable_sum_kernel(const T* __restrict__ a, const T* __restrict__ b,
                                    const T* __restrict__ c, float* __restrict__ out, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float v = wide(a[i]);
    if (b != nullptr) v += wide(b[i]);
    if (c != nullptr) v += wide(c[i]);
    out[i] = v;
  }
}

// Shard gradients of a unit, one table row {start in `packed`, length, offset in the arena} each:
// stored to the arena or added to it.
__global__ void portable_commit_kernel(const float* __restrict__ packed, const int64_t* __restrict__ table,
                                       float* __restrict__ arena, int accumulate) {
  const int64_t* row = table + 3 * blockIdx.y;
  const int64_t start = row[0], n = row[1], off = row[2];
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    arena[off + i] = accumulate ? arena[off + i] + packed[start + i] : packed[start + i];
}

int grid_of(int64_t n) { return static_cast<int>(std::min<int64_t>((n + 255) / 256, sm_count() * 16)); }

template <class F>
cudaError_t with_type(ScalarKind kind, F&& f) {
  if (kind == ScalarKind::f32) f(float{});
  else if (kind == ScalarKind::f16) f(__half{});
  else f(__nv_bfloat16{});
  count_launch();
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_portable_norm_fwd(const float* x, const float* w, float* out, float* inv, int64_t rows,
                                     int cols, float eps, cudaStream_t s) {
  if (rows > INT32_MAX || cols < 1) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  portable_norm_fwd_kernel<<<static_cast<int>(rows), kThreads, 0, s>>>(x, w, out, inv, cols, eps);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_portable_norm_bwd(const float* g, const float* x, const float* inv, const float* w,
                                     float* dx, float* partial, int parts, int64_t rows, int cols,
                                     cudaStream_t s) {
  if (rows > INT32_MAX || cols < 1 || cols > kPortableNormCols || parts < 1) return cudaErrorInvalidValue;
  portable_norm_bwd_kernel<<<parts, kThreads, cols * 4, s>>>(g, x, inv, w, dx, partial,
                                                             static_cast<int>(rows), cols);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_portable_rotate(ScalarKind kind, HeadTensors in, HeadTensors out, const float* cos,
                                   const float* sin, int batch_tables, int64_t batch, int seq, int hq,
                                   int hkv, int d, bool backward, cudaStream_t s) {
  if (batch * seq > INT32_MAX || d % 2 || (batch_tables != 1 && batch_tables != batch))
    return cudaErrorInvalidValue;
  if (batch * seq == 0) return cudaSuccess;
  const int grid = static_cast<int>(batch * seq);
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    if (backward)
      portable_rotate_kernel<T, true><<<grid, kThreads, 0, s>>>(in, out, cos, sin, batch_tables, seq, hq, hkv, d);
    else
      portable_rotate_kernel<T, false><<<grid, kThreads, 0, s>>>(in, out, cos, sin, batch_tables, seq, hq, hkv, d);
  });
}

cudaError_t launch_portable_softmax_fwd(ScalarKind kind, const void* scores, const uint8_t* mask, void* probs,
                                        float* stats, int64_t rows, int64_t rows_per_batch, int seq,
                                        float scale, cudaStream_t s) {
  if (rows > INT32_MAX || rows_per_batch > INT32_MAX || seq < 1) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    portable_softmax_fwd_kernel<T><<<static_cast<int>(rows), kThreads, 0, s>>>(
        static_cast<const T*>(scores), mask, static_cast<T*>(probs), reinterpret_cast<float2*>(stats),
        static_cast<int>(rows_per_batch), seq, scale);
  });
}

cudaError_t launch_portable_softmax_bwd(ScalarKind kind, const void* scores, const uint8_t* mask,
                                        const float* stats, const void* dprobs, void* dscores, int64_t rows,
                                        int64_t rows_per_batch, int seq, float scale, cudaStream_t s) {
  if (rows > INT32_MAX || rows_per_batch > INT32_MAX || seq < 1) return cudaErrorInvalidValue;
  if (rows == 0) return cudaSuccess;
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    portable_softmax_bwd_kernel<T><<<static_cast<int>(rows), kThreads, 0, s>>>(
        static_cast<const T*>(scores), mask, reinterpret_cast<const float2*>(stats),
        static_cast<const T*>(dprobs), static_cast<T*>(dscores), static_cast<int>(rows_per_batch), seq, scale);
  });
}

cudaError_t launch_portable_swiglu_fwd(ScalarKind kind, const void* gate, const void* up, void* out,
                                       int64_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    portable_swiglu_fwd_kernel<T><<<grid_of(n), 256, 0, s>>>(static_cast<const T*>(gate),
                                                             static_cast<const T*>(up), static_cast<T*>(out), n);
  });
}

cudaError_t launch_portable_swiglu_bwd(ScalarKind kind, const void* grad, const void* gate, const void* up,
                                       void* dgate, void* dup, int64_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    portable_swiglu_bwd_kernel<T><<<grid_of(n), 256, 0, s>>>(
        static_cast<const T*>(grad), static_cast<const T*>(gate), static_cast<const T*>(up),
        static_cast<T*>(dgate), static_cast<T*>(dup), n);
  });
}

cudaError_t launch_portable_sum(ScalarKind kind, const void* a, const void* b, const void* c, float* out,
                                int64_t n, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  return with_type(kind, [&](auto t) {
    using T = decltype(t);
    portable_sum_kernel<T><<<grid_of(n), 256, 0, s>>>(static_cast<const T*>(a), static_cast<const T*>(b),
                                                      static_cast<const T*>(c), out, n);
  });
}

cudaError_t launch_portable_commit(const float* packed, const int64_t* table, int n_params, int64_t largest,
                                   float* arena, bool accumulate, cudaStream_t s) {
  if (n_params < 1 || largest < 1) return cudaErrorInvalidValue;
  dim3 grid(static_cast<unsigned>(std::min<int64_t>((largest + 255) / 256, sm_count() * 4)), n_params);
  portable_commit_kernel<<<grid, 256, 0, s>>>(packed, table, arena, accumulate ? 1 : 0);
  count_launch();
  return cudaGetLastError();
}

}  // namespace stb

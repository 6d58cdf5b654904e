// Collectives written as kernels over NVLink peer memory (plain P2P loads through NVSwitch), each
// fused with the compute that follows it in the reference's NCCL pipeline:
//   * parameter all-gather + copy-out + fp32->bf16 cast  (src/sharded_runtime/runtime/materializer.py:31-114,
//     src/sharded_runtime/runtime/layout.py:77-90)
//   * gradient pack + reduce-scatter + 1/F scale + accumulate (+ AdamW)  (materializer.py:116-192,
//     layout.py:93-106, src/sharded_runtime/training/qwen2_trainer.py:48); with a multicast
//     address of the gradient slots the sum over the FSDP members is one `multimem.ld_reduce`
//     per 16 bytes, carried out inside the NVSwitch
//   * sequence-parallel activation gather / reduce-scatter (src/sharded_runtime/runtime/comm.py:781-884)
//   * embedding rows fetched from the owning shard without gathering the table.
// With degree 1 the same kernels read only local memory.  No kernel here waits on another GPU
// except the flag barrier and the small all-reduce, whose waits are bounded in time.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace stb {

namespace {

constexpr int kMaxSegs = 32;
struct SegTable {
  SegmentDesc s[kMaxSegs];
  int n;
};

__device__ __forceinline__ uint32_t pk2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Work is tiled in chunks of kChunk elements of one segment; blockIdx.y = segment.
constexpr int kChunk = 4096;

struct ShadowPtrs {
  const __nv_bfloat16* p[kMaxPeers];
};

// bf16 -> bf16 gather of one segment from the owners' compute-dtype shadow shards: the cast
// already happened where the optimizer wrote the parameter, so only 2 bytes per element cross
// NVLink instead of 4 (rounding before or after the transfer gives the same bits).
constexpr int kChunkB = 8192;
__device__ __forceinline__ void gather_shadow_segment(const ShadowPtrs& sh, const SegmentDesc& sg,
                                                      __nv_bfloat16* __restrict__ full_bf16) {
  const bool vec = (sg.q % 8 == 0) && (sg.shard_off % 8 == 0) && (sg.full_off % 8 == 0);
  for (int64_t chunk = blockIdx.x; chunk * kChunkB < sg.numel; chunk += gridDim.x) {
    const int64_t base = chunk * kChunkB;
    if (vec && base + kChunkB <= sg.numel && blockDim.x * 8 * 4 == kChunkB) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = base + (u * blockDim.x + threadIdx.x) * 8;
        const int r = static_cast<int>(i / sg.q);
        v[u] = *reinterpret_cast<const uint4*>(sh.p[r] + sg.shard_off + (i - r * sg.q));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = base + (u * blockDim.x + threadIdx.x) * 8;
        *reinterpret_cast<uint4*>(full_bf16 + sg.full_off + i) = v[u];
      }
    } else {
      const int64_t end = min(base + kChunkB, sg.numel);
      if (vec) {
        for (int64_t i = base + threadIdx.x * 8; i < end; i += blockDim.x * 8) {
          const int r = static_cast<int>(i / sg.q);
          const __nv_bfloat16* src = sh.p[r] + sg.shard_off + (i - r * sg.q);
          if (i + 7 < sg.numel) {
            *reinterpret_cast<uint4*>(full_bf16 + sg.full_off + i) =
                *reinterpret_cast<const uint4*>(src);
          } else {
            for (int64_t j = i; j < sg.numel; ++j) full_bf16[sg.full_off + j] = src[j - i];
          }
        }
      } else {
        for (int64_t i = base + threadIdx.x; i < end; i += blockDim.x) {
          const int r = static_cast<int>(i / sg.q);
          full_bf16[sg.full_off + i] = sh.p[r][sg.shard_off + (i - r * sg.q)];
        }
      }
    }
  }
}

__global__ void gather_params_kernel(PeerPtrs shards, ShadowPtrs shadows, int use_shadow, int degree,
                                     SegTable tab, __nv_bfloat16* __restrict__ full_bf16,
                                     float* __restrict__ full_fp32) {
  const SegmentDesc sg = tab.s[blockIdx.y];
  if (use_shadow && !sg.keep_fp32) {
    gather_shadow_segment(shadows, sg, full_bf16);
    return;
  }
  const bool vec = (sg.q % 4 == 0) && (sg.shard_off % 4 == 0) && (sg.full_off % 4 == 0);
  for (int64_t chunk = blockIdx.x; chunk * kChunk < sg.numel; chunk += gridDim.x) {
    const int64_t base = chunk * kChunk;
    if (vec && base + kChunk <= sg.numel && blockDim.x * 4 * 4 == kChunk) {
      // full chunk: four independent 16-byte loads in flight per thread before any store
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = base + (u * blockDim.x + threadIdx.x) * 4;
        const int r = static_cast<int>(i / sg.q);
        v[u] = *reinterpret_cast<const float4*>(shards.p[r] + sg.shard_off + (i - r * sg.q));
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = base + (u * blockDim.x + threadIdx.x) * 4;
        if (sg.keep_fp32) {
          *reinterpret_cast<float4*>(full_fp32 + sg.full_off + i) = v[u];
        } else {
          uint2 o;
          o.x = pk2(v[u].x, v[u].y);
          o.y = pk2(v[u].z, v[u].w);
          *reinterpret_cast<uint2*>(full_bf16 + sg.full_off + i) = o;
        }
      }
    } else if (vec) {
      for (int64_t i = base + threadIdx.x * 4; i < min(base + kChunk, sg.numel);
           i += blockDim.x * 4) {
        const int r = static_cast<int>(i / sg.q);  // q % 4 == 0: the 4 elements share a rank
        const int64_t off = i - r * sg.q;
        const float* src = shards.p[r] + sg.shard_off + off;
        if (i + 3 < sg.numel) {
          const float4 v = *reinterpret_cast<const float4*>(src);
          if (sg.keep_fp32) {
            *reinterpret_cast<float4*>(full_fp32 + sg.full_off + i) = v;
          } else {
            uint2 o;
            o.x = pk2(v.x, v.y);
            o.y = pk2(v.z, v.w);
            *reinterpret_cast<uint2*>(full_bf16 + sg.full_off + i) = o;
          }
        } else {
          for (int64_t j = i; j < sg.numel; ++j) {
            const float v = src[j - i];
            if (sg.keep_fp32)
              full_fp32[sg.full_off + j] = v;
            else
              full_bf16[sg.full_off + j] = __float2bfloat16(v);
          }
        }
      }
    } else {
      for (int64_t i = base + threadIdx.x; i < min(base + kChunk, sg.numel); i += blockDim.x) {
        const int r = static_cast<int>(i / sg.q);
        const float v = shards.p[r][sg.shard_off + (i - r * sg.q)];
        if (sg.keep_fp32)
          full_fp32[sg.full_off + i] = v;
        else
          full_bf16[sg.full_off + i] = __float2bfloat16(v);
      }
    }
  }
}

// Gradient reduction (+ AdamW).  Bound by memory: with AdamW 30 bytes per element (gradient read; p, m,
// v read and written; bf16 shadow written).  It runs on its own stream under the backward, which sets its
// shape.  A CTA takes ONE tile and leaves: a kernel of the compute stream (higher priority) that needs
// whole SMs can be placed only when the CTAs in its way have left, and with CTAs that lived for a sixth
// of the sweep every layer's gate|up dW GEMM (pairs of CTAs) stood still for that long -- 65 us at the
// 1.5B widths, 380 us twice a layer at the 7B widths.  The loads of a round are in flight together, the
// first of them before the status word is known: with AdamW and one member 128 bytes a thread, for the
// check alone 32, with several members 32 from each of four and then the 96 of p, m and v (before the sum
// they would spill).  One member with AdamW, alone, in place: 46.8 M elements 217 us (6470 GB/s; 248 us
// before), 233 M 1038 us (1187); the check alone 33 us for 46.8 M (84).  Tiles of 2048 and 8192 elements
// ran the training steps no faster.
// The vectors of a layer are shorter than a tile: 20 of 1536 elements take 9.2 us with one member (11.3
// with the elements of a vector one after the other), five odd segments 13.2 with four members (19).
constexpr int kRsThreads = 256;
constexpr int kRsGroups = 2;                                     // float4 groups a thread loads at once
constexpr int kRsRound = kRsThreads * 4 * kRsGroups;
constexpr int kRsTile = 2 * kRsRound;                            // 4096 elements
struct RsTable {
  SegmentDesc s[kMaxSegs];
  int first[kMaxSegs + 1];                                       // first tile of each segment
  int n;
};

__device__ __forceinline__ void adamw_update(float& p, float& m, float& v, float g, const AdamWArgs& a,
                                             float step_size, float inv_bc2_sqrt) {
  const float gr = g * a.grad_scale;
  p *= 1.f - a.lr * a.weight_decay;
  m = a.beta1 * m + (1.f - a.beta1) * gr;
  v = a.beta2 * v + (1.f - a.beta2) * gr * gr;
  p -= step_size * m / (sqrtf(v) * inv_bc2_sqrt + a.eps);
}

// Rank `rank` owns elements [rank*q, rank*q + q) of each segment (zero beyond numel).
// With a tensor-parallel axis (tp > 1) `full` lists the gradient slots of the whole mesh in rank
// order (index f * tp + t).  A TP-split parameter is summed over the F ranks of this rank's TP
// coordinate; a TP-replicated one (segment flag `pad`) over all F * tp ranks, scaled by
// rep_scale -- the T-way sum that the reference issues as a separate all-reduce after its
// reduce-scatter (src/sharded_runtime/runtime/materializer.py:228-233).
// LOCAL: a single member (degree * tp == 1), plain loads.
template <bool ADAMW, bool LOCAL>
__global__ void __launch_bounds__(kRsThreads, 4)
    reduce_scatter_kernel(PeerPtrs full, int degree, int rank, int tp, int tp_rank, RsTable tab,
                          float* gshard /* may be the slot itself */, float* __restrict__ p,
                          float* __restrict__ m, float* __restrict__ v, float split_scale,
                          float rep_scale, int accumulate, AdamWArgs a, int* __restrict__ flags,
                          __nv_bfloat16* __restrict__ shadow, const int* status,
                          const float* __restrict__ multicast) {
  // A failure recorded earlier (a peer that never signalled) means the slots may hold stale
  // data: neither the gradient shard nor, with ADAMW, the parameters are touched.  (Every thread asks
  // for itself, nothing below needs them to agree.)
  const bool skip = status_failed(status);
  int seg = 0;
  while (seg + 1 < tab.n && static_cast<int>(blockIdx.x) >= tab.first[seg + 1]) ++seg;
  const SegmentDesc& sg = tab.s[seg];
  const bool replicated = !LOCAL && tp > 1 && sg.pad != 0;
  const int n_src = LOCAL ? 1 : replicated ? degree * tp : degree;
  // replicated segments use one fixed summation order so every TP replica computes bit-identical
  // shard gradients (and updates); split segments rotate the order to spread the load
  const int first = replicated ? 0 : rank;
  const int stride = replicated ? 1 : tp;
  const int offset = LOCAL || replicated ? 0 : tp_rank;
  const float scale = replicated ? rep_scale : split_scale;
  const int64_t lo = static_cast<int64_t>(rank) * sg.q;
  const int64_t valid = max(static_cast<int64_t>(0), min(sg.q, sg.numel - lo));
  const bool vec = (sg.q % 4 == 0) && (sg.shard_off % 4 == 0) && (sg.full_off % 4 == 0);
  // a single member whose gradients were written straight into its shard: nothing to store
  const bool in_place = n_src == 1 && scale == 1.f && !accumulate &&
                        full.p[offset] + sg.full_off + lo == gshard + sg.shard_off;
  const float step_size = ADAMW ? a.lr / a.bias_correction1 : 0.f;
  const float inv_bc2_sqrt = ADAMW ? rsqrtf(a.bias_correction2) : 0.f;
  // the gradient check rides along: flags[0] = a non-finite reduced gradient was written,
  // flags[1] = a padding element of the shard is not exactly zero
  int bad = 0, pad_bad = 0;
  const int64_t base = static_cast<int64_t>(blockIdx.x - tab.first[seg]) * kRsTile;
  const int64_t end = min(base + kRsTile, sg.q);
  // G times four elements from i on, all of them data: 16-byte accesses, every load in flight before the
  // first use.  p, m and v stream past (nobody reads them again in this step): they should not push GEMM
  // operands out of L2
  auto vectors = [&](auto count, int64_t i) {
    constexpr int G = decltype(count)::value;
    const int64_t e = sg.shard_off + i;
    float4 g[G], pv[G], mv[G], vv[G];
    auto load_state = [&] {
#pragma unroll
      for (int u = 0; u < G; ++u) {
        pv[u] = __ldcs(reinterpret_cast<const float4*>(p + e + u * kRsThreads * 4));
        mv[u] = __ldcs(reinterpret_cast<const float4*>(m + e + u * kRsThreads * 4));
        vv[u] = __ldcs(reinterpret_cast<const float4*>(v + e + u * kRsThreads * 4));
      }
    };
    if (ADAMW && LOCAL) load_state();
    if (LOCAL) {
      const float* src = full.p[0] + sg.full_off + i;
#pragma unroll
      for (int u = 0; u < G; ++u)
        g[u] = *reinterpret_cast<const float4*>(src + u * kRsThreads * 4);
    } else if (multicast != nullptr && !replicated) {
      // NVLS: one load through the multicast address of the gradient slot; the NVSwitch reads
      // the same 16 bytes of every member's slot, adds them and returns the sum, so only
      // 1 / F of the gradient enters this GPU instead of (F - 1) / F
#pragma unroll
      for (int u = 0; u < G; ++u)
        asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(g[u].x), "=f"(g[u].y), "=f"(g[u].z), "=f"(g[u].w)
                     : "l"(multicast + sg.full_off + lo + i + u * kRsThreads * 4)
                     : "memory");
    } else {
#pragma unroll
      for (int u = 0; u < G; ++u) g[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      // rotate the peer order by rank so the ranks do not all hit one peer at once
#pragma unroll 4
      for (int d = 0; d < n_src; ++d) {
        const int src = ((first + d) % n_src) * stride + offset;
        const float* from = full.p[src] + sg.full_off + lo + i;
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const float4 t = *reinterpret_cast<const float4*>(from + u * kRsThreads * 4);
          g[u].x += t.x; g[u].y += t.y; g[u].z += t.z; g[u].w += t.w;
        }
      }
    }
    if (skip) return;
    if (ADAMW && !LOCAL) load_state();       // (before the sum they would spill)
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const int64_t eu = e + u * kRsThreads * 4;
      g[u].x *= scale; g[u].y *= scale; g[u].z *= scale; g[u].w *= scale;
      if (accumulate) {
        const float4 o = *reinterpret_cast<const float4*>(gshard + eu);
        g[u].x += o.x; g[u].y += o.y; g[u].z += o.z; g[u].w += o.w;
      }
      if (!in_place) *reinterpret_cast<float4*>(gshard + eu) = g[u];
      bad |= !(isfinite(g[u].x) && isfinite(g[u].y) && isfinite(g[u].z) && isfinite(g[u].w));
      if (ADAMW) {
        adamw_update(pv[u].x, mv[u].x, vv[u].x, g[u].x, a, step_size, inv_bc2_sqrt);
        adamw_update(pv[u].y, mv[u].y, vv[u].y, g[u].y, a, step_size, inv_bc2_sqrt);
        adamw_update(pv[u].z, mv[u].z, vv[u].z, g[u].z, a, step_size, inv_bc2_sqrt);
        adamw_update(pv[u].w, mv[u].w, vv[u].w, g[u].w, a, step_size, inv_bc2_sqrt);
        __stcs(reinterpret_cast<float4*>(p + eu), pv[u]);
        __stcs(reinterpret_cast<float4*>(m + eu), mv[u]);
        __stcs(reinterpret_cast<float4*>(v + eu), vv[u]);
        if (shadow != nullptr)                     // compute-dtype copy for the next gather
          *reinterpret_cast<uint2*>(shadow + eu) =
              make_uint2(pk2(pv[u].x, pv[u].y), pk2(pv[u].z, pv[u].w));
      }
    }
  };
  if (vec && base + kRsTile <= valid) {
#pragma unroll 1
    for (int64_t i = base + threadIdx.x * 4; i < base + kRsTile; i += kRsRound)
      vectors(std::integral_constant<int, kRsGroups>{}, i);
  } else {
    // The last tile of a segment (and so every segment that is shorter than a tile), or one that is not
    // aligned: element by element only what 16-byte accesses cannot reach.
    const int step = vec ? 4 : 1;
#pragma unroll 1
    for (int64_t i = base + threadIdx.x * step; i < end; i += kRsThreads * step) {
      if (vec && i + 3 < valid) {
        vectors(std::integral_constant<int, 1>{}, i);
        continue;
      }
      if (skip) break;
#pragma unroll 1
      for (int j = 0; j < step; ++j) {
        const int64_t e = sg.shard_off + i + j;
        float acc = 0.f;
        if (i + j < valid)
          for (int d = 0; d < n_src; ++d) {
            const int src = ((first + d) % n_src) * stride + offset;
            acc += full.p[src][sg.full_off + lo + i + j];
          }
        float g = acc * scale;
        if (accumulate) g += gshard[e];
        if (!in_place) gshard[e] = g;              // padding stays exactly zero: acc is 0 there
        bad |= !isfinite(g);
        if (i + j >= valid && g != 0.f) pad_bad = 1;
        if (ADAMW) {
          float pj = p[e], mj = m[e], vj = v[e];
          adamw_update(pj, mj, vj, g, a, step_size, inv_bc2_sqrt);
          p[e] = pj;                               // padding has p = g = m = v = 0 and stays 0
          m[e] = mj;
          v[e] = vj;
          if (shadow != nullptr) shadow[e] = __float2bfloat16(pj);
        }
      }
    }
  }
  if (flags != nullptr && __syncthreads_or(bad | pad_bad)) {
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(&flags[0], 1);
    if (__syncthreads_or(pad_bad) && threadIdx.x == 0) atomicOr(&flags[1], 1);
  }
}

__global__ void embedding_gather_sharded_kernel(PeerPtrs shards, int degree, int64_t q,
                                                const int64_t* __restrict__ ids,
                                                float* __restrict__ out, int cols) {
  const int64_t row = blockIdx.x;
  const int64_t id = ids[row];
  const int64_t base = id * cols;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const int64_t g = base + c;
    const int r = static_cast<int>(g / q);
    out[row * cols + c] = shards.p[r][g - r * q];
  }
}

struct VoidPeers {
  const void* p[kMaxPeers];
};

// out[b, r*sl + s, :] = peer r's x[b, s, :]   (16-byte vectors)
__global__ void seq_gather_kernel(VoidPeers peers, int degree, uint4* __restrict__ out, int batch,
                                  int seq_local, int64_t row_vec) {
  const int64_t per_peer = static_cast<int64_t>(batch) * seq_local * row_vec;
  const int64_t per_batch = seq_local * row_vec;
  const int64_t total = per_peer * degree;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  // four independent 16-byte loads in flight per thread: remote latency is several microseconds
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < total;
       i0 += 4 * stride) {
    uint4 v[4];
    int64_t dst[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t i = i0 + u * stride;
      dst[u] = -1;
      if (i < total) {
        const int r = static_cast<int>(i / per_peer);
        const int64_t j = i - r * per_peer;
        const int64_t b = j / per_batch;
        v[u] = reinterpret_cast<const uint4*>(peers.p[r])[j];
        dst[u] = (b * degree + r) * per_batch + (j - b * per_batch);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (dst[u] >= 0) out[dst[u]] = v[u];
  }
}

struct FloatPeers {
  const float* p[kMaxPeers];
};

// out[b, s, :] = residual[b, s, :] + sum_r partial_r[b, rank*sl + s, :]
__global__ void seq_reduce_scatter_kernel(FloatPeers peers, int degree, int rank,
                                          const float* __restrict__ residual,
                                          float* __restrict__ out, int batch, int seq_local,
                                          int cols) {
  const int64_t cv = cols / 4;
  const int64_t total = static_cast<int64_t>(batch) * seq_local * cv;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = i / (seq_local * cv);
    const int64_t rest = i - b * seq_local * cv;
    const int64_t src = (b * degree + rank) * seq_local * cv + rest;
    float4 acc = residual ? reinterpret_cast<const float4*>(residual)[i]
                          : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int d = 0; d < degree; ++d) {
      const int r = (rank + d) % degree;
      const float4 t = reinterpret_cast<const float4*>(peers.p[r])[src];
      acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
    }
    reinterpret_cast<float4*>(out)[i] = acc;
  }
}

struct FlagPeers {
  uint32_t* p[kMaxPeers];
};

// First expiry wins the status block: {code, silent peer, epoch waited for, epoch last seen}.
__device__ __forceinline__ void report_flag_timeout(int* status, int peer, uint32_t expected,
                                                    const uint32_t* flag) {
  if (atomicCAS(status, kOk, kErrPeerFlagWait) == kOk) {
    status[1] = peer;
    status[2] = static_cast<int>(expected);
    status[3] = static_cast<int>(*reinterpret_cast<const volatile uint32_t*>(flag));
  }
}

// Bounded wait for `*flag` to reach `epoch` (epochs only grow; the signed distance tolerates
// wrap-around).  The bound is a time budget read from the global nanosecond timer; the wait also
// ends as soon as the status word shows that something already failed.  Returns true when seen.
__device__ __forceinline__ bool wait_flag(const uint32_t* flag, uint32_t epoch, const int* status,
                                          uint64_t budget_ns) {
  uint32_t v;
  for (int i = 0; i < 64; ++i) {   // the common case: the peer is already there or nearly so
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (static_cast<int32_t>(v - epoch) >= 0) return true;
  }
  const uint64_t t0 = global_ns();
  for (;;) {
    for (int i = 0; i < 32; ++i) {
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      if (static_cast<int32_t>(v - epoch) >= 0) return true;
      __nanosleep(64);
    }
    if (status_failed(status)) return false;
    if (global_ns() - t0 > budget_ns) return false;
  }
}

// Thread t tells peer t "rank `rank` reached `epoch`" and then waits until peer t says the same.
// Pad layout: pad[slot * kMaxPeers + source_rank].  The wait is bounded in time; on expiry the
// status block is set and the kernel returns.  When a failure is already recorded on entry the
// kernel still publishes its own epoch (so that healthy peers are not held up by this rank) but
// does not wait: after one silent peer the barriers queued behind it return at once.
__global__ void peer_barrier_kernel(FlagPeers pads, int degree, int rank, uint32_t epoch, int slot,
                                    int* status, uint64_t budget_ns) {
  const int t = threadIdx.x;
  if (t >= degree) return;
  const bool failed_before = status_failed(status);
  __threadfence_system();
  uint32_t* remote = pads.p[t] + slot * kMaxPeers + rank;
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(remote), "r"(epoch) : "memory");
  if (failed_before) return;
  const uint32_t* mine = pads.p[rank] + slot * kMaxPeers + t;
  const bool seen = wait_flag(mine, epoch, status, budget_ns);
  if (!seen && status != nullptr) report_flag_timeout(status, t, epoch, mine);
  __threadfence_system();
}

// Small all-reduce (at most kMetricWidth doubles) in one kernel: thread t pushes this rank's
// vector into peer t's inbox and publishes the epoch, waits (bounded) for peer t's epoch, then
// the first n threads combine the inbox rows in rank order -- every rank computes the same bits.
// Element i is a SUM, or a MIN when bit i of min_mask is set.  Inboxes are double buffered on
// the epoch's parity: a rank can run at most one reduction ahead of its slowest peer.
// Inbox layout: [2][kMaxPeers][kMetricWidth] doubles.
constexpr int kMetricWidth = 16;
struct InboxPeers {
  double* p[kMaxPeers];
};

__global__ void peer_allreduce_small_kernel(FlagPeers pads, InboxPeers inboxes, int degree, int rank,
                                            uint32_t epoch, int slot, const double* __restrict__ in,
                                            double* __restrict__ out, int n, uint32_t min_mask,
                                            int* status, uint64_t budget_ns) {
  const int t = threadIdx.x;
  const int parity = static_cast<int>(epoch & 1u);
  if (t < degree) {
    const bool failed_before = status_failed(status);
    double* dst = inboxes.p[t] + (static_cast<int64_t>(parity) * kMaxPeers + rank) * kMetricWidth;
    for (int i = 0; i < n; ++i) dst[i] = in[i];
    __threadfence_system();
    uint32_t* remote = pads.p[t] + slot * kMaxPeers + rank;
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(remote), "r"(epoch) : "memory");
    if (!failed_before) {
      const uint32_t* mine = pads.p[rank] + slot * kMaxPeers + t;
      const bool seen = wait_flag(mine, epoch, status, budget_ns);
      if (!seen && status != nullptr) report_flag_timeout(status, t, epoch, mine);
    }
    __threadfence_system();
  }
  __syncthreads();
  if (t < n) {
    const volatile double* rows =
        inboxes.p[rank] + static_cast<int64_t>(parity) * kMaxPeers * kMetricWidth;
    double acc = rows[t];
    for (int r = 1; r < degree; ++r) {
      const double v = rows[r * kMetricWidth + t];
      acc = ((min_mask >> t) & 1u) ? fmin(acc, v) : acc + v;
    }
    out[t] = acc;
  }
}

bool fill_table(SegTable* t, const SegmentDesc* segs, int n) {
  if (n < 1 || n > kMaxSegs) return false;
  for (int i = 0; i < n; ++i) t->s[i] = segs[i];
  t->n = n;
  return true;
}

int g_ctas_per_sm = 0;   // 0: read STB_COLLECTIVE_CTAS_PER_SM once (default below)
int chunks_for(const SegmentDesc* segs, int n) {
  if (g_ctas_per_sm == 0) {
    const char* env = getenv("STB_COLLECTIVE_CTAS_PER_SM");
    g_ctas_per_sm = env != nullptr ? std::max(1, atoi(env)) : 48;   // measured: 8..48 equal, 4 slower
  }
  const int kCtasPerSm = g_ctas_per_sm;
  // grid.x of the gather's (chunks, segments) grid.  The kernel loops over chunks, so the grid only
  // has to be large enough to keep the memory system busy; STB_COLLECTIVE_CTAS_PER_SM bounds the total
  // (CTAs per SM over all segments).
  int64_t most = 1;
  for (int i = 0; i < n; ++i) {
    most = std::max<int64_t>(most, (segs[i].numel + kChunk - 1) / kChunk);
  }
  const int64_t budget = std::max<int64_t>(1, (sm_count() * kCtasPerSm) / std::max(1, n));
  // and never more than four CTAs per SM for one segment: more only adds scheduling work
  return static_cast<int>(std::min<int64_t>({most, budget, static_cast<int64_t>(sm_count() * 4)}));
}

// One tile after the other over all segments; false when the table or the grid does not fit.
bool fill_tiles(RsTable* t, const SegmentDesc* segs, int n) {
  if (n < 1 || n > kMaxSegs) return false;
  int64_t tiles = 0;
  for (int i = 0; i < n; ++i) {
    t->s[i] = segs[i];
    t->first[i] = static_cast<int>(tiles);
    tiles += (segs[i].q + kRsTile - 1) / kRsTile;
    if (segs[i].q < 0 || tiles > INT32_MAX) return false;
  }
  t->first[n] = static_cast<int>(tiles);
  t->n = n;
  return true;
}

}  // namespace

cudaError_t launch_gather_params(PeerPtrs shards, int degree, const SegmentDesc* segs, int n_segs,
                                 void* full_bf16, float* full_fp32, int64_t total_full,
                                 cudaStream_t s, const void* const* shadows) {
  (void)total_full;
  SegTable tab;
  if (degree < 1 || degree > kMaxPeers || !fill_table(&tab, segs, n_segs))
    return cudaErrorInvalidValue;
  ShadowPtrs sh{};
  if (shadows != nullptr)
    for (int i = 0; i < degree; ++i) {
      if (shadows[i] == nullptr || (reinterpret_cast<uintptr_t>(shadows[i]) & 15))
        return cudaErrorInvalidValue;
      sh.p[i] = reinterpret_cast<const __nv_bfloat16*>(shadows[i]);
    }
  dim3 grid(chunks_for(segs, n_segs), n_segs);
  gather_params_kernel<<<grid, 256, 0, s>>>(shards, sh, shadows != nullptr ? 1 : 0, degree, tab,
                                            reinterpret_cast<__nv_bfloat16*>(full_bf16), full_fp32);
  count_launch();
  return cudaGetLastError();
}

bool valid_mesh(int degree, int rank, TpAxis tp) {
  return degree >= 1 && tp.degree >= 1 && degree * tp.degree <= kMaxPeers && rank >= 0 &&
         rank < degree && tp.rank >= 0 && tp.rank < tp.degree;
}

cudaError_t launch_reduce_scatter_grads(PeerPtrs full_grads, int degree, int rank,
                                        const SegmentDesc* segs, int n_segs, float* grad_shard,
                                        int64_t shard_total, float scale, bool accumulate,
                                        int* flags, cudaStream_t s, TpAxis tp, const int* status,
                                        const float* multicast) {
  (void)shard_total;
  RsTable tab;
  if (!valid_mesh(degree, rank, tp) || !fill_tiles(&tab, segs, n_segs) ||
      (reinterpret_cast<uintptr_t>(multicast) & 15))
    return cudaErrorInvalidValue;
  if (tab.first[n_segs] == 0) return cudaSuccess;
  auto kernel = degree * tp.degree == 1 && multicast == nullptr ? reduce_scatter_kernel<false, true>
                                                                : reduce_scatter_kernel<false, false>;
  kernel<<<tab.first[n_segs], kRsThreads, 0, s>>>(
      full_grads, degree, rank, tp.degree, tp.rank, tab, grad_shard, nullptr, nullptr, nullptr,
      scale, tp.replicated_scale, accumulate ? 1 : 0, AdamWArgs{}, flags, nullptr, status,
      multicast);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_reduce_scatter_adamw(PeerPtrs full_grads, int degree, int rank,
                                        const SegmentDesc* segs, int n_segs, float* grad_shard,
                                        float* p, float* m, float* v, int64_t shard_total,
                                        float scale, bool accumulate, AdamWArgs a, int* flags,
                                        cudaStream_t s, TpAxis tp, void* shadow, const int* status,
                                        const float* multicast) {
  (void)shard_total;
  RsTable tab;
  if (!valid_mesh(degree, rank, tp) || !fill_tiles(&tab, segs, n_segs) ||
      (reinterpret_cast<uintptr_t>(multicast) & 15))
    return cudaErrorInvalidValue;
  if (tab.first[n_segs] == 0) return cudaSuccess;
  auto kernel = degree * tp.degree == 1 && multicast == nullptr ? reduce_scatter_kernel<true, true>
                                                                : reduce_scatter_kernel<true, false>;
  kernel<<<tab.first[n_segs], kRsThreads, 0, s>>>(
      full_grads, degree, rank, tp.degree, tp.rank, tab, grad_shard, p, m, v, scale,
      tp.replicated_scale, accumulate ? 1 : 0, a, flags,
      reinterpret_cast<__nv_bfloat16*>(shadow), status, multicast);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_embedding_gather_sharded(PeerPtrs shards, int degree, int64_t q,
                                            const int64_t* ids, float* out, int rows, int cols,
                                            cudaStream_t s) {
  if (degree < 1 || degree > kMaxPeers || q < 1) return cudaErrorInvalidValue;
  embedding_gather_sharded_kernel<<<rows, 256, 0, s>>>(shards, degree, q, ids, out, cols);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_seq_gather(const void* const* peers, int degree, void* out, int batch,
                              int seq_local, int64_t row_bytes, cudaStream_t s) {
  if (degree < 1 || degree > kMaxPeers || row_bytes % 16) return cudaErrorInvalidValue;
  VoidPeers vp;
  for (int i = 0; i < degree; ++i) vp.p[i] = peers[i];
  const int64_t total = static_cast<int64_t>(batch) * seq_local * (row_bytes / 16) * degree;
  const int grid = static_cast<int>(std::min<int64_t>((total + 1023) / 1024, sm_count() * 8));
  seq_gather_kernel<<<grid, 256, 0, s>>>(vp, degree, reinterpret_cast<uint4*>(out), batch,
                                         seq_local, row_bytes / 16);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_seq_reduce_scatter_f32(const float* const* peers, int degree, int rank,
                                          const float* residual, float* out, int batch,
                                          int seq_local, int cols, cudaStream_t s) {
  if (degree < 1 || degree > kMaxPeers || cols % 4) return cudaErrorInvalidValue;
  FloatPeers fp;
  for (int i = 0; i < degree; ++i) fp.p[i] = peers[i];
  const int64_t total = static_cast<int64_t>(batch) * seq_local * (cols / 4);
  const int grid = static_cast<int>(std::min<int64_t>((total + 255) / 256, sm_count() * 8));
  seq_reduce_scatter_kernel<<<grid, 256, 0, s>>>(fp, degree, rank, residual, out, batch, seq_local,
                                                 cols);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_peer_allreduce_small(uint32_t* const* flag_pads, double* const* inboxes, int degree,
                                        int rank, uint32_t epoch, int slot, const double* in,
                                        double* out, int n, uint32_t min_mask, int* status,
                                        uint64_t budget_ns, cudaStream_t s) {
  if (degree < 1 || degree > kMaxPeers || rank < 0 || rank >= degree || n < 1 || n > kMetricWidth)
    return cudaErrorInvalidValue;
  FlagPeers fp;
  InboxPeers ip;
  for (int i = 0; i < degree; ++i) {
    fp.p[i] = flag_pads[i];
    ip.p[i] = inboxes[i];
  }
  peer_allreduce_small_kernel<<<1, 32, 0, s>>>(fp, ip, degree, rank, epoch, slot, in, out, n,
                                               min_mask, status, budget_ns);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_peer_barrier(uint32_t* const* flag_pads, int degree, int rank, uint32_t epoch,
                                int slot, int* status, uint64_t budget_ns, cudaStream_t s) {
  if (degree < 1 || degree > kMaxPeers || rank < 0 || rank >= degree)
    return cudaErrorInvalidValue;
  FlagPeers fp;
  for (int i = 0; i < degree; ++i) fp.p[i] = flag_pads[i];
  peer_barrier_kernel<<<1, 32, 0, s>>>(fp, degree, rank, epoch, slot, status, budget_ns);
  count_launch();
  return cudaGetLastError();
}

}  // namespace stb

// Causal grouped-query attention for head_dim 128 on sm_100a: forward, and backward as two
// kernels (dK/dV per key block, dQ per query block).  All five/seven matrix products run on
// tcgen05 with accumulators in TMEM; Q/K/V/dO tiles arrive by TMA from the packed, rope-applied
// qkv buffer; the softmax warps read scores from TMEM with tcgen05.ld and hand P / dS back to the
// tensor core as TMEM operands.  No S x S matrix ever reaches global memory (the reference materialises
// it: src/sharded_runtime/models/qwen2.py:247-257).
//
// Tile = 128 x 128 (rows x head_dim or rows x rows) bf16, held as two 64-column halves of 16 KB
// (128 rows x 128 bytes, TMA SWIZZLE_128B).  The same tile serves as a K-major operand (reduction
// over its columns) or an MN-major operand (reduction over its rows); only the descriptor differs.
//
// Warp 0 = TMA producer, warp 1 = MMA issuer / TMEM owner, the others = softmax: 4 warps with a row
// per thread forward, 8 warps with half a row per thread backward.
// Every mbarrier wait is bounded; on expiry the status word is set and the roles fall through.  Whether
// they do or not, the producer and the MMA warp leave only after the copies and commits that they issued
// have landed.
#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace stb {

bool make_bf16_tensor_map(CUtensorMap* map, const void* base, int64_t rows, int64_t cols,
                          int64_t ld, int box_cols, int box_rows);

namespace {

constexpr int kD = 128;          // head dim
constexpr int kBlk = 128;        // rows per tile
constexpr int kHalf = 16384;     // bytes of one 64-column half tile
constexpr int kTile = 2 * kHalf;
constexpr int kFwdThreads = 192;     // producer, MMA and 4 softmax warps (one row per thread)
constexpr int kBwdThreads = 320;     // producer, MMA and 8 softmax warps (half a row per thread)

// k-th 16-wide reduction slice of a tile used K-major (reduce over columns).
__device__ __forceinline__ uint64_t desc_k(uint32_t tile, int kk) {
  return make_smem_desc_sw128(tile + (kk >> 2) * kHalf + (kk & 3) * 32, 16, 1024);
}
// k-th 16-row reduction slice of a tile used MN-major (reduce over rows).
__device__ __forceinline__ uint64_t desc_mn(uint32_t tile, int kk) {
  return make_smem_desc_sw128(tile + kk * 2048, kHalf, 1024);
}

// The MMAs below are issued by a warp that stays converged, one elected lane doing the work: then
// addresses and descriptors are warp-uniform.  (Issued inside `if (lane == 0)` an MMA cost about 136
// clocks whatever its size.)  Where an MMA overwrites columns of TMEM that the one before it reads as its
// A operand, the kernels take it that MMAs issued by one thread run in that order.

// D[128x128] = A B^T over a 128-long reduction, both tiles K-major: 8 MMAs of K = 16.
__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint32_t a_tile, uint32_t b_tile) {
  constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    tc_mma_f16(tmem_d, desc_k(a_tile, kk), desc_k(b_tile, kk), idesc, kk > 0 ? 1u : 0u);
}
// D[128x128] (+)= A B with A (bf16, 128 x 128) in TMEM and B MN-major in shared memory.  The first
// 64 columns of A are packed at tmem_a, the last 64 at tmem_a + second_half.
__device__ __forceinline__ void mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t second_half,
                                       uint32_t b_tile, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, true);
#pragma unroll
  for (int kk = 0; kk < 8; ++kk)
    tc_mma_f16_ts(tmem_d, tmem_a + (kk >> 2) * second_half + (kk & 3) * 8, desc_mn(b_tile, kk), idesc,
                  (accumulate || kk > 0) ? 1u : 0u);
}

// TMA: one 128x128 tile = two boxes of 64 columns.
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar,
                                          int col, int row) {
  tma_load_2d(dst, map, bar, col, row);
  tma_load_2d(dst + kHalf, map, bar, col + 64, row);
}

// Writes this warp's 32 x 128 bf16 block through shared memory: row `lane` is stored swizzled at
// stage + lane * 256 (8 KB per warp) by put, then leaves as whole 256-byte rows.
struct RowStager {
  uint8_t* stage;
  int lane;
  __device__ __forceinline__ void put(int c16, uint4 v) const {   // 16-byte piece c16 (0..15) of the row
    *reinterpret_cast<uint4*>(stage + lane * 256 + ((c16 ^ (lane & 7)) << 4)) = v;
  }
  // rows row0 .. row0 + n_rows - 1 of the block go to base + row * pitch elements
  __device__ __forceinline__ void flush(__nv_bfloat16* base, int64_t pitch, int n_rows) const {
    __syncwarp();
    const int piece = lane & 15;
#pragma unroll 4
    for (int r = lane >> 4; r < n_rows; r += 2)
      *reinterpret_cast<uint4*>(base + r * pitch + piece * 8) =
          *reinterpret_cast<const uint4*>(stage + r * 256 + ((piece ^ (r & 7)) << 4));
    __syncwarp();
  }
};

__device__ __forceinline__ uint4 pack8(const uint32_t* v, float scale) {
  uint4 pk;
  pk.x = pack_bf16x2(__uint_as_float(v[0]) * scale, __uint_as_float(v[1]) * scale);
  pk.y = pack_bf16x2(__uint_as_float(v[2]) * scale, __uint_as_float(v[3]) * scale);
  pk.z = pack_bf16x2(__uint_as_float(v[4]) * scale, __uint_as_float(v[5]) * scale);
  pk.w = pack_bf16x2(__uint_as_float(v[6]) * scale, __uint_as_float(v[7]) * scale);
  return pk;
}
__device__ __forceinline__ uint4 pack8(const uint32_t* v) {
  uint4 pk;
  pk.x = pack_bf16x2(__uint_as_float(v[0]), __uint_as_float(v[1]));
  pk.y = pack_bf16x2(__uint_as_float(v[2]), __uint_as_float(v[3]));
  pk.z = pack_bf16x2(__uint_as_float(v[4]), __uint_as_float(v[5]));
  pk.w = pack_bf16x2(__uint_as_float(v[6]), __uint_as_float(v[7]));
  return pk;
}

// End of the MMA warp: one more commit, behind every MMA issued so far, committed or not.
__device__ __forceinline__ void commit_all(uint64_t* idle) {
  if (elect_one()) tc_commit(idle);
  __syncwarp();
}

struct FwdParams {
  __nv_bfloat16* out;
  float* lse;
  const uint8_t* key_mask;
  int batch, seq, hq, hkv;
  float scale;
  int* status;
  const uint32_t* key_bits;   // packed key mask (bit i of word w = key 32 w + i), see pack_key_mask
  int bits_pitch;             // words per sample, a multiple of 4
};

// The 128 mask bits of key block j of sample b; all ones without a mask.  With a byte mask the
// bits are assembled on the fly (slow path kept for callers that did not pack the mask).
__device__ __forceinline__ void load_key_bits(const uint32_t* bits, int pitch, const uint8_t* bytes,
                                              int seq, int b, int j, uint32_t (&w)[4]) {
  if (bits != nullptr) {
    const uint4 v = *reinterpret_cast<const uint4*>(bits + static_cast<int64_t>(b) * pitch + j * 4);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else if (bytes != nullptr) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t word = 0;
      for (int i = 0; i < 32; ++i) {
        const int kv = j * 128 + c * 32 + i;
        word |= (kv < seq && bytes[static_cast<int64_t>(b) * seq + kv] != 0) ? (1u << i) : 0u;
      }
      w[c] = word;
    }
  } else {
    w[0] = w[1] = w[2] = w[3] = 0xffffffffu;
  }
}

// Forward: one CTA per (query block, head, sample), two CTAs per SM.  The chain of a key block is
//   S = Q K^T -> softmax -> O += P V,
// serial inside a CTA; the second CTA of the SM fills the gaps (tensor pipe under the other's
// exponentials and the other way round).  To fit twice, a CTA keeps S and O in 256 TMEM columns,
// with P (bf16) written over the S it came from and read by the MMA as a TMEM operand, and one
// stage each of K and V: 97 KB of shared memory.  CTAs start with the longest rows of blocks, so
// the short ones fill the last wave.
// Bound by the latency of the chain, not by a pipe: at 2 x 2048 (12 heads) the tensor pipe is active
// 24 % of the cycles, the exponentials' unit 24 %, issue slots are used to 35 %, and warps mostly wait
// for TMEM loads and barriers.  At 1 x 8192 a block takes 2300 to 3200 clocks of an SM (1.4 to 1.965
// GHz); its exponentials need 1024, its products 1024.
// Measured on B200 (12 heads): 1 x 8192, causal, 1576 us before (one CTA per SM, MMAs issued from
// one lane, P through shared memory) and 269 us now; 8 x 512: 100 and 31 us.
// smem: Q | K | V | barriers
constexpr int kFwdSmem = 3 * kTile + 1024 + 128;

__global__ void __launch_bounds__(kFwdThreads, 2)
attention_fwd_kernel(const __grid_constant__ CUtensorMap map, FwdParams p) {
  extern __shared__ uint8_t raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kTile;
  uint8_t* sV = sK + kTile;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kTile);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 2;
  uint64_t* v_full = bars + 3;
  uint64_t* v_empty = bars + 4;
  uint64_t* s_full = bars + 5;
  uint64_t* p_full = bars + 6;        // 128 arrivals
  uint64_t* o_done = bars + 7;
  uint64_t* idle = bars + 8;          // every MMA is over
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + kBlk - 1) / kBlk;
  const int qb = nblk - 1 - static_cast<int>(blockIdx.x) / (p.hq * p.batch);
  const int hb = static_cast<int>(blockIdx.x) % (p.hq * p.batch);
  const int h = hb % p.hq, b = hb / p.hq;
  const int hk = h / (p.hq / p.hkv);
  const int n_kv = qb + 1;  // causal: key blocks 0..qb
  const int row0 = b * p.seq;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 9; ++i) mbar_init(bars + i, i == 6 ? 128 : 1);
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&map);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  chain_wait();                       // what is above ran under the kernel before
  // (asked in a step of its own: together with the barrier above, the loops below were compiled slower,
  // 1 x 8192 in 299 instead of 269 us)
  if (kernel_should_skip(p.status)) { // an earlier kernel already failed
    if (warp == 1) tmem_dealloc(tmem, 256);
    return;
  }
  const uint32_t tS = tmem, tO = tmem + 128;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, kTile);
      load_tile(sQ, &map, q_full, h * kD, row0 + qb * kBlk);
    }
    __syncwarp();
    int k_loads = 0, v_loads = 0;
    for (int j = 0; j < n_kv; ++j) {
      if (!mbar_wait_warp(k_empty, (j & 1) ^ 1, p.status, kErrAttnWait)) break;
      if (elect_one()) {
        mbar_expect_tx(k_full, kTile);
        load_tile(sK, &map, k_full, (p.hq + hk) * kD, row0 + j * kBlk);
      }
      __syncwarp();
      ++k_loads;
      if (!mbar_wait_warp(v_empty, (j & 1) ^ 1, p.status, kErrAttnWait)) break;
      if (elect_one()) {
        mbar_expect_tx(v_full, kTile);
        load_tile(sV, &map, v_full, (p.hq + p.hkv + hk) * kD, row0 + j * kBlk);
      }
      __syncwarp();
      ++v_loads;
    }
    if (elect_one()) chain_release();
    // q_full, k_full, -, v_full
    mbar_drain(bars + lane, lane == 0 ? 1 : lane == 1 ? k_loads : lane == 3 ? v_loads : 0, p.status);
  } else if (warp == 1) {
    const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aV = smem_u32(sV);
    bool ok = mbar_wait_warp(q_full, 0, p.status, kErrAttnWait);
    int s_done = 0, pv_done = 0;
    for (int j = 0; j < n_kv && ok; ++j) {
      // S(j) may overwrite P(j-1): MMAs run in issue order, so P V of block j-1 has read it
      ok = mbar_wait_warp(k_full, j & 1, p.status, kErrAttnWait);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ss(tS, aQ, aK);                                          // S = Q K^T
        tc_commit(k_empty);
        tc_commit(s_full);
      }
      __syncwarp();
      ++s_done;
      ok = mbar_wait_warp(p_full, j & 1, p.status, kErrAttnWait) &&  // P in TMEM, O rescaled
           mbar_wait_warp(v_full, j & 1, p.status, kErrAttnWait);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ts(tO, tS, 32, aV, j > 0);                               // O += P V
        tc_commit(v_empty);
        if (j + 1 == n_kv) tc_commit(o_done);
      }
      __syncwarp();
      ++pv_done;
    }
    commit_all(idle);
    // k_empty, s_full; v_empty; o_done; idle
    mbar_drain(bars + lane, lane == 2 || lane == 5 ? s_done : lane == 4 ? pv_done
                            : lane == 7 ? pv_done == n_kv : lane == 8, p.status);
  } else {
    const int q = warp & 3;
    const int r = q * 32 + lane;                 // row inside the tile
    const int q_idx = qb * kBlk + r;             // position inside the sequence
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv && ok; ++j) {
      // the block's 128 key-mask bits (one 16-byte load, the same address for the whole warp), cut
      // at the diagonal; a block with every key visible takes the mask-free path
      uint32_t mw[4];
      load_key_bits(p.key_bits, p.bits_pitch, p.key_mask, p.seq, b, j, mw);
      const bool plain = j != qb && (mw[0] & mw[1] & mw[2] & mw[3]) == 0xffffffffu;
      if (j == qb) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int n = r + 1 - c * 32;          // keys c*32 .. of this row up to its own position
          mw[c] &= n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u);
        }
      }
      ok = __all_sync(0xffffffffu, mbar_wait(s_full, j & 1, p.status, kErrAttnWait));
      if (!ok) break;
      tc_fence_after_sync();                      // also: P V of block j-1 is done (issue order)
      float alpha = 1.f, sum = 0.f;
      auto block = [&](auto masked) {
        constexpr bool kMasked = decltype(masked)::value;
        float mx = -INFINITY;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t s[64];
          tmem_ld_32x32(tS + lane_base + g * 64, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
          tmem_ld_32x32(tS + lane_base + g * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
          tmem_ld_wait();
          float part[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four chains of maxima
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            float x = __uint_as_float(s[i]) * p.scale;
            if (kMasked) x = ((mw[g * 2 + (i >> 5)] >> (i & 31)) & 1u) ? x : -INFINITY;
            part[i & 3] = fmaxf(part[i & 3], x);
          }
          mx = fmaxf(mx, fmaxf(fmaxf(part[0], part[1]), fmaxf(part[2], part[3])));
        }
        const float m_new = fmaxf(m, mx);
        const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
        alpha = (m == -INFINITY) ? 0.f : __expf(m - m_use);
        m = m_new;
        // probabilities, rounded to bf16: what the tensor core will see is also what is summed
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t s[32], pk[16];
          tmem_ld_32x32(tS + lane_base + c * 32, s);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float x0 = __uint_as_float(s[i]) * p.scale, x1 = __uint_as_float(s[i + 1]) * p.scale;
            if (kMasked) {
              x0 = ((mw[c] >> i) & 1u) ? x0 : -INFINITY;            // exp gives 0
              x1 = ((mw[c] >> (i + 1)) & 1u) ? x1 : -INFINITY;
            }
            // (rounded product minus m_use: no multiply-add, so both paths round alike)
            const uint32_t e = pack_bf16x2(__expf(__fadd_rn(x0, -m_use)), __expf(__fadd_rn(x1, -m_use)));
            pk[i >> 1] = e;
            sum += __uint_as_float(e << 16) + __uint_as_float(e & 0xffff0000u);
          }
          // columns 16 c .. of S, read above, make room for P
          tmem_st_32x16(tS + lane_base + c * 16, pk);
        }
      };
      if (plain)
        block(std::false_type{});
      else
        block(std::true_type{});
      if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t o[64];
          tmem_ld_32x32(tO + lane_base + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
          tmem_ld_32x32(tO + lane_base + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 64; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(tO + lane_base + c * 64, *reinterpret_cast<uint32_t(*)[32]>(&o[0]));
          tmem_st_32x32(tO + lane_base + c * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&o[32]));
        }
      }
      l = l * alpha + sum;
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(p_full);
    }
    // epilogue: O / l -> bf16, through the Q tile (every S = Q K^T is done with it)
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(o_done, 0, p.status, kErrAttnWait));
    tc_fence_after_sync();
    const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
    const RowStager rows{sQ + q * 8192, lane};
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld_32x32(tO + lane_base + c * 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 4; ++g) rows.put(c * 4 + g, pack8(&v[8 * g], inv_l));
    }
    const int first = qb * kBlk + q * 32;
    if (ok) {
      rows.flush(p.out + (static_cast<int64_t>(row0 + first) * p.hq + h) * kD,
                 static_cast<int64_t>(p.hq) * kD, min(32, p.seq - first));
      if (q_idx < p.seq)
        p.lse[(static_cast<int64_t>(b) * p.hq + h) * p.seq + q_idx] = (l > 0.f) ? m + __logf(l) : 0.f;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 256);
  }
}

// delta[b, h, s] = sum_d dO[b, s, h, d] * O[b, s, h, d]   (one warp per (row, head))
__global__ void attention_delta_kernel(const __nv_bfloat16* out, const __nv_bfloat16* dout, float* delta,
                                       int batch, int seq, int hq) {
  chain_wait();
  chain_release();
  const int64_t w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t total = static_cast<int64_t>(batch) * seq * hq;
  if (w >= total) return;
  const int64_t row = w / hq;
  const int h = static_cast<int>(w % hq);
  const uint2 a = *reinterpret_cast<const uint2*>(out + w * kD + lane * 4);
  const uint2 g = *reinterpret_cast<const uint2*>(dout + w * kD + lane * 4);
  const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
  const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
  const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g.x));
  const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g.y));
  float s = a0.x * g0.x + a0.y * g0.y + a1.x * g1.x + a1.y * g1.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const int64_t b = row / seq, sidx = row % seq;
    delta[(b * hq + h) * seq + sidx] = s;
  }
}

struct BwdParams {
  const float* lse;
  const float* delta;
  __nv_bfloat16* dqkv;
  const uint8_t* key_mask;
  int batch, seq, hq, hkv;
  float scale;
  int* status;
  float* dkv_part;   // [parts, batch*seq, 2*hkv*128] fp32 partial dK|dV when the group is split
  int parts;         // CTAs sharing one kv head's query-head group (1: write bf16 directly)
  const uint32_t* key_bits;
  int bits_pitch;
};

// ---------------------------------------------------------------------------- dQ
// One CTA per (query block, query head, batch).  Per key block j <= i:
//   S = Q K^T, dP = dO V^T  ->  dS = P * (dP - delta) * scale  ->  dQ += dS K.
// S is double buffered in TMEM and dS (bf16) is written over the S it came from, each half row into
// its own 64 columns, and read by the MMA as a TMEM operand.  While the softmax warps work on block
// j, S(j+1) runs; when they are done, dP(j+1) goes first and dQ += dS(j) K(j) and S(j+2) run under
// the softmax of block j+1, so the chain of a block is dP and half a row of exponentials per
// thread.  K has three stages (K(j) is held until dQ), V two.
// The chain is still what bounds it: at 2 x 2048 (12 heads) the tensor pipe is active 34 % of the cycles,
// the exponentials' unit 23 %, issue slots are used to 28 %.  At 1 x 8192 a block takes 3100 to 4300
// clocks (1.4 to 1.965 GHz); its products need 1536.
// Measured on B200 inside a training step (12 heads): 1 x 8192: 764 us before (serial chain, one
// thread per row, MMAs issued from one lane) and 371 us now; 8 x 512: 51 and 38 us.
// smem: Q | dO | K x 3 | V x 2 | barriers
constexpr int kDqSmem = 7 * kTile + 1024 + 256;

__global__ void __launch_bounds__(kBwdThreads, 1)
attention_dq_kernel(const __grid_constant__ CUtensorMap map_qkv,
                    const __grid_constant__ CUtensorMap map_do, BwdParams p) {
  extern __shared__ uint8_t raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + kTile;
  uint8_t* sK = sdO + kTile;          // 3 stages
  uint8_t* sV = sK + 3 * kTile;       // 2 stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * kTile);
  uint64_t* q_full = bars;
  uint64_t* sdp_full = bars + 1;
  uint64_t* ds_full = bars + 2;   // 256 arrivals
  uint64_t* dq_done = bars + 3;
  uint64_t* k_full = bars + 4;    // 3
  uint64_t* k_empty = bars + 7;   // 3
  uint64_t* v_full = bars + 10;   // 2
  uint64_t* v_empty = bars + 12;  // 2
  uint64_t* idle = bars + 14;     // every MMA is over
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (p.seq + kBlk - 1) / kBlk;
  const int qb = nblk - 1 - static_cast<int>(blockIdx.x) / (p.hq * p.batch);   // long rows first
  const int hb = static_cast<int>(blockIdx.x) % (p.hq * p.batch);
  const int h = hb % p.hq, b = hb / p.hq;
  const int hk = h / (p.hq / p.hkv);
  const int n_kv = qb + 1;
  const int row0 = b * p.seq;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 15; ++i) mbar_init(bars + i, i == 2 ? 256 : 1);
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&map_qkv);
    prefetch_tensormap(&map_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  chain_wait();                       // what is above ran under the kernel before
  if (kernel_should_skip(p.status)) { // an earlier kernel already failed
    if (warp == 1) tmem_dealloc(tmem, 512);
    return;
  }
  const uint32_t tS = tmem, tdP = tmem + 256, tdQ = tmem + 384;   // S: two buffers

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, 2 * kTile);
      load_tile(sQ, &map_qkv, q_full, h * kD, row0 + qb * kBlk);
      load_tile(sdO, &map_do, q_full, h * kD, row0 + qb * kBlk);
    }
    __syncwarp();
    int k_loads = 0, v_loads = 0;
    for (int j = 0; j < n_kv; ++j) {
      const int ks = j % 3, vs = j & 1;
      if (!mbar_wait_warp(&k_empty[ks], ((j / 3) & 1) ^ 1, p.status, kErrAttnWait)) break;
      if (elect_one()) {
        mbar_expect_tx(&k_full[ks], kTile);
        load_tile(sK + ks * kTile, &map_qkv, &k_full[ks], (p.hq + hk) * kD, row0 + j * kBlk);
      }
      __syncwarp();
      ++k_loads;
      if (!mbar_wait_warp(&v_empty[vs], ((j >> 1) & 1) ^ 1, p.status, kErrAttnWait)) break;
      if (elect_one()) {
        mbar_expect_tx(&v_full[vs], kTile);
        load_tile(sV + vs * kTile, &map_qkv, &v_full[vs], (p.hq + p.hkv + hk) * kD, row0 + j * kBlk);
      }
      __syncwarp();
      ++v_loads;
    }
    if (elect_one()) chain_release();
    // q_full; k_full[3]; v_full[2]
    mbar_drain(bars + lane, lane == 0 ? 1 : lane >= 4 && lane < 7 ? ring_uses(k_loads, 3, lane - 4)
                            : lane == 10 || lane == 11 ? ring_uses(v_loads, 2, lane - 10) : 0, p.status);
  } else if (warp == 1) {
    const uint32_t aQ = smem_u32(sQ), adO = smem_u32(sdO), aK = smem_u32(sK), aV = smem_u32(sV);
    auto scores = [&](int j) {        // S(j) = Q K(j)^T
      if (!mbar_wait_warp(&k_full[j % 3], (j / 3) & 1, p.status, kErrAttnWait)) return false;
      tc_fence_after_sync();
      if (elect_one()) mma_ss(tS + (j & 1) * 128, aQ, aK + (j % 3) * kTile);
      __syncwarp();
      return true;
    };
    int dp_done = 0, dq_count = 0;
    auto dprobs = [&](int j) {        // dP(j) = dO V(j)^T; with it S(j), issued earlier, is complete too
      if (!mbar_wait_warp(&v_full[j & 1], (j >> 1) & 1, p.status, kErrAttnWait)) return false;
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ss(tdP, adO, aV + (j & 1) * kTile);
        tc_commit(&v_empty[j & 1]);
        tc_commit(sdp_full);
      }
      __syncwarp();
      ++dp_done;
      return true;
    };
    bool ok = mbar_wait_warp(q_full, 0, p.status, kErrAttnWait);
    ok = ok && scores(0) && dprobs(0);
    if (ok && n_kv > 1) ok = scores(1);
    for (int j = 0; j < n_kv && ok; ++j) {
      ok = mbar_wait_warp(ds_full, j & 1, p.status, kErrAttnWait);   // dS(j) written, dP(j) read
      if (!ok) break;
      tc_fence_after_sync();
      if (j + 1 < n_kv) ok = dprobs(j + 1);
      if (!ok) break;
      if (elect_one()) {
        mma_ts(tdQ, tS + (j & 1) * 128, 64, aK + (j % 3) * kTile, j > 0);   // dQ += dS K
        tc_commit(&k_empty[j % 3]);
        if (j + 1 == n_kv) tc_commit(dq_done);
      }
      __syncwarp();
      ++dq_count;
      if (j + 2 < n_kv) ok = scores(j + 2);     // over dS(j), which the MMA before has read
    }
    commit_all(idle);
    // sdp_full; dq_done; k_empty[3]; v_empty[2]; idle
    mbar_drain(bars + lane, lane == 1 ? dp_done : lane == 3 ? dq_count == n_kv
                            : lane >= 7 && lane < 10 ? ring_uses(dq_count, 3, lane - 7)
                            : lane == 12 || lane == 13 ? ring_uses(dp_done, 2, lane - 12) : lane == 14, p.status);
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;   // rows 32 q .., columns 64 half ..
    const int r = q * 32 + lane;
    const int q_idx = qb * kBlk + r;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    const bool q_ok = q_idx < p.seq;
    const int64_t stat = (static_cast<int64_t>(b) * p.hq + h) * p.seq + min(q_idx, p.seq - 1);
    const float lse = p.lse[stat], dlt = p.delta[stat];
    bool ok = true;
    for (int j = 0; j < n_kv && ok; ++j) {
      uint32_t mw[4];
      load_key_bits(p.key_bits, p.bits_pitch, p.key_mask, p.seq, b, j, mw);
      uint32_t word[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        word[c] = half ? mw[2 + c] : mw[c];
        if (j == qb) {
          const int n = r + 1 - (half * 64 + c * 32);
          word[c] &= n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u);
        }
        if (!q_ok) word[c] = 0;
      }
      ok = __all_sync(0xffffffffu, mbar_wait(sdp_full, j & 1, p.status, kErrAttnWait));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t tSj = tS + (j & 1) * 128 + lane_base + half * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32], d[32], pk[16];
        tmem_ld_32x32(tSj + c * 32, s);
        tmem_ld_32x32(tdP + lane_base + half * 64 + c * 32, d);
        tmem_ld_wait();
        const bool all_on = __all_sync(0xffffffffu, word[c] == 0xffffffffu);
        float ds[32];
        if (all_on) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float pr = __expf(__uint_as_float(s[i]) * p.scale - lse);
            ds[i] = pr * (__uint_as_float(d[i]) - dlt) * p.scale;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float pr =
                ((word[c] >> i) & 1u) ? __expf(__uint_as_float(s[i]) * p.scale - lse) : 0.f;
            ds[i] = pr * (__uint_as_float(d[i]) - dlt) * p.scale;
          }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(ds[2 * i], ds[2 * i + 1]);
        tmem_st_32x16(tSj + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(ds_full);
    }
    // dQ is complete; it leaves through the K stages, which nothing reads any more
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(dq_done, 0, p.status, kErrAttnWait));
    tc_fence_after_sync();
    if (half == 0) {
      const RowStager rows{sK + q * 8192, lane};
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tdQ + lane_base + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) rows.put(c * 4 + g, pack8(&v[8 * g]));
      }
      const int first = qb * kBlk + q * 32;
      const int64_t width = static_cast<int64_t>(p.hq + 2 * p.hkv) * kD;
      if (ok)
        rows.flush(p.dqkv + static_cast<int64_t>(row0 + first) * width + h * kD, width,
                   min(32, p.seq - first));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------- dK, dV
// One CTA per (key block j, kv head x part, batch); loops over its share of the query heads of the
// GQA group and the query blocks i >= j, so dK / dV accumulate in TMEM and are written once.
// With parts == 1 the CTA owns the whole group and writes bf16 dK / dV; with parts > 1 (small
// batches would otherwise leave most SMs idle) each part writes an fp32 partial plane and
// attention_dkv_finish_kernel adds the planes in a fixed order.
// Scores are formed transposed (rows = keys): S^T = K Q^T, dP^T = V dO^T, so a softmax thread owns
// half a key row and P^T / dS^T rows are K-major operands of
//   dV += P^T dO,   dK += dS^T Q.
// P^T and dS^T (bf16) are written over the S^T and dP^T they came from, each half row into its own 64
// columns, and read by the MMAs from TMEM.  The two chains S^T -> P^T -> dV and dP^T -> dS^T -> dK
// hand over separately: while the softmax warps take exponentials of block t+1, dK(t) and dP^T(t+1)
// run, and while they form dS^T(t+1), dV(t+1) and S^T(t+2) run.  Q and dO have two stages.
// Bound by the chain of hand-overs and by the grid: at 2 x 2048 (12 heads, 2 kv heads) the tensor pipe is
// active 39 % of the cycles, issue slots are used to 29 %, and SMs are busy for 87 to 149 thousand cycles
// (mean 115): the CTAs of the first key blocks are the longest.  At 1 x 8192 a block takes 4200 to
// 5900 clocks (1.4 to 1.965 GHz); its products need 2048.
// Measured on B200 inside a training step (12 heads, 2 kv heads): 1 x 8192: 1188 us before (serial
// chain, P^T and dS^T through shared memory, one thread per row) and 507 us now; 8 x 512: 80 and 42 us.
// smem: K | V | (Q, dO) x 2 | (lse[128], delta[128]) x 2 | barriers
constexpr int kDkvSmem = 6 * kTile + 2048 + 1024 + 256;

__global__ void __launch_bounds__(kBwdThreads, 1)
attention_dkv_kernel(const __grid_constant__ CUtensorMap map_qkv,
                     const __grid_constant__ CUtensorMap map_do, BwdParams p) {
  extern __shared__ uint8_t raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + kTile;
  uint8_t* sQ = sV + kTile;                     // stage s: Q at sQ + s * 2 * kTile, dO right after
  float* s_stat = reinterpret_cast<float*>(sQ + 4 * kTile);   // buffer s: lse at s * 256, delta + 128
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_stat + 512);
  uint64_t* kv_full = bars;
  uint64_t* s_full = bars + 1;
  uint64_t* dp_full = bars + 2;
  uint64_t* pt_full = bars + 3;   // 256 arrivals
  uint64_t* ds_full = bars + 4;   // 256 arrivals
  uint64_t* done = bars + 5;
  uint64_t* q_full = bars + 6;    // 2
  uint64_t* q_empty = bars + 8;   // 2
  uint64_t* idle = bars + 10;     // every MMA is over
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_q = (p.seq + kBlk - 1) / kBlk;
  const int kb = static_cast<int>(blockIdx.x) / (p.hkv * p.parts * p.batch);   // long loops first
  const int rest = static_cast<int>(blockIdx.x) % (p.hkv * p.parts * p.batch);
  const int b = rest / (p.hkv * p.parts);
  const int hk = rest % (p.hkv * p.parts) / p.parts, part = rest % p.parts;
  const int group = p.hq / p.hkv;
  const int heads_here = group / p.parts;   // parts divides group (checked on the host)
  const int head0 = hk * group + part * heads_here;
  const int per_head = n_q - kb;          // query blocks kb .. n_q-1
  const int iters = heads_here * per_head;
  const int row0 = b * p.seq;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 11; ++i) mbar_init(bars + i, i == 3 || i == 4 ? 256 : 1);
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&map_qkv);
    prefetch_tensormap(&map_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  chain_wait();                       // what is above ran under the kernel before
  if (kernel_should_skip(p.status)) { // an earlier kernel already failed
    if (warp == 1) tmem_dealloc(tmem, 512);
    return;
  }
  const uint32_t tST = tmem, tdPT = tmem + 128, tdV = tmem + 256, tdK = tmem + 384;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * kTile);
      load_tile(sK, &map_qkv, kv_full, (p.hq + hk) * kD, row0 + kb * kBlk);
      load_tile(sV, &map_qkv, kv_full, (p.hq + p.hkv + hk) * kD, row0 + kb * kBlk);
    }
    __syncwarp();
    int loads = 0;
    for (int t = 0; t < iters; ++t) {
      const int h = head0 + t / per_head;
      const int i = kb + t % per_head;
      const int s = t & 1;
      if (!mbar_wait_warp(&q_empty[s], ((t >> 1) & 1) ^ 1, p.status, kErrAttnWait)) break;
      if (elect_one()) {
        mbar_expect_tx(&q_full[s], 2 * kTile);
        load_tile(sQ + s * 2 * kTile, &map_qkv, &q_full[s], h * kD, row0 + i * kBlk);
        load_tile(sQ + s * 2 * kTile + kTile, &map_do, &q_full[s], h * kD, row0 + i * kBlk);
      }
      __syncwarp();
      ++loads;
    }
    if (elect_one()) chain_release();
    // kv_full; q_full[2]
    mbar_drain(bars + lane, lane == 0 ? 1 : lane == 6 || lane == 7 ? ring_uses(loads, 2, lane - 6) : 0, p.status);
  } else if (warp == 1) {
    const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aQ = smem_u32(sQ);
    bool ok = mbar_wait_warp(kv_full, 0, p.status, kErrAttnWait) &&
              mbar_wait_warp(&q_full[0], 0, p.status, kErrAttnWait);
    int s_done = 0, dp_done = 0, dk_done = 0;
    if (ok) {
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ss(tST, aK, aQ);                      // S^T  = K Q^T
        tc_commit(s_full);
        mma_ss(tdPT, aV, aQ + kTile);             // dP^T = V dO^T
        tc_commit(dp_full);
      }
      __syncwarp();
      s_done = dp_done = 1;
    }
    for (int t = 0; t < iters && ok; ++t) {
      const uint32_t q_t = aQ + (t & 1) * 2 * kTile, q_n = aQ + ((t + 1) & 1) * 2 * kTile;
      const bool more = t + 1 < iters;
      ok = mbar_wait_warp(pt_full, t & 1, p.status, kErrAttnWait);
      if (ok && more) ok = mbar_wait_warp(&q_full[(t + 1) & 1], ((t + 1) >> 1) & 1, p.status, kErrAttnWait);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ts(tdV, tST, 64, q_t + kTile, t > 0);           // dV += P^T dO
        if (more) {
          mma_ss(tST, aK, q_n);                             // S^T(t+1), over the P^T just read
          tc_commit(s_full);
        }
      }
      __syncwarp();
      s_done += more;
      ok = mbar_wait_warp(ds_full, t & 1, p.status, kErrAttnWait);
      if (!ok) break;
      tc_fence_after_sync();
      if (elect_one()) {
        mma_ts(tdK, tdPT, 64, q_t, t > 0);                  // dK += dS^T Q
        tc_commit(&q_empty[t & 1]);
        if (more) {
          mma_ss(tdPT, aV, q_n + kTile);                    // dP^T(t+1), over the dS^T just read
          tc_commit(dp_full);
        } else {
          tc_commit(done);
        }
      }
      __syncwarp();
      ++dk_done;
      dp_done += more;
    }
    commit_all(idle);
    // s_full; dp_full; done; q_empty[2]; idle
    mbar_drain(bars + lane, lane == 1 ? s_done : lane == 2 ? dp_done : lane == 5 ? dk_done == iters
                            : lane == 8 || lane == 9 ? ring_uses(dk_done, 2, lane - 8) : lane == 10, p.status);
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int r = q * 32 + lane;              // key row inside the tile
    const int kv_idx = kb * kBlk + r;
    const uint32_t lane_base = static_cast<uint32_t>(q * 32) << 16;
    bool kv_ok = kv_idx < p.seq;
    if (kv_ok && p.key_bits != nullptr)
      kv_ok = (p.key_bits[static_cast<int64_t>(b) * p.bits_pitch + (kv_idx >> 5)] >> (kv_idx & 31)) & 1u;
    else if (kv_ok && p.key_mask != nullptr)
      kv_ok = p.key_mask[b * p.seq + kv_idx] != 0;
    // this thread's share of a query block's statistics: lse (half 0) or delta (half 1) of query r
    const float* stats = half ? p.delta : p.lse;
    auto stat_of = [&](int t) {
      const int h = head0 + t / per_head;
      const int qi = (kb + t % per_head) * kBlk + r;
      return stats[(static_cast<int64_t>(b) * p.hq + h) * p.seq + min(qi, p.seq - 1)];
    };
    float* mine = s_stat + half * 128 + r;
    mine[0] = stat_of(0);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    bool ok = true;
    for (int t = 0; t < iters; ++t) {
      const float next = t + 1 < iters ? stat_of(t + 1) : 0.f;
      const float* lse = s_stat + (t & 1) * 256 + half * 64;
      const float* dlt = lse + 128;
      const int q0 = (kb + t % per_head) * kBlk + half * 64;   // first query of this half
      // queries from the key's own position to the end of the sequence, as bits
      uint32_t word[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int from = kv_idx - (q0 + c * 32), to = p.seq - (q0 + c * 32);
        uint32_t w = kv_ok ? 0xffffffffu : 0u;
        if (from > 0) w = from >= 32 ? 0u : w & (0xffffffffu << from);
        if (to < 32) w = to <= 0 ? 0u : w & ((1u << to) - 1u);
        word[c] = w;
      }
      // after a failed wait the loop keeps its shape (no early exit) so that every thread
      // still reaches the named barrier below the same number of times
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(s_full, t & 1, p.status, kErrAttnWait));
      tc_fence_after_sync();
      float pr[64];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32], pk[16];
        tmem_ld_32x32(tST + lane_base + half * 64 + c * 32, s);
        tmem_ld_wait();
        const bool all_on = __all_sync(0xffffffffu, word[c] == 0xffffffffu);
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(lse + c * 32 + x);
          const float lv[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u)
            pr[c * 32 + x + u] = __expf(__uint_as_float(s[x + u]) * p.scale - lv[u]);
        }
        if (!all_on) {
#pragma unroll
          for (int x = 0; x < 32; ++x) pr[c * 32 + x] = ((word[c] >> x) & 1u) ? pr[c * 32 + x] : 0.f;
        }
#pragma unroll
        for (int x = 0; x < 16; ++x) pk[x] = pack_bf16x2(pr[c * 32 + 2 * x], pr[c * 32 + 2 * x + 1]);
        tmem_st_32x16(tST + lane_base + half * 64 + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(pt_full);
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(dp_full, t & 1, p.status, kErrAttnWait));
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t d[32], pk[16];
        tmem_ld_32x32(tdPT + lane_base + half * 64 + c * 32, d);
        tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const float4 d4 = *reinterpret_cast<const float4*>(dlt + c * 32 + x);
          const float dv[4] = {d4.x, d4.y, d4.z, d4.w};
          float ds[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            ds[u] = pr[c * 32 + x + u] * (__uint_as_float(d[x + u]) - dv[u]) * p.scale;
          pk[x >> 1] = pack_bf16x2(ds[0], ds[1]);
          pk[(x >> 1) + 1] = pack_bf16x2(ds[2], ds[3]);
        }
        tmem_st_32x16(tdPT + lane_base + half * 64 + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(ds_full);
      // the other buffer's readers (iteration t - 1) passed the last barrier
      mine[((t + 1) & 1) * 256] = next;
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(done, 0, p.status, kErrAttnWait));
    tc_fence_after_sync();
    // half 0 writes dK, half 1 dV
    const int first = kb * kBlk + q * 32;
    const uint32_t acc = half ? tdV : tdK;
    if (p.parts > 1) {
      const int64_t pwidth = static_cast<int64_t>(2 * p.hkv) * kD;
      float* row = p.dkv_part + (static_cast<int64_t>(part) * p.batch * p.seq + row0 + kv_idx) * pwidth +
                   (half * p.hkv + hk) * kD;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(acc + lane_base + c * 32, v);
        tmem_ld_wait();
        if (ok && kv_idx < p.seq) {
#pragma unroll
          for (int g = 0; g < 8; ++g)
            *reinterpret_cast<uint4*>(row + c * 32 + g * 4) =
                make_uint4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
        }
      }
    } else {
      // through the Q / dO stages, which nothing reads any more
      const RowStager rows{sQ + (half * 4 + q) * 8192, lane};
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(acc + lane_base + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) rows.put(c * 4 + g, pack8(&v[8 * g]));
      }
      const int64_t width = static_cast<int64_t>(p.hq + 2 * p.hkv) * kD;
      if (ok)
        rows.flush(p.dqkv + static_cast<int64_t>(row0 + first) * width + (p.hq + half * p.hkv + hk) * kD,
                   width, min(32, p.seq - first));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// dqkv[row, K|V columns] = bf16(sum over parts of the fp32 partial planes), fixed order.
__global__ void attention_dkv_finish_kernel(const float* part, int parts, int64_t rows, int hq, int hkv,
                                            __nv_bfloat16* dqkv) {
  chain_wait();
  chain_release();
  const int64_t pwidth = static_cast<int64_t>(2 * hkv) * kD;     // floats per row of a plane
  const int64_t vec = pwidth / 8;
  const int64_t width = static_cast<int64_t>(hq + 2 * hkv) * kD;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < rows * vec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / vec;
    const int64_t col = (i - row * vec) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < parts; ++k) {
      const float4* src = reinterpret_cast<const float4*>(part + (k * rows + row) * pwidth + col);
      const float4 a = src[0], b = src[1];
      acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
      acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
    }
    uint4 pk;
    pk.x = pack_bf16x2(acc[0], acc[1]);
    pk.y = pack_bf16x2(acc[2], acc[3]);
    pk.z = pack_bf16x2(acc[4], acc[5]);
    pk.w = pack_bf16x2(acc[6], acc[7]);
    *reinterpret_cast<uint4*>(dqkv + row * width + static_cast<int64_t>(hq) * kD + col) = pk;
  }
}

template <typename K>
cudaError_t opt_in_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace

cudaError_t launch_attention_fwd(const AttnCall& c, int* status, cudaStream_t s) {
  if (c.seq < 1 || c.hq % c.hkv) return cudaErrorInvalidValue;
  const int64_t rows = static_cast<int64_t>(c.batch) * c.seq;
  const int64_t width = static_cast<int64_t>(c.hq + 2 * c.hkv) * kD;
  CUtensorMap map;
  if (!make_bf16_tensor_map(&map, c.qkv, rows, width, width, 64, kBlk)) return cudaErrorInvalidValue;
  static cudaError_t attr = opt_in_smem(attention_fwd_kernel, kFwdSmem);
  if (attr != cudaSuccess) return attr;
  if (c.key_bits != nullptr &&
      (c.key_bits_pitch < 4 * ((c.seq + kBlk - 1) / kBlk) || (c.key_bits_pitch % 4) ||
       (reinterpret_cast<uintptr_t>(c.key_bits) & 15)))
    return cudaErrorInvalidValue;
  FwdParams p{reinterpret_cast<__nv_bfloat16*>(c.out), c.lse, c.key_mask, c.batch, c.seq, c.hq,
              c.hkv, c.scale, status, c.key_bits, c.key_bits_pitch};
  const int64_t grid = static_cast<int64_t>((c.seq + kBlk - 1) / kBlk) * c.hq * c.batch;
  launch_chained(attention_fwd_kernel, static_cast<unsigned>(grid), kFwdThreads, kFwdSmem, s, map, p);
  count_launch();
  return cudaGetLastError();
}

namespace {
// what dK/dV and dQ launch with, checked
struct BwdLaunch {
  CUtensorMap map_qkv, map_do;
  BwdParams p;
  int nblk;
};
cudaError_t prepare_bwd(const AttnBwdCall& c, int* status, BwdLaunch* out) {
  if (c.seq < 1 || c.hq % c.hkv) return cudaErrorInvalidValue;
  const int64_t rows = static_cast<int64_t>(c.batch) * c.seq;
  const int64_t width = static_cast<int64_t>(c.hq + 2 * c.hkv) * kD;
  const int64_t owidth = static_cast<int64_t>(c.hq) * kD;
  if (!make_bf16_tensor_map(&out->map_qkv, c.qkv, rows, width, width, 64, kBlk) ||
      !make_bf16_tensor_map(&out->map_do, c.dout, rows, owidth, owidth, 64, kBlk))
    return cudaErrorInvalidValue;
  static cudaError_t attr1 = opt_in_smem(attention_dq_kernel, kDqSmem);
  static cudaError_t attr2 = opt_in_smem(attention_dkv_kernel, kDkvSmem);
  if (attr1 != cudaSuccess) return attr1;
  if (attr2 != cudaSuccess) return attr2;
  out->nblk = (c.seq + kBlk - 1) / kBlk;
  int parts = 1;
  if (c.dkv_accum != nullptr) {
    parts = attention_bwd_parts(c.batch, c.seq, c.hq, c.hkv);
    const int64_t need = static_cast<int64_t>(parts) * rows * 2 * c.hkv * kD;
    if (parts > 1 && c.dkv_accum_floats < need) return cudaErrorInvalidValue;
  }
  if (c.key_bits != nullptr &&
      (c.key_bits_pitch < 4 * out->nblk || (c.key_bits_pitch % 4) ||
       (reinterpret_cast<uintptr_t>(c.key_bits) & 15)))
    return cudaErrorInvalidValue;
  out->p = BwdParams{c.lse, c.delta, reinterpret_cast<__nv_bfloat16*>(c.dqkv), c.key_mask, c.batch, c.seq,
                     c.hq, c.hkv, c.scale, status, parts > 1 ? c.dkv_accum : nullptr, parts,
                     c.key_bits, c.key_bits_pitch};
  return cudaSuccess;
}
}  // namespace

cudaError_t launch_attention_bwd_delta(const AttnBwdCall& c, cudaStream_t s) {
  if (c.seq < 1 || c.hq % c.hkv) return cudaErrorInvalidValue;
  const int64_t warps = static_cast<int64_t>(c.batch) * c.seq * c.hq;
  launch_chained(
      attention_delta_kernel, static_cast<int>((warps * 32 + 255) / 256), 256, 0, s,
      reinterpret_cast<const __nv_bfloat16*>(c.out), reinterpret_cast<const __nv_bfloat16*>(c.dout),
      c.delta, c.batch, c.seq, c.hq);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_attention_bwd_dkv(const AttnBwdCall& c, int* status, cudaStream_t s) {
  BwdLaunch l;
  const cudaError_t e = prepare_bwd(c, status, &l);
  if (e != cudaSuccess) return e;
  launch_chained(attention_dkv_kernel,
                 static_cast<unsigned>(static_cast<int64_t>(l.nblk) * c.hkv * l.p.parts * c.batch),
                 kBwdThreads, kDkvSmem, s, l.map_qkv, l.map_do, l.p);
  count_launch();
  if (l.p.parts > 1) {
    const int64_t rows = static_cast<int64_t>(c.batch) * c.seq;
    const int64_t work = rows * (2 * c.hkv * kD / 8);
    const int grid = static_cast<int>(std::min<int64_t>((work + 255) / 256, sm_count() * 8));
    launch_chained(attention_dkv_finish_kernel, grid, 256, 0, s, c.dkv_accum, l.p.parts, rows, c.hq, c.hkv,
                   reinterpret_cast<__nv_bfloat16*>(c.dqkv));
    count_launch();
  }
  return cudaGetLastError();
}

cudaError_t launch_attention_bwd_dq(const AttnBwdCall& c, int* status, cudaStream_t s) {
  BwdLaunch l;
  const cudaError_t e = prepare_bwd(c, status, &l);
  if (e != cudaSuccess) return e;
  launch_chained(attention_dq_kernel, static_cast<unsigned>(static_cast<int64_t>(l.nblk) * c.hq * c.batch),
                 kBwdThreads, kDqSmem, s, l.map_qkv, l.map_do, l.p);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_attention_bwd(const AttnBwdCall& c, int* status, cudaStream_t s) {
  cudaError_t e = launch_attention_bwd_delta(c, s);
  if (e == cudaSuccess) e = launch_attention_bwd_dkv(c, status, s);
  return e != cudaSuccess ? e : launch_attention_bwd_dq(c, status, s);
}

namespace {
// bits[b, w] bit i = (mask[b, 32 w + i] != 0); words beyond the sequence are zero
__global__ void pack_key_mask_kernel(const uint8_t* __restrict__ mask, uint32_t* __restrict__ bits,
                                     int batch, int seq, int pitch) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= batch * pitch) return;
  const int b = idx / pitch, w = idx - b * pitch;
  uint32_t word = 0;
  for (int i = 0; i < 32; ++i) {
    const int kv = w * 32 + i;
    if (kv < seq && mask[static_cast<int64_t>(b) * seq + kv] != 0) word |= 1u << i;
  }
  bits[idx] = word;
}
}  // namespace

cudaError_t launch_pack_key_mask(const uint8_t* mask, uint32_t* bits, int batch, int seq, int pitch,
                                 cudaStream_t s) {
  if (batch < 1 || seq < 1 || pitch < 4 * ((seq + kBlk - 1) / kBlk) || (pitch % 4))
    return cudaErrorInvalidValue;
  const int total = batch * pitch;
  pack_key_mask_kernel<<<(total + 127) / 128, 128, 0, s>>>(mask, bits, batch, seq, pitch);
  count_launch();
  return cudaGetLastError();
}

int attention_bwd_parts(int batch, int seq, int hq, int hkv) {
  // smallest split of the query-head group that puts at least one dK/dV CTA on every SM
  const int group = hq / hkv;
  const int nblk = (seq + kBlk - 1) / kBlk;
  const int base = nblk * hkv * batch;
  for (int parts = 1; parts <= group; ++parts)
    if (group % parts == 0 && base * parts >= sm_count()) return parts;
  return group;
}

}  // namespace stb

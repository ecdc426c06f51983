// Attention with 32-bit probabilities on the tensor cores (tcgen05 / TMEM / TMA): any head dim that is a multiple of 8 up to 64,
// query and key lengths of their own (cross attention), dense 0/1 masks whose masked scores are -10000, causal or full; forward
// and backward.
//
// These calls used to run as unfused fp32 matrix products over [b, a, sq, sk] tensors (head dims 24, 32 and 48 of the shipped GPT,
// BERT and T5 recipes, every dense mask).  They held probabilities and their gradients in 32 bits, and so does this: P and dS go
// to the tensor core as the sum of two bf16 numbers (hi = bf16(x), lo = bf16(x - hi), together 16 bits of mantissa), two MMAs in
// place of one, accumulated in fp32; the row sums of dO ∘ O use O in the same two parts.  Errors against 64 bits are those of the
// unfused form (both end in the rounding of the bf16 results).
//
// Head dims below 64: the tensor maps have the true inner extent, TMA fills columns [d, 64) of the tiles with zeros, which add
// nothing to Q·Kᵀ / dO·Vᵀ; the surplus columns of the other products are not stored.  Masks arrive packed, one bit per (query,
// key), with one fill value per row: -10000 (log2 domain), or 0 for a row without any visible key, whose probabilities are uniform
// whatever the constant (0 keeps its log-sum-exp small and exact).
//
// Bounded by the softmax threads (two passes over S, two roundings per probability), not by the tensor core or memory: key tiles of
// 128, two forward CTAs per SM.  Measured: [16, 512] BERT block with 16 heads of 48 and a padding mask, attention kernels 294 us (181
// backward, 85 forward, 28 around them) where the unfused form took 2470 us; cross attention of 128 on 512 tokens, 12 heads of 32,
// 16 sequences, with self attention 125 us against 780 us.
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

namespace lb {

constexpr int SPL_THREADS = 320;                 // TMA warp, MMA warp, 8 softmax warps
constexpr int SPL_TILE = 128 * 64 * 2;           // one [128, 64] bf16 tile, 128-byte rows, swizzled
constexpr float SPL_LOG2E = 1.4426950408889634f;

struct SplitParams {
  int B, A, Sq, Sk, d;
  int causal, off;              // off = Sk - Sq: query i sees keys [0, i + off] under the causal mask
  float scale, scale_log2;
  const uint32_t* mask;         // [Bm, Am, Sq, pitch] words, bit = visible; nullptr: no mask
  const float* fill;            // [Bm, Am, Sq] score of the masked keys of a row, log2 domain
  long mask_b, mask_a;          // rows between batches / heads (0: shared)
  int pitch;                    // words per row, a multiple of 4
  __nv_bfloat16 *o, *o_lo;      // [B, Sq, A, d]; o_lo (optional): what the rounding of o left over
  float* lse;                   // [B, A, Sq] natural log
  // backward
  const float* delta;           // [B, A, Sq]
  __nv_bfloat16 *dk, *dv;       // [B, A, Sk, d] views
  long dk_strides[3], dv_strides[3];
  int* err;
};

LB_DEVICE uint32_t split_hi(float x0, float x1) { return pack_bf16(x0, x1); }
LB_DEVICE uint32_t split_lo(float x0, float x1, uint32_t hi) {
  const float2 h = unpack_bf16(hi);
  return pack_bf16(x0 - h.x, x1 - h.y);
}

// ------------------------------------------------------------------------------------------------------------ mask -> bits
// one warp per (batch, head, query) row of the mask as it broadcasts; `and_mask` drops the sign of a floating zero
template <typename U>
__global__ void __launch_bounds__(256)
attn_mask_pack_kernel(const U* __restrict__ mask, unsigned long long and_mask, int Bm, int Am, int Sq, int Sk, long sb, long sa, long sq,
                      long sk, int causal, int off, uint32_t* __restrict__ words, float* __restrict__ fill, int pitch) {
  const long rows = static_cast<long>(Bm) * Am * Sq;
  const int lane = threadIdx.x % 32;
  const U keep_bits = static_cast<U>(and_mask);
  for (long r = blockIdx.x * static_cast<long>(blockDim.x / 32) + threadIdx.x / 32; r < rows; r += static_cast<long>(gridDim.x) * (blockDim.x / 32)) {
    const int q = static_cast<int>(r % Sq);
    const U* row = mask + (r / Sq / Am) * sb + ((r / Sq) % Am) * sa + q * sq;
    uint32_t any = 0;
    for (int w0 = 0; w0 < pitch; w0 += 32) {
      uint32_t mine = 0;
      for (int w = w0; w < min(pitch, w0 + 32); ++w) {
        const int k = w * 32 + lane;
        const bool on = k < Sk && (!causal || k <= q + off) && (row[static_cast<long>(k) * sk] & keep_bits) != 0;
        const uint32_t word = __ballot_sync(0xffffffffu, on);
        any |= word;
        if (w - w0 == lane) mine = word;
      }
      if (w0 + lane < pitch) words[r * pitch + w0 + lane] = mine;
    }
    if (lane == 0) fill[r] = any ? -10000.0f * SPL_LOG2E : 0.0f;
  }
}

// ------------------------------------------------------------------------------------------------------------------ forward
// One CTA per (128 queries, head, batch).  S in TMEM columns [0, 128), O in [128, 192), P hi in [192, 256); P lo of a half's 64 keys
// overwrites the first 32 of that half's S columns once its threads have read them, so the whole fits 256 columns and two CTAs
// share an SM.  The MMA warp issues S(j+1) after P(j)·V(j) has completed (it overwrites P lo); the other CTA fills the gap.
constexpr int SPL_FWD_SMEM = 5 * SPL_TILE + 2 * 2 * 128 * 4 + 1024 + 256;

template <bool MASKED>
__global__ void __launch_bounds__(SPL_THREADS, 2)
attn_split_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, SplitParams p) {
  constexpr uint32_t S_COL = 0, O_COL = 128, P_COL = 192;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + SPL_TILE;
  uint8_t* sV = sK + 2 * SPL_TILE;
  float* sXchg = reinterpret_cast<float*>(sV + 2 * SPL_TILE);      // [parity][half][row]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sXchg + 2 * 2 * 128);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 3;
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 9;
  uint64_t* p_full = bars + 10;
  uint64_t* o_full = bars + 11;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 12);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 13);

  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int q_blk = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x);   // late query blocks have the most keys
  const int head = blockIdx.y, batch = blockIdx.z, q0 = q_blk * 128;
  int nkv = (p.Sk + 127) / 128;
  if (p.causal) nkv = min(nkv, (min(q0 + 128, p.Sq) + p.off + 127) / 128);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(o_full, 1);
    *stop = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 1) tmem_alloc<256>(tmem_ptr_smem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp_idx == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(q_full, SPL_TILE);
      tma_load_4d(sQ, &tmap_q, q_full, 0, q0, head, batch);
      for (int j = 0; j < nkv; ++j) {
        const int b = j & 1;
        const uint32_t par = ((j >> 1) & 1) ^ 1;
        if (tc_wait(&k_empty[b], par, stop)) {
          mbar_arrive_expect_tx(&k_full[b], SPL_TILE);
          tma_load_4d(sK + b * SPL_TILE, &tmap_k, &k_full[b], 0, j * 128, head, batch);
        }
        if (tc_wait(&v_empty[b], par, stop)) {
          mbar_arrive_expect_tx(&v_full[b], SPL_TILE);
          tma_load_4d(sV + b * SPL_TILE, &tmap_v, &v_full[b], 0, j * 128, head, batch);
        }
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    constexpr uint32_t idesc_qk = make_idesc_bf16(128, 128, false, false);
    constexpr uint32_t idesc_pv = make_idesc_bf16(128, 64, false, true);
    const int ksteps = (p.d + 15) / 16;                              // the columns behind d are zeros
    const uint32_t q_addr = smem_u32(sQ);
    bool ok = __all_sync(0xffffffffu, tc_wait(q_full, 0, stop));
    for (int j = 0; j < nkv; ++j) {
      const int b = j & 1;
      ok = __all_sync(0xffffffffu, ok && tc_wait(&k_full[b], (j >> 1) & 1, stop));
      if (j > 0) ok = __all_sync(0xffffffffu, ok && tc_wait(o_full, (j - 1) & 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        const uint32_t k_addr = smem_u32(sK + b * SPL_TILE);
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(tmem_base + S_COL, make_smem_desc_sw128(q_addr + kk * 32, 0, 1024), make_smem_desc_sw128(k_addr + kk * 32, 0, 1024),
                      idesc_qk, kk > 0 ? 1u : 0u);
        umma_commit(s_full);
        umma_commit(&k_empty[b]);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, ok && tc_wait(p_full, j & 1, stop));
      ok = __all_sync(0xffffffffu, ok && tc_wait(&v_full[b], (j >> 1) & 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        const uint32_t v_addr = smem_u32(sV + b * SPL_TILE);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint64_t bv = make_smem_desc_sw128(v_addr + kk * (16 * 128), 128 * 128, 1024);
          umma_f16_ts(tmem_base + O_COL, tmem_base + P_COL + kk * 8, bv, idesc_pv, (j > 0 || kk > 0) ? 1u : 0u);
          umma_f16_ts(tmem_base + O_COL, tmem_base + S_COL + (kk / 4) * 64 + (kk % 4) * 8, bv, idesc_pv, 1u);
        }
        umma_commit(o_full);
        umma_commit(&v_empty[b]);
      }
      __syncwarp();
    }
  } else {
    const int quad = warp_idx % 4, half = (warp_idx - 2) / 4;        // this warp's 64 of the 128 key columns
    const int r = quad * 32 + lane, q_idx = q0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_off + S_COL + half * 64;
    const uint32_t p_addr = tmem_base + lane_off + P_COL + half * 32;
    const uint32_t o_addr = tmem_base + lane_off + O_COL + half * 32;
    const int key_lim = p.causal ? min(p.Sk, q_idx + p.off + 1) : p.Sk;
    [[maybe_unused]] const uint32_t* mrow = nullptr;
    [[maybe_unused]] float fill = 0.f;
    if constexpr (MASKED) {
      const long row = batch * p.mask_b + head * p.mask_a + min(q_idx, p.Sq - 1);
      mrow = p.mask + row * p.pitch + half * 2;
      fill = p.fill[row];
    }
    float m_run = -INFINITY, l_run = 0.f;
    for (int j = 0; j < nkv; ++j) {
      [[maybe_unused]] uint2 bits = make_uint2(0, 0);
      if constexpr (MASKED) bits = *reinterpret_cast<const uint2*>(mrow + j * 4);
      tc_wait(s_full, j & 1, stop);
      __syncwarp();
      tc_fence_after_sync();
      const int k0 = j * 128 + half * 64;
      const bool edge = j * 128 + 128 > p.Sk || (p.causal && j * 128 + 127 > q0 + p.off);
      float mx = -INFINITY;
      auto pass1 = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t t[32];
          tmem_ld_32x32b_x32(s_addr + c * 32, t);
          tmem_ld_wait();
          [[maybe_unused]] const uint32_t word = c == 0 ? bits.x : bits.y;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float x = __uint_as_float(t[i]) * p.scale_log2;
            if constexpr (MASKED) x = (word >> i) & 1u ? x : fill;
            if constexpr (EDGE) x = k0 + c * 32 + i < key_lim ? x : -INFINITY;
            mx = fmaxf(mx, x);
          }
        }
      };
      if (edge) pass1(std::true_type{}); else pass1(std::false_type{});
      float* xch = sXchg + (j & 1) * 256;
      xch[half * 128 + r] = mx;
      tc_pair_sync(quad);
      mx = fmaxf(mx, xch[(half ^ 1) * 128 + r]);
      const float m_cand = fmaxf(m_run, mx);
      const bool bump = (m_cand - m_run > 8.0f) || (m_run == -INFINITY && m_cand != -INFINITY);   // lazy rescale
      float alpha = 1.0f;
      if (bump) { alpha = fast_exp2(m_run - m_cand); m_run = m_cand; }                            // 0 on the first tile
      const bool bump_any = __any_sync(0xffffffffu, bump && j > 0);
      const float m_use = m_run == -INFINITY ? 0.f : m_run;
      float rowsum = 0.f;
      auto pass2 = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t t[32], hi[16], lo[16];
          tmem_ld_32x32b_x32(s_addr + c * 32, t);
          tmem_ld_wait();
          [[maybe_unused]] const uint32_t word = c == 0 ? bits.x : bits.y;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float x0 = __uint_as_float(t[i]) * p.scale_log2, x1 = __uint_as_float(t[i + 1]) * p.scale_log2;
            if constexpr (MASKED) {
              x0 = (word >> i) & 1u ? x0 : fill;
              x1 = (word >> (i + 1)) & 1u ? x1 : fill;
            }
            x0 = fast_exp2(x0 - m_use);
            x1 = fast_exp2(x1 - m_use);
            if constexpr (EDGE) {
              x0 = k0 + c * 32 + i < key_lim ? x0 : 0.f;
              x1 = k0 + c * 32 + i + 1 < key_lim ? x1 : 0.f;
            }
            rs0 += x0;
            rs1 += x1;
            hi[i / 2] = split_hi(x0, x1);
            lo[i / 2] = split_lo(x0, x1, hi[i / 2]);
          }
          // (S(j) follows the completion of P(j-1)·V(j-1): both sets of columns are free; lo covers S columns read above)
          tmem_st_32x32b_x16(p_addr + c * 16, hi);
          tmem_st_32x32b_x16(s_addr + c * 16, lo);
        }
        rowsum = rs0 + rs1;
      };
      if (edge) pass2(std::true_type{}); else pass2(std::false_type{});
      l_run = l_run * alpha + rowsum;
      if (bump_any) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(o_addr, t);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
        tmem_st_32x32b_x32(o_addr, t);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    float* xch = sXchg + (nkv & 1) * 256;
    xch[half * 128 + r] = l_run;
    tc_pair_sync(quad);
    l_run += xch[(half ^ 1) * 128 + r];
    tc_wait(o_full, (nkv - 1) & 1, stop);
    __syncwarp();
    tc_fence_after_sync();
    const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
    uint32_t t[32];
    tmem_ld_32x32b_x32(o_addr, t);
    tmem_ld_wait();
    if (q_idx < p.Sq) {
      const size_t at = ((static_cast<size_t>(batch) * p.Sq + q_idx) * p.A + head) * p.d + half * 32;
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        if (half * 32 + i >= p.d) break;                             // d is a multiple of 8
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x0 = __uint_as_float(t[i + 2 * e]) * inv, x1 = __uint_as_float(t[i + 2 * e + 1]) * inv;
          hi[e] = split_hi(x0, x1);
          lo[e] = split_lo(x0, x1, hi[e]);
        }
        *reinterpret_cast<uint4*>(p.o + at + i) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        if (p.o_lo != nullptr) *reinterpret_cast<uint4*>(p.o_lo + at + i) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      if (half == 0)
        p.lse[(static_cast<size_t>(batch) * p.A + head) * p.Sq + q_idx] =
            m_run == -INFINITY ? -INFINITY : (m_run + log2f(l_run)) * 0.6931471805599453f;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*stop) {                                                       // copies in flight land before the shared memory goes away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) { *const_cast<volatile int*>(p.err) = 1; __threadfence_system(); }
    __syncthreads();
  }
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc<256>(tmem_base);
  }
}

// ----------------------------------------------------------------------------------------------------------------- backward
// One CTA per (128 keys, head, batch), looping over the query blocks that see them:
//   S = Q·Kᵀ, dP = dO·Vᵀ;  P = exp(S - lse), dS = P ∘ (dP - δ) · scale, both to shared memory in two bf16 parts;
//   dV += Pᵀ·dO, dK += dSᵀ·Q, dQ_i = dS·K (added to the fp32 accumulator by TMA reductions).
// Shared memory: K, V, Q, dO 64 KB, the four P / dS tiles 128 KB, dQ staging 32 KB.
constexpr int SPL_PS = 128 * 128 * 2;
constexpr int SPL_DQ_BOX = 32 * 128;
constexpr int SPL_BWD_SMEM = 4 * SPL_TILE + 4 * SPL_PS + 8 * SPL_DQ_BOX + 1024 + 256;
static_assert(SPL_BWD_SMEM <= 232448, "split attention backward: shared memory");

template <bool MASKED>
__global__ void __launch_bounds__(SPL_THREADS, 1)
attn_split_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                      const __grid_constant__ CUtensorMap tmap_dq, SplitParams p) {
  constexpr uint32_t S_COL = 0, DP_COL = 128, DV_COL = 256, DK_COL = 320, DQ_COL = 384;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + SPL_TILE;
  uint8_t* sQ = sV + SPL_TILE;
  uint8_t* sDO = sQ + SPL_TILE;
  uint8_t* sP = sDO + SPL_TILE;                 // hi, lo
  uint8_t* sDS = sP + 2 * SPL_PS;               // hi, lo
  uint8_t* sDQ = sDS + 2 * SPL_PS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDQ + 8 * SPL_DQ_BOX);
  uint64_t* kv_full = bars;
  uint64_t* qdo_full = bars + 1;
  uint64_t* qdo_empty = bars + 2;               // also: P / dS tiles and dQ columns may be written again (with dq_empty)
  uint64_t* sdp_full = bars + 3;
  uint64_t* pds_full = bars + 4;
  uint64_t* dq_full = bars + 5;
  uint64_t* dq_empty = bars + 6;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 9);

  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int head = blockIdx.y, batch = blockIdx.z, k0 = blockIdx.x * 128;
  const int nq = (p.Sq + 127) / 128;
  const int i_begin = p.causal ? max(0, k0 - p.off) / 128 : 0;      // the first query that sees key k0 is k0 - off
  const int iters = nq - i_begin;                                    // >= 1: off >= 0 under the causal mask

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_dq);
    for (int i = 0; i < 7; ++i) mbar_init(bars + i, (i == 4 || i == 6) ? 8 : 1);
    *stop = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 1) tmem_alloc<512>(tmem_ptr_smem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp_idx == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * SPL_TILE);
      tma_load_4d(sK, &tmap_k, kv_full, 0, k0, head, batch);
      tma_load_4d(sV, &tmap_v, kv_full, 0, k0, head, batch);
      for (int it = 0; it < iters; ++it) {
        if (!tc_wait(qdo_empty, (it & 1) ^ 1, stop)) continue;
        mbar_arrive_expect_tx(qdo_full, 2 * SPL_TILE);
        tma_load_4d(sQ, &tmap_q, qdo_full, 0, (i_begin + it) * 128, head, batch);
        tma_load_4d(sDO, &tmap_do, qdo_full, 0, (i_begin + it) * 128, head, batch);
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);   // Q·Kᵀ, dO·Vᵀ
    constexpr uint32_t idesc_t = make_idesc_bf16(128, 64, true, true);      // Pᵀ·dO, dSᵀ·Q
    constexpr uint32_t idesc_q = make_idesc_bf16(128, 64, false, true);     // dS·K
    const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV), q_addr = smem_u32(sQ), do_addr = smem_u32(sDO);
    const uint32_t p_addr = smem_u32(sP), ds_addr = smem_u32(sDS);
    const int ksteps = (p.d + 15) / 16;
    bool ok = __all_sync(0xffffffffu, tc_wait(kv_full, 0, stop));
    for (int it = 0; it < iters; ++it) {
      ok = __all_sync(0xffffffffu, ok && tc_wait(qdo_full, it & 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(tmem_base + S_COL, make_smem_desc_sw128(q_addr + kk * 32, 0, 1024), make_smem_desc_sw128(k_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(tmem_base + DP_COL, make_smem_desc_sw128(do_addr + kk * 32, 0, 1024), make_smem_desc_sw128(v_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        umma_commit(sdp_full);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, ok && tc_wait(pds_full, it & 1, stop));
      ok = __all_sync(0xffffffffu, ok && tc_wait(dq_empty, (it & 1) ^ 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
#pragma unroll
        for (int part = 0; part < 2; ++part) {       // dQ first: its drain is the only consumer that is waited for
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ss(tmem_base + DQ_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + (kk / 4) * (128 * 128) + (kk % 4) * 32, 0, 1024),
                        make_smem_desc_sw128(k_addr + kk * 2048, 128 * 128, 1024), idesc_q, (part > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(dq_full);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ss(tmem_base + DV_COL, make_smem_desc_sw128(p_addr + part * SPL_PS + kk * 2048, 128 * 128, 1024),
                        make_smem_desc_sw128(do_addr + kk * 2048, 128 * 128, 1024), idesc_t, (it > 0 || part > 0 || kk > 0) ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ss(tmem_base + DK_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + kk * 2048, 128 * 128, 1024),
                        make_smem_desc_sw128(q_addr + kk * 2048, 128 * 128, 1024), idesc_t, (it > 0 || part > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(qdo_empty);
      }
      __syncwarp();
    }
  } else {
    const int quad = warp_idx % 4, half = (warp_idx - 2) / 4;        // this warp's 64 of the 128 key columns
    const int r = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const size_t bh = static_cast<size_t>(batch) * p.A + head;
    for (int it = 0; it < iters; ++it) {
      const int q_blk = i_begin + it, q_idx = q_blk * 128 + r;
      const bool q_ok = q_idx < p.Sq;
      const float lse2 = q_ok ? p.lse[bh * p.Sq + q_idx] * SPL_LOG2E : 0.f;
      const float delta_s = q_ok ? p.delta[bh * p.Sq + q_idx] * p.scale : 0.f;
      [[maybe_unused]] uint2 bits = make_uint2(0, 0);
      [[maybe_unused]] float fill = 0.f;
      if constexpr (MASKED) {
        const long row = batch * p.mask_b + head * p.mask_a + min(q_idx, p.Sq - 1);
        bits = *reinterpret_cast<const uint2*>(p.mask + row * p.pitch + (k0 / 32) + half * 2);
        fill = p.fill[row];
      }
      const int key_lim = !q_ok ? 0 : (p.causal ? min(p.Sk, q_idx + p.off + 1) : p.Sk);
      tc_wait(sdp_full, it & 1, stop);        // S(it) was issued after the products of block it-1 had read the P / dS tiles (one Q stage)
      __syncwarp();
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < 4; ++c) {            // 16 keys at a time: four packed tiles of 32 would spill
        uint32_t ts[16], td[16];
        tmem_ld_32x32b_x16(tmem_base + lane_off + S_COL + half * 64 + c * 16, ts);
        tmem_ld_32x32b_x16(tmem_base + lane_off + DP_COL + half * 64 + c * 16, td);
        tmem_ld_wait();
        [[maybe_unused]] const uint32_t word = (c < 2 ? bits.x : bits.y) >> ((c & 1) * 16);
        uint32_t ph[8], pl[8], dh[8], dl[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float pv[2], dv[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float x = __uint_as_float(ts[i + e]) * p.scale_log2;
            bool on = true;
            if constexpr (MASKED) {
              on = (word >> (i + e)) & 1u;
              x = on ? x : fill;
            }
            const bool in = k0 + half * 64 + c * 16 + i + e < key_lim;
            pv[e] = in ? fast_exp2(x - lse2) : 0.f;
            dv[e] = on ? pv[e] * fmaf(__uint_as_float(td[i + e]), p.scale, -delta_s) : 0.f;    // a masked score is a constant
          }
          ph[i / 2] = split_hi(pv[0], pv[1]);
          pl[i / 2] = split_lo(pv[0], pv[1], ph[i / 2]);
          dh[i / 2] = split_hi(dv[0], dv[1]);
          dl[i / 2] = split_lo(dv[0], dv[1], dh[i / 2]);
        }
        uint8_t* prow = sP + half * (128 * 128) + r * 128;
        uint8_t* drow = sDS + half * (128 * 128) + r * 128;
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int phys = ((c * 2 + v) ^ (r & 7)) * 16;
          *reinterpret_cast<uint4*>(prow + phys) = make_uint4(ph[4 * v], ph[4 * v + 1], ph[4 * v + 2], ph[4 * v + 3]);
          *reinterpret_cast<uint4*>(prow + SPL_PS + phys) = make_uint4(pl[4 * v], pl[4 * v + 1], pl[4 * v + 2], pl[4 * v + 3]);
          *reinterpret_cast<uint4*>(drow + phys) = make_uint4(dh[4 * v], dh[4 * v + 1], dh[4 * v + 2], dh[4 * v + 3]);
          *reinterpret_cast<uint4*>(drow + SPL_PS + phys) = make_uint4(dl[4 * v], dl[4 * v + 1], dl[4 * v + 2], dl[4 * v + 3]);
        }
      }
      tc_fence_before_sync();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(pds_full);
      // ---- dQ of this block: TMEM -> swizzled [32 rows x 32 floats] box -> TMA reduction into the fp32 accumulator
      const bool dq_ok = tc_wait(dq_full, it & 1, stop);
      __syncwarp();
      tc_fence_after_sync();
      if (lane == 0) tma_store_wait_read<0>();                       // this warp's previous box has been read
      __syncwarp();
      uint8_t* box = sDQ + (quad * 2 + half) * SPL_DQ_BOX;
      {
        uint32_t t[32];
        tmem_ld_32x32b_x32(tmem_base + lane_off + DQ_COL + half * 32, t);
        tmem_ld_wait();
        uint8_t* brow = box + lane * 128;
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<uint4*>(brow + ((v ^ (lane & 7)) * 16)) = make_uint4(t[4 * v], t[4 * v + 1], t[4 * v + 2], t[4 * v + 3]);
      }
      tc_fence_before_sync();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(dq_empty);
        if (dq_ok && half * 32 < p.d && q_blk * 128 + quad * 32 < p.Sq) {   // boxes start inside the accumulator; its edge clips them
          asm volatile(
              "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(
                  reinterpret_cast<uint64_t>(&tmap_dq)),
              "r"(half * 32), "r"(q_blk * 128 + quad * 32), "r"(static_cast<int>(bh)), "r"(smem_u32(box))
              : "memory");
        }
        tma_store_commit();
      }
      __syncwarp();
    }
    if (lane == 0) tma_store_wait<0>();
    __syncwarp();
    // ---- dV / dK: thread r <-> key row r
    tc_wait(qdo_empty, (iters - 1) & 1, stop);
    __syncwarp();
    tc_fence_after_sync();
    const int k_idx = k0 + r;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      uint32_t t[32];
      tmem_ld_32x32b_x32(tmem_base + lane_off + (which == 0 ? DV_COL : DK_COL) + half * 32, t);
      tmem_ld_wait();
      if (k_idx < p.Sk) {
        const long* st = which == 0 ? p.dv_strides : p.dk_strides;
        __nv_bfloat16* row = (which == 0 ? p.dv : p.dk) + batch * st[0] + head * st[1] + k_idx * st[2] + half * 32;
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          if (half * 32 + i >= p.d) break;
          *reinterpret_cast<uint4*>(row + i) = make_uint4(
              pack_bf16(__uint_as_float(t[i]), __uint_as_float(t[i + 1])), pack_bf16(__uint_as_float(t[i + 2]), __uint_as_float(t[i + 3])),
              pack_bf16(__uint_as_float(t[i + 4]), __uint_as_float(t[i + 5])), pack_bf16(__uint_as_float(t[i + 6]), __uint_as_float(t[i + 7])));
        }
      }
      __syncwarp();                                                  // whole warps read tensor memory
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*stop) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) { *const_cast<volatile int*>(p.err) = 1; __threadfence_system(); }
    __syncthreads();
  }
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc<512>(tmem_base);
  }
}

// delta[b, a, s] = Σ_d dO · (O + O_lo); 8 lanes per row, rows in memory order of the [b, s, a, d] tensors; clears the dQ accumulator
__global__ void __launch_bounds__(256)
attn_split_delta_kernel(const __nv_bfloat16* __restrict__ dout, long sb, long sa, long ss, const __nv_bfloat16* __restrict__ o,
                        const __nv_bfloat16* __restrict__ o_lo, float* __restrict__ delta, int B, int A, int S, int d,
                        float4* __restrict__ zero_fill, long zero_n4) {
  const long total = static_cast<long>(B) * A * S;
  const long gid = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x, threads = static_cast<long>(gridDim.x) * blockDim.x;
  for (long z = gid; z < zero_n4; z += threads) zero_fill[z] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int sub = threadIdx.x % 8;
  const long warp_first = (gid - threadIdx.x % 32) / 8;
  for (long base = 0; warp_first + base < total; base += threads / 8) {
    const long r = gid / 8 + base;
    float acc = 0.f;
    const int a = static_cast<int>(r % A), s = static_cast<int>((r / A) % S);
    const long b = r / (static_cast<long>(A) * S);
    if (r < total && sub * 8 < d) {
      const uint4 x = *reinterpret_cast<const uint4*>(dout + b * sb + a * sa + s * ss + sub * 8);
      const uint4 y = *reinterpret_cast<const uint4*>(o + r * d + sub * 8), z = *reinterpret_cast<const uint4*>(o_lo + r * d + sub * 8);
      const uint32_t *xw = &x.x, *yw = &y.x, *zw = &z.x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 u = unpack_bf16(xw[e]), v = unpack_bf16(yw[e]), w = unpack_bf16(zw[e]);
        acc += u.x * (v.x + w.x) + u.y * (v.y + w.y);
      }
    }
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (sub == 0 && r < total) delta[(b * A + a) * static_cast<long>(S) + s] = acc;
  }
}

// dq (bf16 view) = accumulator (fp32 [B, A, S, d]), 8 values per thread
__global__ void __launch_bounds__(256)
attn_split_dq_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int B, int A, int S, int d, long sb, long sa, long ss) {
  const long nvec = static_cast<long>(B) * A * S * d / 8;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nvec; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float4 lo = reinterpret_cast<const float4*>(acc)[2 * i], hi = reinterpret_cast<const float4*>(acc)[2 * i + 1];
    const long row = i * 8 / d;
    const int c = static_cast<int>(i * 8 % d), s = static_cast<int>(row % S), a = static_cast<int>((row / S) % A);
    const long b = row / (static_cast<long>(S) * A);
    *reinterpret_cast<uint4*>(dq + b * sb + a * sa + s * ss + c) =
        make_uint4(pack_bf16(lo.x, lo.y), pack_bf16(lo.z, lo.w), pack_bf16(hi.x, hi.y), pack_bf16(hi.z, hi.w));
  }
}

}  // namespace lb

namespace {

// [B, A, S, d] view (strides in elements) as 128-row boxes of 64 columns; the columns behind d are filled with zeros
bool split_tmap(CUtensorMap* m, const void* ptr, int B, int A, int S, int d, const long* st) {
  uint64_t dims[4] = {(uint64_t)d, (uint64_t)S, (uint64_t)A, (uint64_t)B};
  uint64_t strides[4] = {2, (uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
  uint32_t box[4] = {64, 128, 1, 1};
  return lb_host::make_tmap_bf16(m, ptr, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}
bool split_view_ok(const void* ptr, const long* st) {
  return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && st[0] > 0 && st[1] > 0 && st[2] > 0 && ((st[0] | st[1] | st[2]) % 8) == 0;
}
template <typename K>
cudaError_t split_configure(K kern, int smem, bool& done) {
  if (done) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  done = e == cudaSuccess;
  return e;
}
lb::SplitParams split_params(int B, int A, int Sq, int Sk, int d, int causal, float scale, const uint32_t* mask, const float* fill, long mask_b,
                             long mask_a, int* err) {
  lb::SplitParams p{};
  p.B = B; p.A = A; p.Sq = Sq; p.Sk = Sk; p.d = d;
  p.causal = causal; p.off = Sk - Sq;
  p.scale = scale; p.scale_log2 = scale * lb::SPL_LOG2E;
  p.mask = mask; p.fill = fill; p.mask_b = mask_b; p.mask_a = mask_a;
  p.pitch = (Sk + 127) / 128 * 4;
  p.err = err;
  return p;
}
bool split_sizes_ok(int B, int A, int Sq, int Sk, int d, int causal, float scale) {
  return B > 0 && A > 0 && Sq > 0 && Sk > 0 && d >= 8 && d <= 64 && d % 8 == 0 && B <= 65535 && A <= 65535 && scale > 0.f && (!causal || Sk >= Sq);
}
}  // namespace

// words [Bm, Am, Sq, 4 ceil(Sk / 128)], fill [Bm, Am, Sq]; `elem` bytes per mask element, `and_mask` the bits that make it non-zero
extern "C" int lb_attn_mask_pack(const void* mask, int elem, unsigned long long and_mask, int Bm, int Am, int Sq, int Sk, const long* strides,
                                 int causal, int off, uint32_t* words, float* fill, cudaStream_t s) {
  const long rows = (long)Bm * Am * Sq;
  if (rows == 0) return 0;
  const int pitch = (Sk + 127) / 128 * 4;
  long blocks = (rows + 7) / 8;
  if (blocks > 148L * 8) blocks = 148L * 8;
#define LB_GO(U) lb::attn_mask_pack_kernel<U><<<(unsigned)blocks, 256, 0, s>>>((const U*)mask, and_mask, Bm, Am, Sq, Sk, strides[0], strides[1], strides[2], strides[3], causal, off, words, fill, pitch)
  if (elem == 1) LB_GO(uint8_t);
  else if (elem == 2) LB_GO(uint16_t);
  else if (elem == 4) LB_GO(uint32_t);
  else if (elem == 8) LB_GO(unsigned long long);
  else return -1;
#undef LB_GO
  return (int)cudaGetLastError();
}

extern "C" int lb_attn_split_fwd(const void* q, const void* k, const void* v, void* o, void* o_lo, float* lse, int B, int A, int Sq, int Sk, int d,
                                 const long* qs, const long* ks, const long* vs, int causal, float scale, const uint32_t* mask,
                                 const float* fill, long mask_b, long mask_a, int* err, cudaStream_t s) {
  if (!split_sizes_ok(B, A, Sq, Sk, d, causal, scale)) return -1;
  if (!split_view_ok(q, qs) || !split_view_ok(k, ks) || !split_view_ok(v, vs)) return -3;
  CUtensorMap tq, tk, tv;
  if (!split_tmap(&tq, q, B, A, Sq, d, qs) || !split_tmap(&tk, k, B, A, Sk, d, ks) || !split_tmap(&tv, v, B, A, Sk, d, vs)) return -2;
  lb::SplitParams p = split_params(B, A, Sq, Sk, d, causal, scale, mask, fill, mask_b, mask_a, err);
  p.o = (__nv_bfloat16*)o; p.o_lo = (__nv_bfloat16*)o_lo; p.lse = lse;
  static bool c0 = false, c1 = false;
  const dim3 grid((Sq + 127) / 128, A, B);
  cudaError_t e = mask ? split_configure(lb::attn_split_fwd_kernel<true>, lb::SPL_FWD_SMEM, c1) : split_configure(lb::attn_split_fwd_kernel<false>, lb::SPL_FWD_SMEM, c0);
  if (e != cudaSuccess) return (int)e;
  if (mask) lb::attn_split_fwd_kernel<true><<<grid, lb::SPL_THREADS, lb::SPL_FWD_SMEM, s>>>(tq, tk, tv, p);
  else lb::attn_split_fwd_kernel<false><<<grid, lb::SPL_THREADS, lb::SPL_FWD_SMEM, s>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

// dq / dk / dv: [B, A, S, d] views; delta fp32 [B, A, Sq] and dq_acc fp32 [B, A, Sq, d] are scratch
extern "C" int lb_attn_split_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o, const void* o_lo, const float* lse,
                                 void* dq, void* dk, void* dv, float* delta, float* dq_acc, int B, int A, int Sq, int Sk, int d, const long* qs,
                                 const long* ks, const long* vs, const long* dos, const long* dqs, const long* dks, const long* dvs, int causal,
                                 float scale, const uint32_t* mask, const float* fill, long mask_b, long mask_a, int* err, cudaStream_t s) {
  if (!split_sizes_ok(B, A, Sq, Sk, d, causal, scale)) return -1;
  if (!split_view_ok(q, qs) || !split_view_ok(k, ks) || !split_view_ok(v, vs) || !split_view_ok(dout, dos) || !split_view_ok(dq, dqs) ||
      !split_view_ok(dk, dks) || !split_view_ok(dv, dvs))
    return -3;
  CUtensorMap tq, tk, tv, tdo, tdq;
  if (!split_tmap(&tq, q, B, A, Sq, d, qs) || !split_tmap(&tk, k, B, A, Sk, d, ks) || !split_tmap(&tv, v, B, A, Sk, d, vs) ||
      !split_tmap(&tdo, dout, B, A, Sq, d, dos))
    return -2;
  {
    uint64_t dims[3] = {(uint64_t)d, (uint64_t)Sq, (uint64_t)B * A};
    uint64_t strides[3] = {4, (uint64_t)d * 4, (uint64_t)Sq * d * 4};
    uint32_t box[3] = {32, 32, 1};
    if (!lb_host::make_tmap_typed(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, dq_acc, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -2;
  }
  const long rows = (long)B * A * Sq;
  long blocks = (rows * 8 + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  lb::attn_split_delta_kernel<<<(unsigned)blocks, 256, 0, s>>>((const __nv_bfloat16*)dout, dos[0], dos[1], dos[2], (const __nv_bfloat16*)o,
                                                               (const __nv_bfloat16*)o_lo, delta, B, A, Sq, d, (float4*)dq_acc, rows * d / 4);
  lb::SplitParams p = split_params(B, A, Sq, Sk, d, causal, scale, mask, fill, mask_b, mask_a, err);
  p.lse = const_cast<float*>(lse);
  p.delta = delta;
  p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  for (int i = 0; i < 3; ++i) { p.dk_strides[i] = dks[i]; p.dv_strides[i] = dvs[i]; }
  static bool c0 = false, c1 = false;
  const dim3 grid((Sk + 127) / 128, A, B);
  cudaError_t e = mask ? split_configure(lb::attn_split_bwd_kernel<true>, lb::SPL_BWD_SMEM, c1) : split_configure(lb::attn_split_bwd_kernel<false>, lb::SPL_BWD_SMEM, c0);
  if (e != cudaSuccess) return (int)e;
  if (mask) lb::attn_split_bwd_kernel<true><<<grid, lb::SPL_THREADS, lb::SPL_BWD_SMEM, s>>>(tq, tk, tv, tdo, tdq, p);
  else lb::attn_split_bwd_kernel<false><<<grid, lb::SPL_THREADS, lb::SPL_BWD_SMEM, s>>>(tq, tk, tv, tdo, tdq, p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  blocks = (rows * d / 8 + 255) / 256;
  if (blocks > 148L * 8) blocks = 148L * 8;
  lb::attn_split_dq_kernel<<<(unsigned)blocks, 256, 0, s>>>(dq_acc, (__nv_bfloat16*)dq, B, A, Sq, d, dqs[0], dqs[1], dqs[2]);
  return (int)cudaGetLastError();
}

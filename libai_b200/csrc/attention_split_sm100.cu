// Attention with 32-bit probabilities on the tensor cores (tcgen05 / TMEM / TMA): any head dim that is a multiple of 8 up to 64,
// query and key lengths of their own (cross attention), dense 0/1 masks whose masked scores are -10000, causal or full; forward
// and backward.
//
// These calls used to run as unfused fp32 matrix products over [b, a, sq, sk] tensors (head dims 24, 32 and 48 of the shipped GPT,
// BERT and T5 recipes where they run without dropout on the probabilities, every dense mask).  They held probabilities and their
// gradients in 32 bits, and so does this: P and dS go to the tensor core as the sum of three bf16 numbers, which holds all 24 bits of
// an fp32 significand, three MMAs in place of one, accumulated in fp32; the row sums of dO ∘ O use O in fp32.  Two parts (16 bits) are
// not enough: where keys and values share a large common part, dP - δ and Σ dS·K cancel, and dQ of [4, 16, 512, 48] with a
// common part of 20 standard deviations was 1.5e-2 off where the unfused form is 1.7e-3 off (the rounding of its bf16 result);
// now 1.8e-3.  Without a common part all outputs are as far off as the unfused form's to three digits.
// An infinity or NaN comes out as an infinity or NaN, an infinity mostly as a NaN (0 times it in the smaller parts).
//
// Head dims below 64: the tensor maps have the true inner extent, TMA fills columns [d, 64) of the tiles with zeros, which add
// nothing to Q·Kᵀ / dO·Vᵀ; the surplus columns of the other products are not stored.  Masks arrive packed, one bit per (query,
// key), with one fill value per row: -10000 (log2 domain), or 0 for a row without any visible key, whose probabilities are uniform
// whatever the constant (0 keeps its log-sum-exp small and exact).
//
// Bounded by the softmax threads (two passes over S, three roundings per probability), not by the tensor core or memory: key tiles of
// 128, two forward CTAs per SM.  Measured: [16, 512] BERT block with 16 heads of 48 and a padding mask, attention kernels 334 us (199
// backward, 96 forward, 39 around them; 294 us with two parts and unordered sums) where the unfused form took 2470 us; the block 3100 us with
// the unfused form, 877 us with two parts, 918 us now.
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

#include <atomic>

namespace lb {

constexpr int SPL_THREADS = 320;                 // backward: TMA warp, MMA warp, 8 softmax warps
constexpr int SPL_FWD_THREADS = 256;             // forward: 8 softmax warps, one thread of which issues loads and MMAs: two CTAs of more warps get 96 registers, and spill
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
  __nv_bfloat16* o;             // [B, Sq, A, d]
  float* o32;                   // optional: the same before its rounding, for the backward
  float* lse;                   // [B, A, Sq] natural log
  // backward
  const float* delta;           // [B, A, Sq]
  __nv_bfloat16 *dk, *dv;       // [B, A, Sk, d] views
  long dk_strides[3], dv_strides[3];
  int* err;
};

// two fp32 numbers as three bf16 parts each, h + m + l = x to the last bit (8 + 8 + 8 bits of significand; normal range)
LB_DEVICE void split3(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(x0, x1);
  const float2 a = unpack_bf16(h);
  x0 -= a.x;
  x1 -= a.y;
  m = pack_bf16(x0, x1);
  const float2 b = unpack_bf16(m);
  l = pack_bf16(x0 - b.x, x1 - b.y);
}

// ------------------------------------------------------------------------------------------------------------ mask -> bits
// one warp per (batch, head, query) row of the mask as it broadcasts; `and_mask` drops the sign of a floating zero
template <typename U>
__global__ void __launch_bounds__(256)
attn_mask_pack_kernel(const U* __restrict__ mask, unsigned long long and_mask, int Bm, int Am, int Sq, int Sk, long sb, long sa, long sq,
                      long sk, int causal, int off, uint32_t* __restrict__ words, float* __restrict__ fill, int pitch) {
  chain_wait(mask);
  chain_next();
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
// One CTA per (128 queries, head, batch).  S in TMEM columns [0, 128), O in [128, 192), P's first part in [192, 256); the second and third
// parts of 16 keys (8 columns each) overwrite the 16 S columns of those keys once their thread has read them, so the whole fits 256 columns
// and two CTAs share an SM.  S(j+1) is issued after P(j)·V(j) has completed (it overwrites them); the other CTA fills the gap.
// O is added up over the key blocks in registers: the tensor core rounds every addition into its accumulator towards zero, and 24 of them
// per key block leave O, with it δ, some 1e-6 short (dQ of the example above: 8.5e-3 off).
constexpr int SPL_FWD_SMEM = 5 * SPL_TILE + 2 * 2 * 128 * 4 + 1024 + 256;

template <bool MASKED>
__global__ void __launch_bounds__(SPL_FWD_THREADS, 2)
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
  uint64_t* k_full = bars + 1;       // 2
  uint64_t* v_full = bars + 3;       // 2
  uint64_t* s_full = bars + 5;
  uint64_t* p_full = bars + 6;
  uint64_t* o_full = bars + 7;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 9);

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
    for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(o_full, 1);
    *stop = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 0) tmem_alloc<256>(tmem_ptr_smem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  chain_wait();
  chain_next();

  // The block's chain is serial whoever issues it (the other CTA of the SM fills its gaps), so a thread of the softmax warps does.  K(j+1) and
  // V(j+1) go where K(j-1) and V(j-1) were, and o_full(j-1) has said that nothing reads those any more.
  const int ksteps = (p.d + 15) / 16;                                // the columns behind d are zeros
  auto load = [&](int j) {
    const int b = j & 1;
    mbar_arrive_expect_tx(&k_full[b], SPL_TILE);
    tma_load_4d(sK + b * SPL_TILE, &tmap_k, &k_full[b], 0, j * 128, head, batch);
    mbar_arrive_expect_tx(&v_full[b], SPL_TILE);
    tma_load_4d(sV + b * SPL_TILE, &tmap_v, &v_full[b], 0, j * 128, head, batch);
  };
  auto scores = [&](int j) {                                         // S(j)
    constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
    const int b = j & 1;
    if (!tc_wait(&k_full[b], (j >> 1) & 1, stop)) return;
    tc_fence_after_sync();
    const uint32_t q_addr = smem_u32(sQ), k_addr = smem_u32(sK + b * SPL_TILE);
    for (int kk = 0; kk < ksteps; ++kk)
      umma_f16_ss(tmem_base + S_COL, make_smem_desc_sw128(q_addr + kk * 32, 0, 1024), make_smem_desc_sw128(k_addr + kk * 32, 0, 1024), idesc,
                  kk > 0 ? 1u : 0u);
    umma_commit(s_full);
    if (j + 1 < nkv) load(j + 1);
  };
  auto values = [&](int j) {                                         // P(j)·V(j)
    constexpr uint32_t idesc = make_idesc_bf16(128, 64, false, true);
    const int b = j & 1;
    if (!tc_wait(p_full, j & 1, stop) || !tc_wait(&v_full[b], (j >> 1) & 1, stop)) return;
    tc_fence_after_sync();
    const uint32_t v_addr = smem_u32(sV + b * SPL_TILE);
    const uint64_t dv = make_smem_desc_sw128(v_addr, 128 * 128, 1024);
#pragma unroll 1
    for (int part = 2; part >= 0; --part) {                          // smallest first: the accumulator's roundings stay small until the last eight steps
      const uint32_t at = tmem_base + (part == 0 ? P_COL : S_COL + (part - 1) * 8), step = part == 0 ? 8 : 16;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_f16_ts(tmem_base + O_COL, at + kk * step, dv + kk * ((16 * 128) >> 4), idesc, (part < 2 || kk > 0) ? 1u : 0u);
    }
    umma_commit(o_full);
  };
  if (warp_idx == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(q_full, SPL_TILE);
      tma_load_4d(sQ, &tmap_q, q_full, 0, q0, head, batch);
      load(0);
      if (tc_wait(q_full, 0, stop)) scores(0);
    }
    __syncwarp();
  }
  {
    const int quad = warp_idx % 4, half = warp_idx / 4;              // this warp's 64 of the 128 key columns
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
    float m_run = -INFINITY, l_run = 0.f, acc[32];                   // acc: this half's 32 columns of the output row
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
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
        for (int c = 0; c < 4; ++c) {
          uint32_t t[16];
          tmem_ld_32x32b_x16(s_addr + c * 16, t);
          tmem_ld_wait();
          [[maybe_unused]] const uint32_t word = (c < 2 ? bits.x : bits.y) >> ((c & 1) * 16);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float x = __uint_as_float(t[i]) * p.scale_log2;
            if constexpr (MASKED) x = (word >> i) & 1u ? x : fill;
            if constexpr (EDGE) x = k0 + c * 16 + i < key_lim ? x : -INFINITY;
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
      const float m_use = m_run == -INFINITY ? 0.f : m_run;
      float rowsum = 0.f;
      auto pass2 = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {          // 16 keys at a time: 32 would spill
          uint32_t t[16], part[3][8];
          tmem_ld_32x32b_x16(s_addr + c * 16, t);
          tmem_ld_wait();
          [[maybe_unused]] const uint32_t word = (c < 2 ? bits.x : bits.y) >> ((c & 1) * 16);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float x0 = __uint_as_float(t[i]) * p.scale_log2, x1 = __uint_as_float(t[i + 1]) * p.scale_log2;
            if constexpr (MASKED) {
              x0 = (word >> i) & 1u ? x0 : fill;
              x1 = (word >> (i + 1)) & 1u ? x1 : fill;
            }
            x0 = fast_exp2(x0 - m_use);
            x1 = fast_exp2(x1 - m_use);
            if constexpr (EDGE) {
              x0 = k0 + c * 16 + i < key_lim ? x0 : 0.f;
              x1 = k0 + c * 16 + i + 1 < key_lim ? x1 : 0.f;
            }
            rs0 += x0;
            rs1 += x1;
            split3(x0, x1, part[0][i / 2], part[1][i / 2], part[2][i / 2]);
          }
          // (S(j) follows the completion of P(j-1)·V(j-1): all columns are free; the last two parts cover S columns read above)
          tmem_st_32x32b_x8(p_addr + c * 8, part[0]);
          tmem_st_32x32b_x8(s_addr + c * 16, part[1]);
          tmem_st_32x32b_x8(s_addr + c * 16 + 8, part[2]);
        }
        rowsum = rs0 + rs1;
      };
      if (edge) pass2(std::true_type{}); else pass2(std::false_type{});
      l_run = l_run * alpha + rowsum;
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (warp_idx == 0) {
        if (elect_one()) values(j);
        __syncwarp();
      }
      // ---- O = O · alpha + P(j)·V(j), while S(j+1) is computed
      tc_wait(o_full, j & 1, stop);
      __syncwarp();
      tc_fence_after_sync();
      if (warp_idx == 0 && j + 1 < nkv) {
        if (elect_one()) scores(j + 1);
        __syncwarp();
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[16];
        tmem_ld_32x32b_x16(o_addr + c * 16, t);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c * 16 + i] = fmaf(acc[c * 16 + i], alpha, __uint_as_float(t[i]));
      }
    }
    float* xch = sXchg + (nkv & 1) * 256;
    xch[half * 128 + r] = l_run;
    tc_pair_sync(quad);
    l_run += xch[(half ^ 1) * 128 + r];
    const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
    if (q_idx < p.Sq) {
      const size_t at = ((static_cast<size_t>(batch) * p.Sq + q_idx) * p.A + head) * p.d + half * 32;
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        if (half * 32 + i >= p.d) break;                             // d is a multiple of 8
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = acc[i + e] * inv;
        *reinterpret_cast<uint4*>(p.o + at + i) = make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
        if (p.o32 != nullptr) {
          *reinterpret_cast<float4*>(p.o32 + at + i) = make_float4(x[0], x[1], x[2], x[3]);
          *reinterpret_cast<float4*>(p.o32 + at + i + 4) = make_float4(x[4], x[5], x[6], x[7]);
        }
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
  if (warp_idx == 0) {
    tc_fence_after_sync();
    tmem_dealloc<256>(tmem_base);
  }
}

// ----------------------------------------------------------------------------------------------------------------- backward
// One CTA per (128 keys, head, batch), looping over the query blocks that see them, with the keys on the M side:
//   Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ;  P = exp(S - lse), dS = P ∘ (dP - δ) · scale, in three bf16 parts each;
//   dV += Pᵀ·dO with Pᵀ from TMEM, dK += dSᵀ·Q and dQ_i = dS·K with dSᵀ from shared memory.
// dQ_i goes out in fp32, one layer per key block (attn_split_dq_kernel adds the layers up in order): the unfused product had a fixed order,
// and additions into one accumulator by several CTAs have none.
// Six tiles of parts do not fit shared memory beside the operands, so Pᵀ stays in TMEM, which wants it as [keys, queries]: the first part in
// columns of its own, the second and third of 16 queries over the 16 Sᵀ columns that their thread has read.
// Shared memory: K, V, Q, dO 64 KB, three dSᵀ tiles 96 KB, dQ staging 32 KB, two stages of what a query's thread row needs: log-sum-exp, δ, the
// probability of a masked key and the mask bits, one word per (32 keys, query).
constexpr int SPL_PS = 128 * 128 * 2;
constexpr int SPL_DQ_BOX = 32 * 128;
constexpr int SPL_STAT = (3 + 4) * 128;                              // 32-bit words per stage
constexpr int SPL_BWD_SMEM = 4 * SPL_TILE + 3 * SPL_PS + 8 * SPL_DQ_BOX + 2 * SPL_STAT * 4 + 1024 + 256;
static_assert(SPL_BWD_SMEM <= 232448, "split attention backward: shared memory");

template <bool MASKED>
__global__ void __launch_bounds__(SPL_THREADS, 1)
attn_split_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                      const __grid_constant__ CUtensorMap tmap_dq, SplitParams p) {
  constexpr uint32_t S_COL = 0, DP_COL = 128, DV_COL = 256, DK_COL = 320, DQ_COL = 384, P_COL = 448;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + SPL_TILE;
  uint8_t* sQ = sV + SPL_TILE;
  uint8_t* sDO = sQ + SPL_TILE;
  uint8_t* sDS = sDO + SPL_TILE;                // three parts: two chunks of 64 queries, 128 key rows x 128 bytes each
  uint8_t* sDQ = sDS + 3 * SPL_PS;
  uint32_t* sStat = reinterpret_cast<uint32_t*>(sDQ + 8 * SPL_DQ_BOX);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + 2 * SPL_STAT);
  uint64_t* kv_full = bars;
  uint64_t* qdo_full = bars + 1;
  uint64_t* qdo_empty = bars + 2;               // also: the parts of P and dS may be written again (and, with dq_empty, the dQ columns)
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
  chain_wait();
  chain_next();

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
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);   // K·Qᵀ, V·dOᵀ
    constexpr uint32_t idesc_t = make_idesc_bf16(128, 64, false, true);     // Pᵀ·dO, dSᵀ·Q
    constexpr uint32_t idesc_q = make_idesc_bf16(128, 64, true, true);      // dS·K
    const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV), q_addr = smem_u32(sQ), do_addr = smem_u32(sDO), ds_addr = smem_u32(sDS);
    const int ksteps = (p.d + 15) / 16;
    bool ok = __all_sync(0xffffffffu, tc_wait(kv_full, 0, stop));
    for (int it = 0; it < iters; ++it) {
      ok = __all_sync(0xffffffffu, ok && tc_wait(qdo_full, it & 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(tmem_base + S_COL, make_smem_desc_sw128(k_addr + kk * 32, 0, 1024), make_smem_desc_sw128(q_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(tmem_base + DP_COL, make_smem_desc_sw128(v_addr + kk * 32, 0, 1024), make_smem_desc_sw128(do_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        umma_commit(sdp_full);
      }
      __syncwarp();
      ok = __all_sync(0xffffffffu, ok && tc_wait(pds_full, it & 1, stop));
      ok = __all_sync(0xffffffffu, ok && tc_wait(dq_empty, (it & 1) ^ 1, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
#pragma unroll
        for (int part = 0; part < 3; ++part) {       // dQ first: its drain is the only consumer that is waited for
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)             // 16 keys per step
            umma_f16_ss(tmem_base + DQ_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + kk * 2048, 128 * 128, 1024),
                        make_smem_desc_sw128(k_addr + kk * 2048, 128 * 128, 1024), idesc_q, (part > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(dq_full);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {             // 16 queries per step
          const uint64_t bo = make_smem_desc_sw128(do_addr + kk * 2048, 128 * 128, 1024), bq = make_smem_desc_sw128(q_addr + kk * 2048, 128 * 128, 1024);
          umma_f16_ts(tmem_base + DV_COL, tmem_base + P_COL + kk * 8, bo, idesc_t, (it > 0 || kk > 0) ? 1u : 0u);
          umma_f16_ts(tmem_base + DV_COL, tmem_base + S_COL + kk * 16, bo, idesc_t, 1u);
          umma_f16_ts(tmem_base + DV_COL, tmem_base + S_COL + kk * 16 + 8, bo, idesc_t, 1u);
#pragma unroll
          for (int part = 0; part < 3; ++part)
            umma_f16_ss(tmem_base + DK_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + (kk / 4) * (128 * 128) + (kk % 4) * 32, 0, 1024), bq, idesc_t,
                        (it > 0 || kk > 0 || part > 0) ? 1u : 0u);
        }
        umma_commit(qdo_empty);
      }
      __syncwarp();
    }
  } else {
    const int quad = warp_idx % 4, half = (warp_idx - 2) / 4;        // this warp's 32 of the 128 keys, its 64 of a tile's 128 queries
    const int r = quad * 32 + lane, k_idx = k0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const size_t bh = static_cast<size_t>(batch) * p.A + head;
    // what a tile's queries bring along: 128 threads fetch a query's numbers, the other 128 its mask words, one tile ahead
    const int tid = static_cast<int>(threadIdx.x) - 64, fq = tid & 127;
    float f_lse = 0.f, f_delta = 0.f;
    [[maybe_unused]] float f_fill = 0.f;
    [[maybe_unused]] uint4 f_bits = make_uint4(0, 0, 0, 0);
    auto fetch = [&](int it) {
      const int q = min((i_begin + it) * 128 + fq, p.Sq - 1);        // (queries behind Sq are masked below)
      [[maybe_unused]] const long row = MASKED ? batch * p.mask_b + head * p.mask_a + q : 0;
      if (tid < 128) {
        f_lse = p.lse[bh * p.Sq + q];
        f_delta = p.delta[bh * p.Sq + q];
        if constexpr (MASKED) f_fill = p.fill[row];
      } else if constexpr (MASKED) {
        f_bits = *reinterpret_cast<const uint4*>(p.mask + row * p.pitch + k0 / 32);
      }
    };
    fetch(0);
    for (int it = 0; it < iters; ++it) {
      const int q_blk = i_begin + it;
      uint32_t* st = sStat + (it & 1) * SPL_STAT;                    // (whoever still reads the tile before last has not passed the barrier below)
      if (tid < 128) {
        const float lse2 = f_lse * SPL_LOG2E;
        st[fq] = __float_as_uint(lse2);
        st[128 + fq] = __float_as_uint(f_delta * p.scale);
        if constexpr (MASKED) st[256 + fq] = __float_as_uint(fast_exp2(f_fill - lse2));
      } else if constexpr (MASKED) {
        st[384 + fq] = f_bits.x;
        st[512 + fq] = f_bits.y;
        st[640 + fq] = f_bits.z;
        st[768 + fq] = f_bits.w;
      }
      __syncwarp();
      asm volatile("bar.sync 1, 256;\n" ::: "memory");              // the eight warps of this branch
      if (it + 1 < iters) fetch(it + 1);
      // queries [q_lo, q_hi) of this half see key k_idx (the mask apart)
      const int q_first = q_blk * 128 + half * 64;
      const int q_lo = k_idx >= p.Sk ? 128 : (p.causal ? k_idx - p.off - q_first : 0), q_hi = p.Sq - q_first;
      const bool edge = k0 + 128 > p.Sk || q_blk * 128 + 128 > p.Sq || (p.causal && k0 + 127 - p.off > q_blk * 128);
      tc_wait(sdp_full, it & 1, stop);        // S(it) was issued after the products of block it-1 had read the parts of P and dS (one Q stage)
      __syncwarp();
      tc_fence_after_sync();
      auto tile = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
        for (int c = 0; c < 4; ++c) {          // 16 queries at a time
          const int kk = half * 4 + c;
          uint32_t ts[16], td[16];
          tmem_ld_32x32b_x16(tmem_base + lane_off + S_COL + kk * 16, ts);
          tmem_ld_32x32b_x16(tmem_base + lane_off + DP_COL + kk * 16, td);
          tmem_ld_wait();
          uint32_t pp[3][8], dd[3][8];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int at = kk * 16 + v * 4;
            const float4 l4 = *reinterpret_cast<const float4*>(st + at), d4 = *reinterpret_cast<const float4*>(st + 128 + at);
            float4 m4 = make_float4(0.f, 0.f, 0.f, 0.f);
            uint4 w4 = make_uint4(0, 0, 0, 0);
            if constexpr (MASKED) {
              m4 = *reinterpret_cast<const float4*>(st + 256 + at);
              w4 = *reinterpret_cast<const uint4*>(st + 384 + quad * 128 + at);
            }
            const float ls[4] = {l4.x, l4.y, l4.z, l4.w}, de[4] = {d4.x, d4.y, d4.z, d4.w};
            [[maybe_unused]] const float pm[4] = {m4.x, m4.y, m4.z, m4.w};
            [[maybe_unused]] const uint32_t wd[4] = {w4.x, w4.y, w4.z, w4.w};
            float pv[4], dv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int i = 4 * v + e;
              pv[e] = fast_exp2(fmaf(__uint_as_float(ts[i]), p.scale_log2, -ls[e]));
              dv[e] = pv[e] * fmaf(__uint_as_float(td[i]), p.scale, -de[e]);
              if constexpr (MASKED) {
                const bool on = (wd[e] >> lane) & 1u;
                pv[e] = on ? pv[e] : pm[e];
                dv[e] = on ? dv[e] : 0.f;                            // a masked score is a constant
              }
              if constexpr (EDGE) {
                const bool in = c * 16 + i >= q_lo && c * 16 + i < q_hi;
                pv[e] = in ? pv[e] : 0.f;
                dv[e] = in ? dv[e] : 0.f;
              }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              split3(pv[2 * e], pv[2 * e + 1], pp[0][2 * v + e], pp[1][2 * v + e], pp[2][2 * v + e]);
              split3(dv[2 * e], dv[2 * e + 1], dd[0][2 * v + e], dd[1][2 * v + e], dd[2][2 * v + e]);
            }
          }
          tmem_st_32x32b_x8(tmem_base + lane_off + P_COL + kk * 8, pp[0]);
          tmem_st_32x32b_x8(tmem_base + lane_off + S_COL + kk * 16, pp[1]);
          tmem_st_32x32b_x8(tmem_base + lane_off + S_COL + kk * 16 + 8, pp[2]);
          uint8_t* drow = sDS + half * (128 * 128) + r * 128;
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const int phys = ((c * 2 + v) ^ (r & 7)) * 16;
#pragma unroll
            for (int part = 0; part < 3; ++part)
              *reinterpret_cast<uint4*>(drow + part * SPL_PS + phys) = make_uint4(dd[part][4 * v], dd[part][4 * v + 1], dd[part][4 * v + 2], dd[part][4 * v + 3]);
          }
        }
      };
      if (edge) tile(std::true_type{}); else tile(std::false_type{});
      tmem_st_wait();
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
        if (dq_ok && half * 32 < p.d && q_blk * 128 + quad * 32 < p.Sq) {   // boxes start inside the layer; its edge clips them
          asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(reinterpret_cast<uint64_t>(&tmap_dq)),
                       "r"(half * 32), "r"(q_blk * 128 + quad * 32), "r"(static_cast<int>(blockIdx.x * gridDim.z * gridDim.y + bh)), "r"(smem_u32(box))
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

// delta[b, a, s] = Σ_d dO · O, O as the forward left it in fp32; 8 lanes per row, rows in memory order of the [b, s, a, d] tensors
__global__ void __launch_bounds__(256)
attn_split_delta_kernel(const __nv_bfloat16* __restrict__ dout, long sb, long sa, long ss, const float* __restrict__ o32,
                        float* __restrict__ delta, int B, int A, int S, int d) {
  chain_wait(dout, o32);
  chain_next();
  const long total = static_cast<long>(B) * A * S;
  const long gid = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x, threads = static_cast<long>(gridDim.x) * blockDim.x;
  const int sub = threadIdx.x % 8;
  const long warp_first = (gid - threadIdx.x % 32) / 8;
  for (long base = 0; warp_first + base < total; base += threads / 8) {
    const long r = gid / 8 + base;
    float acc = 0.f;
    const int a = static_cast<int>(r % A), s = static_cast<int>((r / A) % S);
    const long b = r / (static_cast<long>(A) * S);
    if (r < total && sub * 8 < d) {
      const uint4 x = *reinterpret_cast<const uint4*>(dout + b * sb + a * sa + s * ss + sub * 8);
      const float4 y = *reinterpret_cast<const float4*>(o32 + r * d + sub * 8), z = *reinterpret_cast<const float4*>(o32 + r * d + sub * 8 + 4);
      const float2 u0 = unpack_bf16(x.x), u1 = unpack_bf16(x.y), u2 = unpack_bf16(x.z), u3 = unpack_bf16(x.w);
      acc = ((u0.x * y.x + u0.y * y.y) + (u1.x * y.z + u1.y * y.w)) + ((u2.x * z.x + u2.y * z.y) + (u3.x * z.z + u3.y * z.w));
    }
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (sub == 0 && r < total) delta[(b * A + a) * static_cast<long>(S) + s] = acc;
  }
}

// dq (bf16 view) = the sum of its layers (fp32 [key blocks, B, A, S, d]) in the order of the key blocks, 8 values per thread.  Under the causal
// mask (off >= 0) a block of 128 queries has the layers of the key blocks that it sees.
__global__ void __launch_bounds__(256)
attn_split_dq_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int B, int A, int S, int d, long sb, long sa, long ss,
                     int key_blocks, int causal, int off) {
  chain_next();
  const long nvec = static_cast<long>(B) * A * S * d / 8;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nvec; i += static_cast<long>(gridDim.x) * blockDim.x) {
    const long row = i * 8 / d;
    const int c = static_cast<int>(i * 8 % d), s = static_cast<int>(row % S), a = static_cast<int>((row / S) % A);
    const long b = row / (static_cast<long>(S) * A);
    const int layers = causal ? min(key_blocks, (s / 128 * 128 + 127 + off) / 128 + 1) : key_blocks;
    const float4* src = reinterpret_cast<const float4*>(acc) + 2 * i;
    float4 lo = src[0], hi = src[1];
#pragma unroll 4
    for (int k = 1; k < layers; ++k) {
      const float4 x = src[2 * nvec * k], y = src[2 * nvec * k + 1];
      lo.x += x.x; lo.y += x.y; lo.z += x.z; lo.w += x.w;
      hi.x += y.x; hi.y += y.y; hi.z += y.z; hi.w += y.w;
    }
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
// a function's limit on dynamic shared memory is per device: these calls ran on any device of a process before, and do
template <typename K>
cudaError_t split_configure(K kern, int smem, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
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
#define LB_GO(U) lb_host::launch_chained(lb::attn_mask_pack_kernel<U>, dim3((unsigned)blocks), dim3(256), 0, s, 0, (const U*)mask, and_mask, Bm, Am, Sq, Sk, strides[0], strides[1], strides[2], strides[3], causal, off, words, fill, pitch)
  if (elem == 1) LB_GO(uint8_t);
  else if (elem == 2) LB_GO(uint16_t);
  else if (elem == 4) LB_GO(uint32_t);
  else if (elem == 8) LB_GO(unsigned long long);
  else return -1;
#undef LB_GO
  return (int)cudaGetLastError();
}

extern "C" int lb_attn_split_fwd(const void* q, const void* k, const void* v, void* o, float* o32, float* lse, int B, int A, int Sq, int Sk, int d,
                                 const long* qs, const long* ks, const long* vs, int causal, float scale, const uint32_t* mask,
                                 const float* fill, long mask_b, long mask_a, int* err, cudaStream_t s) {
  if (!split_sizes_ok(B, A, Sq, Sk, d, causal, scale)) return -1;
  if (!split_view_ok(q, qs) || !split_view_ok(k, ks) || !split_view_ok(v, vs)) return -3;
  CUtensorMap tq, tk, tv;
  if (!split_tmap(&tq, q, B, A, Sq, d, qs) || !split_tmap(&tk, k, B, A, Sk, d, ks) || !split_tmap(&tv, v, B, A, Sk, d, vs)) return -2;
  lb::SplitParams p = split_params(B, A, Sq, Sk, d, causal, scale, mask, fill, mask_b, mask_a, err);
  p.o = (__nv_bfloat16*)o; p.o32 = o32; p.lse = lse;
  static std::atomic<unsigned long long> c0{0}, c1{0};
  const dim3 grid((Sq + 127) / 128, A, B);
  cudaError_t e = mask ? split_configure(lb::attn_split_fwd_kernel<true>, lb::SPL_FWD_SMEM, c1) : split_configure(lb::attn_split_fwd_kernel<false>, lb::SPL_FWD_SMEM, c0);
  if (e != cudaSuccess) return (int)e;
  return (int)lb_host::launch_chained(mask ? lb::attn_split_fwd_kernel<true> : lb::attn_split_fwd_kernel<false>, grid, dim3(lb::SPL_FWD_THREADS), lb::SPL_FWD_SMEM, s, 0,
                                      tq, tk, tv, p);
}

// dq / dk / dv: [B, A, S, d] views; delta fp32 [B, A, Sq] and dq_acc fp32 [ceil(Sk / 128), B, A, Sq, d] are scratch
extern "C" int lb_attn_split_bwd(const void* dout, const void* q, const void* k, const void* v, const float* o32, const float* lse, void* dq,
                                 void* dk, void* dv, float* delta, float* dq_acc, int B, int A, int Sq, int Sk, int d, const long* qs,
                                 const long* ks, const long* vs, const long* dos, const long* dqs, const long* dks, const long* dvs, int causal,
                                 float scale, const uint32_t* mask, const float* fill, long mask_b, long mask_a, int* err, cudaStream_t s) {
  if (!split_sizes_ok(B, A, Sq, Sk, d, causal, scale)) return -1;
  if (!split_view_ok(q, qs) || !split_view_ok(k, ks) || !split_view_ok(v, vs) || !split_view_ok(dout, dos) || !split_view_ok(dq, dqs) ||
      !split_view_ok(dk, dks) || !split_view_ok(dv, dvs))
    return -3;
  const int key_blocks = (Sk + 127) / 128;
  if ((long)B * A * key_blocks > 0x7fffffffL) return -1;
  CUtensorMap tq, tk, tv, tdo, tdq;
  if (!split_tmap(&tq, q, B, A, Sq, d, qs) || !split_tmap(&tk, k, B, A, Sk, d, ks) || !split_tmap(&tv, v, B, A, Sk, d, vs) ||
      !split_tmap(&tdo, dout, B, A, Sq, d, dos))
    return -2;
  {
    uint64_t dims[3] = {(uint64_t)d, (uint64_t)Sq, (uint64_t)B * A * key_blocks};
    uint64_t strides[3] = {4, (uint64_t)d * 4, (uint64_t)Sq * d * 4};
    uint32_t box[3] = {32, 32, 1};
    if (!lb_host::make_tmap_typed(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, dq_acc, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -2;
  }
  const long rows = (long)B * A * Sq;
  long blocks = (rows * 8 + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  lb_host::launch_chained(lb::attn_split_delta_kernel, dim3((unsigned)blocks), dim3(256), 0, s, 0, (const __nv_bfloat16*)dout, dos[0], dos[1], dos[2], o32, delta, B, A, Sq, d);
  lb::SplitParams p = split_params(B, A, Sq, Sk, d, causal, scale, mask, fill, mask_b, mask_a, err);
  p.lse = const_cast<float*>(lse);
  p.delta = delta;
  p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  for (int i = 0; i < 3; ++i) { p.dk_strides[i] = dks[i]; p.dv_strides[i] = dvs[i]; }
  static std::atomic<unsigned long long> c0{0}, c1{0};
  const dim3 grid(key_blocks, A, B);
  cudaError_t e = mask ? split_configure(lb::attn_split_bwd_kernel<true>, lb::SPL_BWD_SMEM, c1) : split_configure(lb::attn_split_bwd_kernel<false>, lb::SPL_BWD_SMEM, c0);
  if (e != cudaSuccess) return (int)e;
  lb_host::launch_chained(mask ? lb::attn_split_bwd_kernel<true> : lb::attn_split_bwd_kernel<false>, grid, dim3(lb::SPL_THREADS), lb::SPL_BWD_SMEM, s, 0, tq, tk, tv, tdo,
                          tdq, p);
  e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  blocks = (rows * d / 8 + 255) / 256;
  if (blocks > 148L * 8) blocks = 148L * 8;
  lb::attn_split_dq_kernel<<<(unsigned)blocks, 256, 0, s>>>(dq_acc, (__nv_bfloat16*)dq, B, A, Sq, d, dqs[0], dqs[1], dqs[2], key_blocks,
                                                              causal, Sk - Sq);
  return (int)cudaGetLastError();
}

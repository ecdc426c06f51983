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
// 128, two forward CTAs per SM.  Measured: [16, 512] BERT block with 16 heads of 48 and a padding mask, attention kernels 285 us (168
// backward, 78 forward, 39 around them) where the unfused form took 2470 us; forward 101 -> 78 us since rows of the mask that are all visible or all masked for a warp's
// keys take no look at single bits, the largest score is scaled once and remainders need no unpacking (without a mask 152 -> 144, [4, 2048] 16 x 48 causal).
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

#include <atomic>

namespace lb {

constexpr int SPL_THREADS = 384;                 // backward: TMA warp, MMA warp, two that keep their warpgroup whole, 8 softmax warps
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
// x0 - the lower, x1 - the upper bf16 of h, exactly (the multiply-add takes a bf16 factor as it is: no unpacking)
LB_DEVICE void minus_bf16x2(float& x0, float& x1, uint32_t h) {
  asm("{\n\t.reg .b16 a, b, m;\n\tmov.b32 {a, b}, %2;\n\tmov.b16 m, 0xBF80;\n\t"
      "fma.rn.f32.bf16 %0, a, m, %0;\n\tfma.rn.f32.bf16 %1, b, m, %1;\n\t}\n"
      : "+f"(x0), "+f"(x1)
      : "r"(h));
}
LB_DEVICE void split3(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16(x0, x1);
  minus_bf16x2(x0, x1, h);
  m = pack_bf16(x0, x1);
  minus_bf16x2(x0, x1, m);
  l = pack_bf16(x0, x1);
}

// two numbers per instruction: x * f + c and x * y
LB_DEVICE float2 fma2(float x0, float x1, float f, float c0, float c1) {
  float2 r;
  asm("{\n\t.reg .b64 x, f, c;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 f, {%4, %4};\n\tmov.b64 c, {%5, %6};\n\tfma.rn.f32x2 x, x, f, c;\n\tmov.b64 {%0, %1}, x;\n\t}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x0), "f"(x1), "f"(f), "f"(c0), "f"(c1));
  return r;
}
LB_DEVICE float2 mul2(float x0, float x1, float2 y) {
  float2 r;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}\n"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x0), "f"(x1), "f"(y.x), "f"(y.y));
  return r;
}
// a 32 x 32 matrix of bits, one row per lane, transposed
LB_DEVICE uint32_t transpose_bits(uint32_t x, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? (x & ~m) | ((y & ~m) >> j) : (x & m) | ((y & m) << j);
  }
  return x;
}
// bits [lo, hi) of a word
LB_DEVICE uint32_t bit_range(int lo, int hi) {
  const uint32_t below_hi = hi >= 32 ? 0xffffffffu : hi <= 0 ? 0u : (1u << hi) - 1u, below_lo = lo >= 32 ? 0xffffffffu : lo <= 0 ? 0u : (1u << lo) - 1u;
  return below_hi & ~below_lo;
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
    const uint32_t idesc = make_idesc_bf16(128, ksteps * 16, false, true);
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
      // MASK: a warp's 32 queries and 64 keys are looked at one by one (1), all masked (2) or all visible (0)
      float mx = -INFINITY;
      auto pass1 = [&](auto edge_tag, auto mask_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        constexpr int MASK = decltype(mask_tag)::value;
        if constexpr (MASK == 2) {
          mx = fill;
          return;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t t[16];
          tmem_ld_32x32b_x16(s_addr + c * 16, t);
          tmem_ld_wait();
          [[maybe_unused]] const uint32_t word = (c < 2 ? bits.x : bits.y) >> ((c & 1) * 16);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float x = __uint_as_float(t[i]);
            if constexpr (MASK == 1) x = word & (1u << i) ? x : -INFINITY;
            if constexpr (EDGE) x = k0 + c * 16 + i < key_lim ? x : -INFINITY;
            mx = fmaxf(mx, x);
          }
        }
        mx *= p.scale_log2;                      // (scale > 0: the largest product)
        if constexpr (MASK == 1) {               // a masked key within the sequence counts with its fill
          const int keys = EDGE ? min(64, key_lim - k0) : 64;
          const bool any = ((~bits.x & bit_range(0, keys)) | (~bits.y & bit_range(0, keys - 32))) != 0u;
          mx = any ? fmaxf(mx, fill) : mx;
        }
      };
      using std::integral_constant;
      [[maybe_unused]] int mode = 0;
      if constexpr (MASKED) {
        const bool on = __all_sync(0xffffffffu, (bits.x & bits.y) == 0xffffffffu), off = __all_sync(0xffffffffu, (bits.x | bits.y) == 0u);
        mode = edge ? 1 : on ? 0 : off ? 2 : 1;
      }
      auto by_mode = [&](auto f) {
        if constexpr (MASKED) {
          if (edge) f(std::true_type{}, integral_constant<int, 1>{});
          else if (mode == 0) f(std::false_type{}, integral_constant<int, 0>{});
          else if (mode == 2) f(std::false_type{}, integral_constant<int, 2>{});
          else f(std::false_type{}, integral_constant<int, 1>{});
        } else {
          if (edge) f(std::true_type{}, integral_constant<int, 0>{}); else f(std::false_type{}, integral_constant<int, 0>{});
        }
      };
      by_mode(pass1);
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
      auto pass2 = [&](auto edge_tag, auto mask_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
        constexpr int MASK = decltype(mask_tag)::value;
        [[maybe_unused]] float masked = 0.f;     // probability of a masked key
        if constexpr (MASK != 0) masked = fast_exp2(fill - m_use);
        float rs0 = 0.f, rs1 = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {          // 16 keys at a time: 32 would spill
          uint32_t t[16], part[3][8];
          if constexpr (MASK != 2) {
            tmem_ld_32x32b_x16(s_addr + c * 16, t);
            tmem_ld_wait();
          }
          [[maybe_unused]] const uint32_t word = (c < 2 ? bits.x : bits.y) >> ((c & 1) * 16);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float2 x = make_float2(masked, masked);
            if constexpr (MASK != 2) {
              x = fma2(__uint_as_float(t[i]), __uint_as_float(t[i + 1]), p.scale_log2, -m_use, -m_use);
              x.x = fast_exp2(x.x);
              x.y = fast_exp2(x.y);
            }
            if constexpr (MASK == 1) {
              x.x = word & (1u << i) ? x.x : masked;
              x.y = word & (2u << i) ? x.y : masked;
            }
            if constexpr (EDGE) {
              x.x = k0 + c * 16 + i < key_lim ? x.x : 0.f;
              x.y = k0 + c * 16 + i + 1 < key_lim ? x.y : 0.f;
            }
            rs0 += x.x;
            rs1 += x.y;
            split3(x.x, x.y, part[0][i / 2], part[1][i / 2], part[2][i / 2]);
          }
          // (S(j) follows the completion of P(j-1)·V(j-1): all columns are free; the last two parts cover S columns read above)
          tmem_st_32x32b_x8(p_addr + c * 8, part[0]);
          tmem_st_32x32b_x8(s_addr + c * 16, part[1]);
          tmem_st_32x32b_x8(s_addr + c * 16 + 8, part[2]);
        }
        rowsum = rs0 + rs1;
      };
      by_mode(pass2);
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
// Work items of (128 keys, head, batch), looping over the query blocks that see them, with the keys on the M side:
//   Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ;  P = exp(S - lse), dS = P ∘ (dP - δ) · scale, in three bf16 parts each;
//   dV += Pᵀ·dO with Pᵀ from TMEM, dK += dSᵀ·Q and dQ_i = dS·K with dSᵀ from shared memory.
// dQ_i goes out in fp32, one layer per key block (attn_split_dq_kernel adds the layers up in order): the unfused product had a fixed order,
// and additions into one accumulator by several CTAs have none.
// Six tiles of parts do not fit shared memory beside the operands, so Pᵀ stays in TMEM, which wants it as [keys, queries]: the first part in
// columns of its own, the second and third of 16 queries over the 16 Sᵀ columns that their thread has read.
// Shared memory: K, V 32 KB, two stages of Q and dO 64 KB, three dSᵀ tiles 96 KB, dQ staging 32 KB, what a query's thread row needs: log-sum-exp, δ, the
// probability of a masked key (mask words are transposed between the lanes).
// Bounded by the softmax threads' instructions (1700 per warp and block of 128 x 128, 3400 cycles on their schedulers) and the 72 small products (26 to 60 cycles
// each: their A operands are 4 KB for 128 x 64 results).  So the two run side by side as far as the one buffer of dSᵀ allows: P is made first and dV runs while dS
// is made from the probabilities kept in registers; Sᵀ and dPᵀ of the next block go out as soon as dS is there, in front of dK and dQ, Sᵀ to where dPᵀ was and the other way
// round; the threads make the next P meanwhile and wait for dQ before they write its dSᵀ.  CTAs stay for several work items: the next one's Q and dO are loaded and its numbers
// fetched while this one ends.  A block took 14200 cycles with everything in turn, now 8000.  Rows of the mask that are all visible or all masked for a warp's keys take
// no look at single bits.  The split into three parts takes its remainders with a multiply-add that reads bf16 factors (310 -> 283 us; 2048 below), scales two scores per instruction.
// Measured, us: [16, 512] 16 heads of 48 with a padding mask 201 -> 169, [4, 2048] 16 x 48 causal 375 -> 280, [8, 1024] 16 x 24 causal 211 -> 156, [1, 1024] 16 x 48 47 -> 38,
// [64, 128] 16 x 32 63 -> 54, 128 queries against 512 keys (16, 12 x 32, masked) 53 -> 46; [16, 128] 12 x 32 masked 19.5 -> 20.5 (192 items, two for some CTAs).
constexpr int SPL_PS = 128 * 128 * 2;
constexpr int SPL_DQ_BOX = 32 * 128;
constexpr int SPL_BWD_SMEM = 6 * SPL_TILE + 3 * SPL_PS + 8 * SPL_DQ_BOX + 3 * 128 * 4 + 1024 + 128;
static_assert(SPL_BWD_SMEM <= 232448, "split attention backward: shared memory");

template <bool MASKED>
__global__ void __launch_bounds__(SPL_THREADS, 1)
attn_split_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                      const __grid_constant__ CUtensorMap tmap_dq, SplitParams p) {
  constexpr uint32_t DV_COL = 256, DK_COL = 320, DQ_COL = 384, P_COL = 448;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + SPL_TILE;
  uint8_t* sQ = sV + SPL_TILE;                  // 2
  uint8_t* sDO = sQ + 2 * SPL_TILE;             // 2
  uint8_t* sDS = sDO + 2 * SPL_TILE;            // three parts: two chunks of 64 queries, 128 key rows x 128 bytes each
  uint8_t* sDQ = sDS + 3 * SPL_PS;
  uint32_t* sStat = reinterpret_cast<uint32_t*>(sDQ + 8 * SPL_DQ_BOX);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + 3 * 128);
  uint64_t* kv_full = bars;
  uint64_t* sdp_full = bars + 1;
  uint64_t* p_full = bars + 2;
  uint64_t* ds_full = bars + 10;                // and dPᵀ and the dQ of the block before are read
  uint64_t* dv_done = bars + 3;
  uint64_t* dq_done = bars + 4;                 // and everything issued before: dS may be written again
  uint64_t* qdo_full = bars + 5;                // 2
  uint64_t* qdo_empty = bars + 7;               // 2
  uint64_t* kv_empty = bars + 9;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 12);

  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  // work items: blocks of 128 keys of a head, those with the most query blocks first; CTA c takes c, c + CTAs, ..
  const int heads = p.A * p.B, items = (p.Sk + 127) / 128 * heads, nq = (p.Sq + 127) / 128;
  struct Item {
    int k0, head, batch, i_begin, iters;
  };
  auto item_of = [&](int item) {
    Item w;
    const int bh = item % heads;
    w.k0 = item / heads * 128;
    w.head = bh % p.A;
    w.batch = bh / p.A;
    w.i_begin = p.causal ? max(0, w.k0 - p.off) / 128 : 0;           // the first query that sees key k0 is k0 - off
    w.iters = nq - w.i_begin;                                        // >= 1: off >= 0 under the causal mask
    return w;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_dq);
    for (int i = 0; i < 11; ++i) mbar_init(bars + i, i == 2 || i == 10 ? 8 : 1);
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
  // The softmax threads hold a block's probabilities: 3 x 168 registers as launched, 88 + 2 x 208 from here on.
  if (warp_idx < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;\n");
    if (warp_idx == 0) {
      if (elect_one()) {
        int t = 0, n = 0;                                              // blocks and items so far
        for (int item = blockIdx.x; item < items; item += gridDim.x, ++n) {
          const Item w = item_of(item);
          for (int it = 0; it < w.iters; ++it, ++t) {
            const int b = t & 1, q = (w.i_begin + it) * 128;
            if (!tc_wait(&qdo_empty[b], ((t >> 1) & 1) ^ 1, stop)) continue;
            mbar_arrive_expect_tx(&qdo_full[b], 2 * SPL_TILE);
            tma_load_4d(sQ + b * SPL_TILE, &tmap_q, &qdo_full[b], 0, q, w.head, w.batch);
            tma_load_4d(sDO + b * SPL_TILE, &tmap_do, &qdo_full[b], 0, q, w.head, w.batch);
            if (it == 0 && tc_wait(kv_empty, (n & 1) ^ 1, stop)) {     // (the item's first Q and dO do not wait for this)
              mbar_arrive_expect_tx(kv_full, 2 * SPL_TILE);
              tma_load_4d(sK, &tmap_k, kv_full, 0, w.k0, w.head, w.batch);
              tma_load_4d(sV, &tmap_v, kv_full, 0, w.k0, w.head, w.batch);
            }
          }
        }
      }
      __syncwarp();
    } else if (warp_idx == 1) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);   // K·Qᵀ, V·dOᵀ
      const int dcols = (p.d + 15) / 16 * 16;                                 // columns of the products with d (those behind d are zeros, and not stored)
      const uint32_t idesc_t = make_idesc_bf16(128, dcols, false, true);      // Pᵀ·dO, dSᵀ·Q
      const uint32_t idesc_q = make_idesc_bf16(128, dcols, true, true);       // dS·K
      const uint32_t k_addr = smem_u32(sK), v_addr = smem_u32(sV), ds_addr = smem_u32(sDS);
      const int ksteps = (p.d + 15) / 16;
      auto s_col = [&](int t) { return tmem_base + (t & 1) * 128; };          // Sᵀ of block t, dPᵀ of the block before
      auto scores = [&](int t) {                       // Sᵀ and dPᵀ of block t
        const uint32_t q_addr = smem_u32(sQ + (t & 1) * SPL_TILE), do_addr = smem_u32(sDO + (t & 1) * SPL_TILE);
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(s_col(t), make_smem_desc_sw128(k_addr + kk * 32, 0, 1024), make_smem_desc_sw128(q_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        for (int kk = 0; kk < ksteps; ++kk)
          umma_f16_ss(s_col(t + 1), make_smem_desc_sw128(v_addr + kk * 32, 0, 1024), make_smem_desc_sw128(do_addr + kk * 32, 0, 1024), idesc_s,
                      kk > 0 ? 1u : 0u);
        umma_commit(sdp_full);
      };
      bool ok = true;
      int t = 0, n = 0;
      for (int item = blockIdx.x; item < items; item += gridDim.x, ++n) {
        const int iters = item_of(item).iters;
        ok = __all_sync(0xffffffffu, ok && tc_wait(kv_full, n & 1, stop) && tc_wait(&qdo_full[t & 1], (t >> 1) & 1, stop));
        tc_fence_after_sync();
        if (ok && elect_one()) scores(t);                // (K came after every product of the item before had completed)
        __syncwarp();
        for (int it = 0; it < iters; ++it, ++t) {
          const int b = t & 1;
          const uint32_t q_addr = smem_u32(sQ + b * SPL_TILE), do_addr = smem_u32(sDO + b * SPL_TILE);
          ok = __all_sync(0xffffffffu, ok && tc_wait(p_full, t & 1, stop));
          tc_fence_after_sync();
          if (ok && elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {             // 16 queries per step
              const uint64_t bo = make_smem_desc_sw128(do_addr + kk * 2048, 128 * 128, 1024);
              umma_f16_ts(tmem_base + DV_COL, tmem_base + P_COL + kk * 8, bo, idesc_t, (it > 0 || kk > 0) ? 1u : 0u);
              umma_f16_ts(tmem_base + DV_COL, s_col(t) + kk * 16, bo, idesc_t, 1u);
              umma_f16_ts(tmem_base + DV_COL, s_col(t) + kk * 16 + 8, bo, idesc_t, 1u);
            }
            umma_commit(dv_done);
          }
          __syncwarp();
          ok = __all_sync(0xffffffffu, ok && tc_wait(ds_full, t & 1, stop));
          tc_fence_after_sync();
          if (it + 1 < iters) {
            ok = __all_sync(0xffffffffu, ok && tc_wait(&qdo_full[b ^ 1], ((t + 1) >> 1) & 1, stop));
            ok = __all_sync(0xffffffffu, ok && tc_wait(dv_done, t & 1, stop));
            tc_fence_after_sync();
            if (ok && elect_one()) scores(t + 1);
            __syncwarp();
          }
          if (ok && elect_one()) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
              const uint64_t bq = make_smem_desc_sw128(q_addr + kk * 2048, 128 * 128, 1024);
#pragma unroll
              for (int part = 0; part < 3; ++part)
                umma_f16_ss(tmem_base + DK_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + (kk / 4) * (128 * 128) + (kk % 4) * 32, 0, 1024), bq, idesc_t,
                            (it > 0 || kk > 0 || part > 0) ? 1u : 0u);
            }
            umma_commit(&qdo_empty[b]);
#pragma unroll
            for (int part = 0; part < 3; ++part) {
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)             // 16 keys per step
                umma_f16_ss(tmem_base + DQ_COL, make_smem_desc_sw128(ds_addr + part * SPL_PS + kk * 2048, 128 * 128, 1024),
                            make_smem_desc_sw128(k_addr + kk * 2048, 128 * 128, 1024), idesc_q, (part > 0 || kk > 0) ? 1u : 0u);
            }
            umma_commit(dq_done);
            if (it + 1 == iters) umma_commit(kv_empty);
          }
          __syncwarp();
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;\n");
    const int quad = warp_idx % 4, half = warp_idx / 4 - 1;          // this warp's 32 of the 128 keys, its 64 of a tile's 128 queries
    const int r = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    // what a block's queries bring along, fetched one block ahead: 128 threads a query's numbers, every warp the mask words of its 64 queries, two per lane
    const int tid = static_cast<int>(threadIdx.x) - 128, fq = tid & 127;
    float f_lse = 0.f, f_delta = 0.f;
    [[maybe_unused]] float f_fill = 0.f;
    [[maybe_unused]] uint32_t f_bits[2] = {0u, 0u};
    auto fetch = [&](const Item& w, int it) {
      const int q_tile = (w.i_begin + it) * 128, q = min(q_tile + fq, p.Sq - 1);      // (queries behind Sq are masked below)
      [[maybe_unused]] const long base = MASKED ? w.batch * p.mask_b + w.head * p.mask_a : 0;
      const size_t bh = static_cast<size_t>(w.batch) * p.A + w.head;
      if (tid < 128) {
        f_lse = p.lse[bh * p.Sq + q];
        f_delta = p.delta[bh * p.Sq + q];
        if constexpr (MASKED) f_fill = p.fill[base + q];
      }
      if constexpr (MASKED) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          f_bits[i] = p.mask[(base + min(q_tile + half * 64 + i * 32 + lane, p.Sq - 1)) * p.pitch + w.k0 / 32 + quad];
      }
    };
    // dQ of block t, query block q_blk of the item: TMEM -> swizzled [32 rows x 32 floats] box -> TMA store into its layer of the fp32 accumulator
    auto drain = [&](int t, int item, int q_blk) {
      const bool dq_ok = tc_wait(dq_done, t & 1, stop);
      __syncwarp();
      tc_fence_after_sync();
      if (lane == 0) tma_store_wait_read<0>();                       // this warp's previous box has been read
      __syncwarp();
      uint8_t* box = sDQ + (quad * 2 + half) * SPL_DQ_BOX;
      uint8_t* brow = box + lane * 128;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[16];
        tmem_ld_32x32b_x16(tmem_base + lane_off + DQ_COL + half * 32 + c * 16, t);
        tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 4; ++v)
          *reinterpret_cast<uint4*>(brow + (((c * 4 + v) ^ (lane & 7)) * 16)) = make_uint4(t[4 * v], t[4 * v + 1], t[4 * v + 2], t[4 * v + 3]);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        const int q = q_blk * 128 + quad * 32;
        if (dq_ok && half * 32 < p.d && q < p.Sq) {                  // boxes start inside the layer; its edge clips them
          asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(reinterpret_cast<uint64_t>(&tmap_dq)),
                       "r"(half * 32), "r"(q), "r"(item), "r"(smem_u32(box))
                       : "memory");
        }
        tma_store_commit();
      }
      __syncwarp();
    };
    int t = 0;
    fetch(item_of(blockIdx.x), 0);
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const Item w = item_of(item);
      const int k0 = w.k0, k_idx = k0 + r, i_begin = w.i_begin, iters = w.iters;
      for (int it = 0; it < iters; ++it, ++t) {
        const int q_blk = i_begin + it;
        uint32_t* st = sStat;
        [[maybe_unused]] const uint32_t bits[2] = {f_bits[0], f_bits[1]};
        if (t > 0) asm volatile("bar.sync 1, 256;\n" ::: "memory");   // the eight warps of this branch have read the block before's
        if (tid < 128) {
          const float lse2 = f_lse * SPL_LOG2E;
          st[fq] = __float_as_uint(-lse2);                         // (negative: addends as they are)
          st[128 + fq] = __float_as_uint(-(f_delta * p.scale));
          if constexpr (MASKED) st[256 + fq] = __float_as_uint(fast_exp2(f_fill - lse2));
        }
        __syncwarp();
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (it + 1 < iters) fetch(w, it + 1);
        else if (item + static_cast<int>(gridDim.x) < items) fetch(item_of(item + gridDim.x), 0);
        // queries [q_lo, q_hi) of this half see key k_idx (the mask apart)
        const int q_first = q_blk * 128 + half * 64;
        const int q_lo = k_idx >= p.Sk ? 128 : (p.causal ? k_idx - p.off - q_first : 0), q_hi = p.Sq - q_first;
        const bool edge = k0 + 128 > p.Sk || q_blk * 128 + 128 > p.Sq || (p.causal && k0 + 127 - p.off > q_blk * 128);
        tc_wait(sdp_full, t & 1, stop);         // S(t) and dP(t) were issued after dV of block t-1 had read the parts of P
        __syncwarp();
        tc_fence_after_sync();
        const uint32_t s_addr = tmem_base + lane_off + (t & 1) * 128 + half * 64, dp_addr = tmem_base + lane_off + (~t & 1) * 128 + half * 64;
        // MASK: the warp's 32 keys and 64 queries are looked at one by one (1), all masked (2) or all visible (0)
        auto tile = [&](auto edge_tag, auto mask_tag) {
          constexpr bool EDGE = decltype(edge_tag)::value;
          constexpr int MASK = decltype(mask_tag)::value;
          float pv[64];
          // this key's 64 queries, a bit each: visible; in range
          [[maybe_unused]] uint32_t seen[2] = {0xffffffffu, 0xffffffffu}, in[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if constexpr (MASK == 1) seen[i] = transpose_bits(bits[i], lane);
            if constexpr (EDGE) in[i] = bit_range(q_lo - 32 * i, q_hi - 32 * i);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {          // P, 16 queries at a time
            uint32_t ts[16], pp[3][8];
            if constexpr (MASK != 2) {
              tmem_ld_32x32b_x16(s_addr + c * 16, ts);
              tmem_ld_wait();
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int at = half * 64 + c * 16 + v * 4;
              const float4 l4 = *reinterpret_cast<const float4*>(st + (MASK == 2 ? 256 : 0) + at);
              float4 m4 = l4;
              if constexpr (MASK == 1) m4 = *reinterpret_cast<const float4*>(st + 256 + at);
              const float ls[4] = {l4.x, l4.y, l4.z, l4.w};
              [[maybe_unused]] const float pm[4] = {m4.x, m4.y, m4.z, m4.w};
              float z[4] = {ls[0], ls[1], ls[2], ls[3]};
              if constexpr (MASK != 2) {
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                  const float2 y = fma2(__uint_as_float(ts[4 * v + e]), __uint_as_float(ts[4 * v + e + 1]), p.scale_log2, ls[e], ls[e + 1]);
                  z[e] = fast_exp2(y.x);
                  z[e + 1] = fast_exp2(y.y);
                }
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int i = 4 * v + e;
                float x = z[e];
                if constexpr (MASK == 1) x = seen[c / 2] & (1u << ((c & 1) * 16 + i)) ? x : pm[e];
                if constexpr (EDGE) x = in[c / 2] & (1u << ((c & 1) * 16 + i)) ? x : 0.f;
                pv[c * 16 + i] = x;
              }
#pragma unroll
              for (int e = 0; e < 2; ++e) split3(pv[c * 16 + 4 * v + 2 * e], pv[c * 16 + 4 * v + 2 * e + 1], pp[0][2 * v + e], pp[1][2 * v + e], pp[2][2 * v + e]);
            }
            tmem_st_32x32b_x8(tmem_base + lane_off + P_COL + half * 32 + c * 8, pp[0]);
            tmem_st_32x32b_x8(s_addr + c * 16, pp[1]);
            tmem_st_32x32b_x8(s_addr + c * 16 + 8, pp[2]);
          }
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full);                      // dV runs while dS is made
          seen[0] &= in[0];
          seen[1] &= in[1];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t td[16], dd[3][8];
            if constexpr (MASK != 2) {
              tmem_ld_32x32b_x16(dp_addr + c * 16, td);
              tmem_ld_wait();
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              float4 d4 = make_float4(0.f, 0.f, 0.f, 0.f);
              if constexpr (MASK != 2) d4 = *reinterpret_cast<const float4*>(st + 128 + half * 64 + c * 16 + v * 4);
              const float de[4] = {d4.x, d4.y, d4.z, d4.w};
              float dv[4];
#pragma unroll
              for (int e = 0; e < 4; e += 2) {
                float2 y = make_float2(0.f, 0.f);
                if constexpr (MASK != 2) {
                  const int i = 4 * v + e;
                  y = mul2(pv[c * 16 + i], pv[c * 16 + i + 1], fma2(__uint_as_float(td[i]), __uint_as_float(td[i + 1]), p.scale, de[e], de[e + 1]));
                }
                dv[e] = y.x;
                dv[e + 1] = y.y;
              }
              if constexpr (MASK == 1 || EDGE) {
#pragma unroll
                for (int e = 0; e < 4; ++e) dv[e] = seen[c / 2] & (1u << ((c & 1) * 16 + 4 * v + e)) ? dv[e] : 0.f;      // a masked score is a constant
              }
#pragma unroll
              for (int e = 0; e < 2; ++e) split3(dv[2 * e], dv[2 * e + 1], dd[0][2 * v + e], dd[1][2 * v + e], dd[2][2 * v + e]);
            }
            if (c == 0 && it > 0) drain(t - 1, item, q_blk - 1);   // dK and dQ of the block before have read its dS
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
        using std::integral_constant;
        if constexpr (MASKED) {
          const bool on = __all_sync(0xffffffffu, (bits[0] & bits[1]) == 0xffffffffu), off = __all_sync(0xffffffffu, (bits[0] | bits[1]) == 0u);
          if (edge) tile(std::true_type{}, integral_constant<int, 1>{});
          else if (on) tile(std::false_type{}, integral_constant<int, 0>{});
          else if (off) tile(std::false_type{}, integral_constant<int, 2>{});
          else tile(std::false_type{}, integral_constant<int, 1>{});
        } else {
          if (edge) tile(std::true_type{}, integral_constant<int, 0>{}); else tile(std::false_type{}, integral_constant<int, 0>{});
        }
        tc_fence_before_sync();
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_full);
      }
      drain(t - 1, item, i_begin + iters - 1);                         // (all products of the item have completed)
      // ---- dV / dK: thread r <-> key row r
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(tmem_base + lane_off + (which == 0 ? DV_COL : DK_COL) + half * 32, t);
        tmem_ld_wait();
        if (k_idx < p.Sk) {
          const long* st = which == 0 ? p.dv_strides : p.dk_strides;
          __nv_bfloat16* row = (which == 0 ? p.dv : p.dk) + w.batch * st[0] + w.head * st[1] + k_idx * st[2] + half * 32;
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
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
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
  const long items = (long)key_blocks * A * B;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -2;
  const dim3 grid((unsigned)(items < sms ? items : sms));
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

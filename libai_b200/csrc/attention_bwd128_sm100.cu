// Flash attention backward for head dim 128 (bf16, causal or full, right-padded batches; no bias, no dropout: those stay with
// attn_bwd_kernel in attention_sm100.cu), pipelined.
//
// The general kernel ran its chain Q,dO load → S,dP → softmax → dV,dK,dQ → dQ drain strictly in sequence: its tiles of 128 queries
// leave no shared memory for a second Q/dO stage and no tensor memory beside S, dP, dV and dK (5.9 us per 128 x 128 tile where the
// products take 1.6 us).  Here a CTA owns 128 keys and walks tiles of 64 queries, everything transposed:
//   Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ      [128 keys, 64 queries], TMEM, two buffers: the next tile's are computed under this tile's softmax
//   Pᵀ, dSᵀ                      back into TMEM as bf16 over Sᵀ / dPᵀ: the A operands of the next two, never in shared memory
//   dV += Pᵀ·dO, dK += dSᵀ·Q     [128 keys, 128], TMEM, for the whole CTA
//   dQᵀ = Kᵀ·dSᵀ                 [128, 64 queries], TMEM, in the 64 columns that Pᵀ and dSᵀ leave free between them; dSᵀ is its B operand, the
//                                one tile that also goes through shared memory; drained one tile late into the fp32 accumulator by TMA reductions
// TMEM: 2 x (Sᵀ 64 + dPᵀ 64) + dV 128 + dK 128 = 512 columns.  Shared memory: K, V 64 KB, three stages of Q, dO 96 KB and their
// row statistics, two dSᵀ tiles 32 KB, dQ staging 32 KB.
// Two groups of eight softmax warps, one per buffer: a thread owns one key and 32 queries of every other tile; the row statistics
// (log-sum-exp, δ) arrive per tile with Q and dO.  Four more warps drain dQ.  One thread issues every product.
// What bounds it is shared memory: per tile the products read 176 KB of operands, and loads, dSᵀ and the dQ boxes move 112 KB, 2300
// cycles at 128 bytes of the 2600 that a tile takes.  [1, 8192, 16, 128] causal 1317 -> 743 us, [1, 2048, 32, 128] 224 -> 145 us.  On the way:
// one warp waiting per product group and Sᵀ, dPᵀ behind the whole group before 950; one group of softmax warps 768; dQ added by the drain
// warps themselves (32-bit reductions from registers, no boxes) 890; without the reductions altogether the time is the same.
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

namespace lb {

constexpr int B128_THREADS = 704;                    // TMA warp, MMA warp, 2 x 8 softmax warps, 4 warps that drain dQ
constexpr int B128_KV = 128 * 128 * 2, B128_Q = 64 * 128 * 2, B128_DS = 128 * 64 * 2, B128_BOX = 32 * 128, B128_STAT = 2 * 64 * 4;
constexpr int B128_ST = 3;                            // Q / dO stages: with two a tile's loads waited for the products of the tile before last
constexpr int B128_SMEM = 2 * B128_KV + 2 * B128_ST * B128_Q + 2 * B128_DS + 8 * B128_BOX + B128_ST * B128_STAT + 1024 + 256;
static_assert(B128_SMEM <= 232448, "attention backward, head dim 128: shared memory");

struct Bwd128Params {
  const float* stats;       // [B * A, tiles of 64 queries, 2, 64]: log-sum-exp in the log2 domain, δ · scale; rows behind S are zero
  __nv_bfloat16 *dk, *dv;   // [B, A, S, 128] views
  long g_strides[3];
  int A, S, causal;
  float scale, scale_log2;
  const int* kv_lens;       // optional [B]
  int* err;
};

__global__ void __launch_bounds__(B128_THREADS, 1)
attn_bwd128_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                   const __grid_constant__ CUtensorMap tmap_dq, Bwd128Params p) {
  constexpr uint32_t DV_COL = 256, DK_COL = 384;       // buffer b: Sᵀ [128 b, +64), dPᵀ [128 b + 64, +64); Pᵀ [128 b, +32), dQᵀ [128 b + 32, +64), dSᵀ [128 b + 96, +32)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;                                  // two chunks of 64 columns, 128 rows x 128 bytes each
  uint8_t* sV = sK + B128_KV;
  uint8_t* sQ = sV + B128_KV;                          // B128_ST stages of two chunks, 64 rows x 128 bytes each
  uint8_t* sDO = sQ + B128_ST * B128_Q;
  uint8_t* sDS = sDO + B128_ST * B128_Q;                     // 2 x dSᵀ: 128 key rows x 128 bytes
  uint8_t* sDQ = sDS + 2 * B128_DS;                    // two [32 queries x 32 floats] boxes per warp that drains dQ
  float* sStat = reinterpret_cast<float*>(sDQ + 8 * B128_BOX);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + B128_ST * 128);
  uint64_t* kv_full = bars;          // 1
  uint64_t* q_full = bars + 1;       // 3
  uint64_t* q_empty = bars + 4;      // 3
  uint64_t* s_full = bars + 7;       // 2
  uint64_t* pds_full = bars + 9;     // 2
  uint64_t* dq_full = bars + 11;     // 2
  uint64_t* dq_empty = bars + 13;    // 2
  uint64_t* dp_full = bars + 15;     // 2
  uint64_t* dv_done = bars + 17;     // 2
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 20);

  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int head = blockIdx.y, batch = blockIdx.z, k0 = blockIdx.x * 128;
  const int kv_len = p.kv_lens != nullptr ? max(1, min(p.S, p.kv_lens[batch])) : p.S;
  const int nq = (p.S + 63) / 64;
  const int i_begin = p.causal ? k0 / 64 : 0;
  const int iters = nq - i_begin;                      // >= 1: k0 < S
  const int bh = batch * p.A + head;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_do);
    tma_prefetch_desc(&tmap_dq);
    mbar_init(kv_full, 1);
    for (int i = 0; i < B128_ST; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&pds_full[i], 8);
      mbar_init(&dq_full[i], 1);
      mbar_init(&dq_empty[i], 4);
      mbar_init(&dp_full[i], 1);
      mbar_init(&dv_done[i], 1);
    }
    *stop = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 1) tmem_alloc<512>(tmem_ptr_smem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  chain_next();

  // phases are taken in order, so one that is there needs no look at *stop (30 cycles, up to six times per tile)
  auto ready = [&](uint64_t* bar, uint32_t parity) { return mbar_try_wait(bar, parity) || tc_wait(bar, parity, stop); };
  if (warp_idx == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * B128_KV);
      for (int c = 0; c < 2; ++c) {
        tma_load_4d(sK + c * (128 * 128), &tmap_k, kv_full, c * 64, k0, head, batch);
        tma_load_4d(sV + c * (128 * 128), &tmap_v, kv_full, c * 64, k0, head, batch);
      }
      for (int it = 0; it < iters; ++it) {
        const int st = it % B128_ST, q0 = (i_begin + it) * 64;
        if (!tc_wait(&q_empty[st], ((it / B128_ST) & 1) ^ 1, stop)) break;
        mbar_arrive_expect_tx(&q_full[st], 2 * B128_Q + B128_STAT);
        for (int c = 0; c < 2; ++c) {
          tma_load_4d(sQ + st * B128_Q + c * (64 * 128), &tmap_q, &q_full[st], c * 64, q0, head, batch);
          tma_load_4d(sDO + st * B128_Q + c * (64 * 128), &tmap_do, &q_full[st], c * 64, q0, head, batch);
        }
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_u32(sStat + st * 128)),
                     "l"(p.stats + (static_cast<long>(bh) * nq + i_begin + it) * 128), "r"(B128_STAT), "r"(smem_u32(&q_full[st]))
                     : "memory");
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    constexpr uint32_t idesc_s = make_idesc_bf16(128, 64, false, false);    // K·Qᵀ, V·dOᵀ
    constexpr uint32_t idesc_t = make_idesc_bf16(128, 128, false, true);    // Pᵀ·dO, dSᵀ·Q (A from TMEM)
    constexpr uint32_t idesc_q = make_idesc_bf16(128, 64, true, true);      // Kᵀ·dSᵀ
    const uint64_t dk_s = make_smem_desc_sw128(smem_u32(sK), 0, 1024), dv_s = make_smem_desc_sw128(smem_u32(sV), 0, 1024);
    const uint64_t dk_t = make_smem_desc_sw128(smem_u32(sK), 128 * 128, 1024);
    // A tile's scores overwrite the buffer of the tile before last.  Sᵀ waits for its dQᵀ to be drained and its dV product to have read
    // Pᵀ, under its dK product; dPᵀ waits for that one, under Sᵀ: the tensor pipe stays fed over both waits.
    auto issue_s = [&](int it) {
      const int b = it & 1, st = it % B128_ST;
      if (!ready(&q_full[st], (it / B128_ST) & 1)) return false;
      if (it >= 2 && !(ready(&dq_empty[b], ((it - 2) >> 1) & 1) && ready(&dv_done[b], ((it - 2) >> 1) & 1))) return false;
      tc_fence_after_sync();
      const uint64_t q_s = make_smem_desc_sw128(smem_u32(sQ + st * B128_Q), 0, 1024), do_s = make_smem_desc_sw128(smem_u32(sDO + st * B128_Q), 0, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_f16_ss(tmem_base + b * 128, dk_s + (((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4), q_s + (((kk / 4) * (64 * 128) + (kk % 4) * 32) >> 4),
                    idesc_s, kk > 0 ? 1u : 0u);
      umma_commit(&s_full[b]);
      if (it >= 2) {
        if (!ready(&q_empty[(it - 2) % B128_ST], ((it - 2) / B128_ST) & 1)) return false;
        tc_fence_after_sync();
      }
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_f16_ss(tmem_base + b * 128 + 64, dv_s + (((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4), do_s + (((kk / 4) * (64 * 128) + (kk % 4) * 32) >> 4),
                    idesc_s, kk > 0 ? 1u : 0u);
      umma_commit(&dp_full[b]);
      return true;
    };
    if (elect_one() && ready(kv_full, 0) && issue_s(0)) {
      for (int it = 0; it < iters; ++it) {
        const int b = it & 1, st = it % B128_ST;
        if (it + 1 < iters && !issue_s(it + 1)) break;
        if (!ready(&pds_full[b], (it >> 1) & 1)) break;
        tc_fence_after_sync();
        const uint64_t q_t = make_smem_desc_sw128(smem_u32(sQ + st * B128_Q), 64 * 128, 1024), do_t = make_smem_desc_sw128(smem_u32(sDO + st * B128_Q), 64 * 128, 1024);
        const uint64_t ds_t = make_smem_desc_sw128(smem_u32(sDS + b * B128_DS), 128 * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // dQᵀ first: its drain takes longest
          umma_f16_ss(tmem_base + b * 128 + 32, dk_t + ((kk * 2048) >> 4), ds_t + ((kk * 2048) >> 4), idesc_q, kk > 0 ? 1u : 0u);
        umma_commit(&dq_full[b]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16_ts(tmem_base + DV_COL, tmem_base + b * 128 + kk * 8, do_t + ((kk * 2048) >> 4), idesc_t, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&dv_done[b]);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16_ts(tmem_base + DK_COL, tmem_base + b * 128 + 96 + kk * 8, q_t + ((kk * 2048) >> 4), idesc_t, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&q_empty[st]);          // Q, dO, Pᵀ, dSᵀ of this tile have been read
      }
    }
    __syncwarp();
  } else if (warp_idx >= 18) {
    // dQᵀ of every tile: thread = one of the 128 columns of dQ, 2 x 32 queries -> [32 queries x 32 floats] boxes (128-byte rows, swizzled) -> reduction
    const int quad = warp_idx % 4;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    for (int it = 0; it < iters; ++it) {
      const int b = it & 1;
      const bool fine = tc_wait(&dq_full[b], (it >> 1) & 1, stop);
      __syncwarp();
      tc_fence_after_sync();
      uint32_t t[2][32];
      tmem_ld_32x32b_x32(tmem_base + lane_off + b * 128 + 32, t[0]);
      tmem_ld_32x32b_x32(tmem_base + lane_off + b * 128 + 64, t[1]);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dq_empty[b]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (lane == 0) tma_store_wait_read<1>();       // the reduction before last, of this box, has read it
        __syncwarp();
        uint8_t* box = sDQ + (quad * 2 + h) * B128_BOX;
        const uint32_t base = smem_u32(box) + static_cast<uint32_t>((lane & 3) * 4);
#pragma unroll
        for (int q = 0; q < 32; ++q)
          asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(base + q * 128 + (((lane >> 2) ^ (q & 7)) << 4)), "r"(t[h][q]) : "memory");
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          const int q0 = (i_begin + it) * 64 + h * 32;
          if (fine && q0 < p.S)                        // boxes start inside the accumulator; its edge clips them
            asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(
                             reinterpret_cast<uint64_t>(&tmap_dq)),
                         "r"(quad * 32), "r"(q0), "r"(bh), "r"(smem_u32(box))
                         : "memory");
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait<0>();
    __syncwarp();
  } else {
    // TMEM lanes of this warp; its 32 of the tile's 64 queries; the buffer whose tiles it takes
    const int quad = warp_idx % 4, half = (warp_idx - 2) / 4 % 2, b = (warp_idx - 2) / 8;
    const int r = quad * 32 + lane, k_idx = k0 + r;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    for (int it = b; it < iters; it += 2) {
      const int st = it % B128_ST, q0 = (i_begin + it) * 64;
      const bool edge = (p.causal && q0 < k0 + 127) || q0 + 64 > p.S || k0 + 128 > kv_len;
      // queries [q_lo, q_hi) of this half see key k_idx
      const int q_lo = (k_idx < kv_len ? (p.causal ? k_idx : 0) : p.S) - q0 - half * 32, q_hi = p.S - q0 - half * 32;
      // The tile's statistics: this group sees a stage's phases two apart (tiles it, it + 6), whose parity is the same, so q_full alone
      // may answer for the phase before last.  Behind s_full it cannot: Sᵀ was issued after q_full's phase had come.
      ready(&s_full[b], (it >> 1) & 1);
      ready(&q_full[st], (it / B128_ST) & 1);
      __syncwarp();
      tc_fence_after_sync();
      const float4* lse4 = reinterpret_cast<const float4*>(sStat + st * 128 + half * 32);
      const float4* del4 = reinterpret_cast<const float4*>(sStat + st * 128 + 64 + half * 32);
      uint32_t pk[16];
      uint32_t pv[32];
      tmem_ld_32x32b_x32(tmem_base + lane_off + b * 128 + half * 32, pv);
      tmem_ld_wait();
      auto exps = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const float4 l4 = lse4[v];
          const float ls[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = 4 * v + e;
            float x = fast_exp2(fmaf(__uint_as_float(pv[i]), p.scale_log2, -ls[e]));
            if constexpr (EDGE) x = (i >= q_lo && i < q_hi) ? x : 0.f;
            pv[i] = __float_as_uint(x);
          }
          pk[2 * v] = pack_bf16(__uint_as_float(pv[4 * v]), __uint_as_float(pv[4 * v + 1]));
          pk[2 * v + 1] = pack_bf16(__uint_as_float(pv[4 * v + 2]), __uint_as_float(pv[4 * v + 3]));
        }
      };
      if (edge) exps(std::true_type{}); else exps(std::false_type{});
      tc_fence_before_sync();
      tc_pair_sync(b * 4 + quad);                      // Pᵀ of both halves overwrites the first half's scores
      tc_fence_after_sync();
      tmem_st_32x32b_x16(tmem_base + lane_off + b * 128 + half * 16, pk);
      ready(&dp_full[b], (it >> 1) & 1);
      __syncwarp();
      tc_fence_after_sync();
      auto grads = [&](auto edge_tag) {
        constexpr bool EDGE = decltype(edge_tag)::value;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t td[16];
          tmem_ld_32x32b_x16(tmem_base + lane_off + b * 128 + 64 + half * 32 + c * 16, td);
          tmem_ld_wait();
#pragma unroll
          for (int v = 4 * c; v < 4 * c + 4; ++v) {
            const float4 d4 = del4[v];
            const float de[4] = {d4.x, d4.y, d4.z, d4.w};
            float dv[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int i = 4 * v + e;
              dv[e] = __uint_as_float(pv[i]) * fmaf(__uint_as_float(td[i - 16 * c]), p.scale, -de[e]);
              if constexpr (EDGE) dv[e] = (i >= q_lo && i < q_hi) ? dv[e] : 0.f;
            }
            pk[2 * v] = pack_bf16(dv[0], dv[1]);
            pk[2 * v + 1] = pack_bf16(dv[2], dv[3]);
          }
        }
      };
      if (edge) grads(std::true_type{}); else grads(std::false_type{});
      tc_fence_before_sync();
      tc_pair_sync(b * 4 + quad);                      // dSᵀ of both halves overwrites the second half's dPᵀ
      tc_fence_after_sync();
      tmem_st_32x32b_x16(tmem_base + lane_off + b * 128 + 96 + half * 16, pk);
      uint8_t* drow = sDS + b * B128_DS + r * 128;
#pragma unroll
      for (int v = 0; v < 4; ++v)
        *reinterpret_cast<uint4*>(drow + (((half * 4 + v) ^ (r & 7)) << 4)) = make_uint4(pk[4 * v], pk[4 * v + 1], pk[4 * v + 2], pk[4 * v + 3]);
      tmem_st_wait();
      tc_fence_before_sync();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_full[b]);
    }
    // ---- dV (first group) / dK (second): thread = key row, this half's 64 columns
    tc_wait(&q_empty[(iters - 1) % B128_ST], ((iters - 1) / B128_ST) & 1, stop);
    __syncwarp();
    tc_fence_after_sync();
    __nv_bfloat16* row = (b == 0 ? p.dv : p.dk) + batch * p.g_strides[0] + head * p.g_strides[1] + static_cast<long>(k_idx) * p.g_strides[2] + half * 64;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t t[32];
      tmem_ld_32x32b_x32(tmem_base + lane_off + (b == 0 ? DV_COL : DK_COL) + half * 64 + c * 32, t);
      tmem_ld_wait();
      if (k_idx < p.S) {
#pragma unroll
        for (int i = 0; i < 32; i += 8)
          *reinterpret_cast<uint4*>(row + c * 32 + i) = make_uint4(
              pack_bf16(__uint_as_float(t[i]), __uint_as_float(t[i + 1])), pack_bf16(__uint_as_float(t[i + 2]), __uint_as_float(t[i + 3])),
              pack_bf16(__uint_as_float(t[i + 4]), __uint_as_float(t[i + 5])), pack_bf16(__uint_as_float(t[i + 6]), __uint_as_float(t[i + 7])));
      }
      __syncwarp();                                    // whole warps read tensor memory
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*stop) {                                         // copies in flight land before the shared memory goes away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) { *const_cast<volatile int*>(p.err) = 1; __threadfence_system(); }
    __syncthreads();
  }
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc<512>(tmem_base);
  }
}

// Row statistics per tile of 64 queries: log-sum-exp · log2 e, then δ · scale with δ = Σ_d dO · O; zeros behind row S.  16 lanes per row;
// clears the fp32 dQ accumulator as well.
__global__ void __launch_bounds__(256)
attn_bwd128_stats_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ o, const float* __restrict__ lse,
                         float* __restrict__ stats, int A, int S, long bh_count, long sb, long sa, long ss, float scale,
                         float4* __restrict__ zero_fill, long zero_n4) {
  chain_wait(dout, o, lse, zero_fill);
  chain_next();
  const long gid = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x, threads = static_cast<long>(gridDim.x) * blockDim.x;
  for (long z = gid; z < zero_n4; z += threads) zero_fill[z] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int nq = (S + 63) / 64, sub = threadIdx.x % 16;
  const long rows = bh_count * nq * 64;                // rows in the order (batch, query, head): memory order of the [b, s, a, d] tensors
  const long warp_first = (gid - threadIdx.x % 32) / 16;
  for (long base = 0; warp_first + base < rows; base += threads / 16) {
    const long row = gid / 16 + base;
    const int a = static_cast<int>(row % A), s = static_cast<int>((row / A) % (nq * 64));
    const long b = row / (static_cast<long>(A) * nq * 64);
    float acc = 0.f;
    const bool in = row < rows && s < S;
    if (in) {
      const long off = b * sb + a * sa + s * ss + sub * 8;
      const uint4 x = *reinterpret_cast<const uint4*>(dout + off), y = *reinterpret_cast<const uint4*>(o + off);
      const uint32_t *xw = &x.x, *yw = &y.x;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 u = unpack_bf16(xw[e]), v = unpack_bf16(yw[e]);
        acc += u.x * v.x + u.y * v.y;
      }
    }
#pragma unroll
    for (int m = 8; m >= 1; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (sub == 0 && row < rows) {
      float* dst = stats + ((b * A + a) * nq + s / 64) * 128 + s % 64;
      dst[0] = in ? lse[(b * A + a) * S + s] * 1.4426950408889634f : 0.f;
      dst[64] = in ? acc * scale : 0.f;
    }
  }
}

}  // namespace lb

extern "C" int lb_attn_dq_convert(const float* acc, void* dq, int B, int A, int S, int D, const long* st, cudaStream_t s);

// dq, dk, dv: [B, A, S, 128] views with g_strides; dq_acc: fp32 scratch [B, A, S, 128]; dout and o share do_strides; stats: scratch of
// B * A * ceil(S / 64) * 128 floats.  Returns 0, a cudaError_t or a negative code.
extern "C" int lb_attn_bwd128(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse, void* dq, void* dk,
                              void* dv, float* stats, float* dq_acc, int B, int A, int S, const long* qs, const long* ks, const long* vs, const long* dos,
                              const long* g_strides, int causal, float scale, const int* kv_lens, int* err, cudaStream_t s) {
  for (int i = 0; i < 3; ++i)
    if ((qs[i] % 8) || (ks[i] % 8) || (vs[i] % 8) || (dos[i] % 8)) return -3;
  CUtensorMap tq, tk, tv, tdo, tdq;
  auto map = [&](CUtensorMap* m, const void* ptr, const long* st, int rows) {
    uint64_t dims[4] = {128, (uint64_t)S, (uint64_t)A, (uint64_t)B};
    uint64_t strides[4] = {2, (uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
    uint32_t box[4] = {64, (uint32_t)rows, 1, 1};
    return lb_host::make_tmap_bf16(m, ptr, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  if (!map(&tq, q, qs, 64) || !map(&tk, k, ks, 128) || !map(&tv, v, vs, 128) || !map(&tdo, dout, dos, 64)) return -2;
  {
    uint64_t dims[3] = {128, (uint64_t)S, (uint64_t)B * A};
    uint64_t strides[3] = {4, 512, (uint64_t)S * 512};
    uint32_t box[3] = {32, 32, 1};
    if (!lb_host::make_tmap_typed(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, dq_acc, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -2;
  }
  const long rows = (long)B * A * ((S + 63) / 64) * 64;
  long blocks = (rows * 16 + 255) / 256;
  if (blocks > 148L * 16) blocks = 148L * 16;
  lb_host::launch_chained(lb::attn_bwd128_stats_kernel, dim3((unsigned)blocks), dim3(256), 0, s, 0, (const __nv_bfloat16*)dout, (const __nv_bfloat16*)o, lse, stats, A, S, (long)B * A, dos[0],
                                                                dos[1], dos[2], scale, (float4*)dq_acc, (long)B * A * S * 32);
  lb::Bwd128Params p{};
  p.stats = stats;
  p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  for (int i = 0; i < 3; ++i) p.g_strides[i] = g_strides[i];
  p.A = A; p.S = S; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.kv_lens = kv_lens;
  p.err = err;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(lb::attn_bwd128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lb::B128_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  lb::attn_bwd128_kernel<<<dim3((S + 127) / 128, A, B), lb::B128_THREADS, lb::B128_SMEM, s>>>(tq, tk, tv, tdo, tdq, p);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? (int)e : lb_attn_dq_convert(dq_acc, dq, B, A, S, 128, g_strides, s);
}

// Flash attention forward (bf16, head dim 64 or 128, causal or full, right-padded batches; no bias, no dropout: those stay with
// attn_fwd_v2_kernel in attention_sm100.cu), two query tiles per CTA and CTAs that take the next work item themselves.
//
// attn_fwd_v2_kernel gives a tile to eight softmax warps, two threads per row that exchange their maxima, reads every score twice from tensor
// memory, and its chain Q·Kᵀ -> max -> exchange -> exponentials -> P·V takes 2840 cycles per 128 x 128 scores (3000 at head dim 64 with two
// CTAs per SM), where the products take 1024 (512) and the exponentials 1024.  Here a CTA works on two tiles of 128 queries of one head in
// units of 64 keys, a warpgroup per tile, two score buffers per tile:
//   warp 0      TMA: Q of both tiles, K / V tiles of 128 keys through one ring; asks for the next work item (cluster launch control) once
//               the loads of this one are issued
//   warps 1, 2  issue the products of tile 0 / 1: S = Q·Kᵀ of the unit after next goes into the buffer whose P·V has just been issued, also
//               over the end of a work item where nothing has to be waited for
//   warps 4-7, 8-11  softmax of tile 0 / 1: a thread owns a row and holds a unit's 64 scores in registers (one read of tensor memory, no
//               exchange), P goes back over the scores as bf16; the reference maximum moves when it grows by more than 2^8
// TMEM: two tiles x two buffers of 64 columns (P over the first 32), O_0, O_1.  The products of a tile are issued by one thread in the order P·V,
// next Q·Kᵀ into the same buffer, so scores are not overwritten before P has been read.  The last unit is as wide as its keys need
// (multiples of 16).  Work items are pairs of query tiles, heaviest first within groups of heads whose keys and values stay in L2.
//
// [1, 8192, 16, 128] causal 334 -> 236 us, [1, 2048, 32, 128] 65 -> 42, [8, 1024, 16, 64] 55.6 -> 46.5, [64, 197, 16, 64] full 56.4 -> 43.4,
// [1, 8192, 16, 64] 295 -> 204.  What bounds it are the softmax warps, not the products (without those 6 to 14 % less): a unit takes its warp 1500 to
// 1700 cycles, 850 to 1000 of them exponentials (512 of a warp alone), the rest waiting for the scores' barrier (120), reading them (65), the
// maximum (340), storing P and handing it over (190), and two warps per scheduler do not fill each other's gaps.  Measured and not kept:
// blocks of 128 keys per thread (P over S keeps the next Q·Kᵀ waiting 1400 cycles per block; 246 and 187 us at 8192), two threads per row (305; 190 at
// head dim 64, slower at short lengths), two CTAs per SM at head dim 64 (217), the next unit's scores fetched under the exponentials (280; 260).
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

#include <atomic>

namespace lb {

constexpr int FA_THREADS = 384;                               // TMA warp, two MMA warps, one without work, 2 x 4 softmax warps

template <int D>
struct FaCfg {
  static constexpr int TILE = 128 * D * 2;                    // 128 rows of Q, K or V
  static constexpr int CHUNKS = D / 64;                       // of 64 columns: 128 rows x 128 bytes
  static constexpr int QB = D == 64 ? 2 : 1;                  // Q buffers: head dim 128 has room for one (its Q arrives under the last P·V and the epilogue)
  static constexpr int RING = D == 64 ? 6 : 4;                // K, V tiles
  static constexpr int SMEM = (2 * QB + RING) * TILE + 1024 + 512;
  static constexpr uint32_t O_COL = 256;                      // scores of tile t at 128 t (64 per unit), O_t at 256 + D t
};
static_assert(FaCfg<64>::SMEM <= 232448 && FaCfg<128>::SMEM <= 232448, "attention forward: shared memory");

struct FaParams {
  __nv_bfloat16* o;       // [B, S, A, D]
  float* lse;             // [B, A, S]
  int A, S, BA, causal;
  int rows, parts, group; // queries per work item (256, or 128: one tile), work items per head, heads per group
  float scale_log2;
  const int* kv_lens;     // optional [B]
  int* err;
};

struct FaItem {
  int q0, bh, head, batch, kv_len, n0, n1;                    // units of 64 keys that the two tiles look at (0: no such tile)
};
LB_DEVICE int fa_units(const FaItem& w, int t) { return t ? w.n1 : w.n0; }
LB_DEVICE int fa_blocks(const FaItem& w) { return (max(w.n0, w.n1) + 1) / 2; }   // K / V tiles of 128 keys
LB_DEVICE FaItem fa_item(const FaParams& p, int idx) {
  FaItem w;
  const int grp = idx / (p.group * p.parts), rem = idx - grp * p.group * p.parts;
  const int heads = min(p.group, p.BA - grp * p.group);
  const int part = p.parts - 1 - rem / heads;
  w.bh = grp * p.group + rem % heads;
  w.batch = w.bh / p.A;
  w.head = w.bh - w.batch * p.A;
  w.q0 = part * p.rows;
  w.kv_len = p.kv_lens != nullptr ? max(1, min(p.S, p.kv_lens[w.batch])) : p.S;
  w.n0 = ((p.causal ? min(w.kv_len, w.q0 + 128) : w.kv_len) + 63) / 64;
  w.n1 = p.rows == 128 || w.q0 + 128 >= p.S ? 0 : ((p.causal ? min(w.kv_len, w.q0 + 256) : w.kv_len) + 63) / 64;
  return w;
}

// two fp32 multiply-adds / additions per instruction
LB_DEVICE void fma2(float& x, float& y, float a, float b, float m, float c) {
  asm("{\n\t.reg .b64 v, s, t;\n\t"
      "mov.b64 v, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\tmov.b64 t, {%5, %5};\n\t"
      "fma.rn.ftz.f32x2 v, v, s, t;\n\t"
      "mov.b64 {%0, %1}, v;\n\t}\n"
      : "=f"(x), "=f"(y)
      : "f"(a), "f"(b), "f"(m), "f"(c));
}
LB_DEVICE void add2(float& x, float& y, float a, float b) {
  asm("{\n\t.reg .b64 v, s;\n\t"
      "mov.b64 v, {%0, %1};\n\tmov.b64 s, {%2, %3};\n\t"
      "add.rn.ftz.f32x2 v, v, s;\n\t"
      "mov.b64 {%0, %1}, v;\n\t}\n"
      : "+f"(x), "+f"(y)
      : "f"(a), "f"(b));
}
LB_DEVICE float max3(float a, float b, float c) {
  float d;
  asm("max.ftz.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// asks the hardware for a block that has not started yet; the 16-byte answer completes on `bar`
LB_DEVICE void clc_try_cancel(void* answer, uint64_t* bar) {
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n" ::"r"(smem_u32(answer)), "r"(smem_u32(bar))
               : "memory");
}
// its blockIdx.x, or -1
LB_DEVICE int clc_answer(const void* answer) {
  int x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%1];\n\t"
      "mov.b32 %0, -1;\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, _, _, _}, r;\n\t}\n"
      : "=r"(x)
      : "r"(smem_u32(answer))
      : "memory");
  fence_proxy_async();                                        // read before the next answer may be written
  return x;
}

template <int D>
__global__ void __launch_bounds__(FA_THREADS, 1)
attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                     const FaParams p) {
  using Cfg = FaCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                         // [buffer][tile]
  uint8_t* sKV = sQ + 2 * Cfg::QB * Cfg::TILE;
  uint8_t* answers = sKV + Cfg::RING * Cfg::TILE;             // 2 x 16 bytes
  uint64_t* bars = reinterpret_cast<uint64_t*>(answers + 32);
  uint64_t* q_full = bars;                                    // [buffer * 2 + tile]
  uint64_t* q_empty = bars + 4;
  uint64_t* kv_full = bars + 8;                               // [RING]
  uint64_t* kv_empty = bars + 14;
  uint64_t* s_full = bars + 20;                               // [tile * 2 + buffer]
  uint64_t* p_full = bars + 24;
  uint64_t* o_full = bars + 28;                               // P·V of the unit in this buffer
  uint64_t* next_full = bars + 32;                            // [2]
  uint64_t* next_empty = bars + 34;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 36);
  volatile int* stop = reinterpret_cast<volatile int*>(bars + 37);

  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1);
    }
    for (int i = 0; i < Cfg::RING; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 2);                             // one MMA thread per tile
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&next_full[i], 1);
      mbar_init(&next_empty[i], 11);                          // TMA thread, two MMA threads, eight softmax warps
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
  chain_wait();
  chain_next();
  auto ready = [&](uint64_t* bar, uint32_t parity) { return mbar_try_wait(bar, parity) || tc_wait(bar, parity, stop); };

  if (warp_idx < 4) {
    if (warp_idx == 0 && elect_one()) {
      uint32_t kv = 0;                                        // K and V tiles loaded so far
      uint32_t qn[2] = {0, 0};                                // Q tiles loaded so far, by tile
      int idx = blockIdx.x;
      bool fine = true;
      for (uint32_t it = 0; fine && idx >= 0; ++it) {
        const FaItem w = fa_item(p, idx);
        auto load_q = [&](int t) {
          if (fa_units(w, t) == 0) return true;
          const uint32_t buf = qn[t] % Cfg::QB * 2 + t;
          if (!ready(&q_empty[buf], ((qn[t] / Cfg::QB) & 1) ^ 1)) return false;
          mbar_arrive_expect_tx(&q_full[buf], Cfg::TILE);
          for (int c = 0; c < Cfg::CHUNKS; ++c)
            tma_load_4d(sQ + buf * Cfg::TILE + c * (128 * 128), &tmap_q, &q_full[buf], c * 64, w.q0 + t * 128, w.head, w.batch);
          ++qn[t];
          return true;
        };
        auto load_kv = [&](const CUtensorMap* map, int j) {
          const uint32_t st = kv % Cfg::RING;
          if (!ready(&kv_empty[st], ((kv / Cfg::RING) & 1) ^ 1)) return false;
          mbar_arrive_expect_tx(&kv_full[st], Cfg::TILE);
          for (int c = 0; c < Cfg::CHUNKS; ++c)
            tma_load_4d(sKV + st * Cfg::TILE + c * (128 * 128), map, &kv_full[st], c * 64, j * 128, w.head, w.batch);
          ++kv;
          return true;
        };
        fine = load_q(0) && load_kv(&tmap_k, 0) && load_q(1) && load_kv(&tmap_v, 0);
        const int n = fa_blocks(w);
        for (int j = 1; fine && j < n; ++j) fine = load_kv(&tmap_k, j) && load_kv(&tmap_v, j);
        if (!fine) break;
        const uint32_t s = it & 1;
        if (!ready(&next_empty[s], ((it >> 1) & 1) ^ 1)) break;
        mbar_arrive_expect_tx(&next_full[s], 16);
        clc_try_cancel(answers + s * 16, &next_full[s]);
        if (!ready(&next_full[s], (it >> 1) & 1)) break;
        idx = clc_answer(answers + s * 16);
        mbar_arrive(&next_empty[s]);
      }
    } else if ((warp_idx == 1 || warp_idx == 2) && elect_one()) {
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, D, false, true);
      const int t = warp_idx - 1;
      const uint32_t s_col = tmem_base + t * 128, o_col = tmem_base + Cfg::O_COL + t * D;
      uint32_t qn = 0, sn = 0, pn = 0;                        // Q tiles; units whose Q·Kᵀ / P·V has been issued
      auto width = [](int kv_len, int u) { return min(64, (kv_len - u * 64 + 15) & ~15); };   // keys of unit u that the products take
      // `kv`: K and V tiles of the work items before this one
      auto qk_ready = [&](uint32_t kv, int u) {
        const uint32_t at = kv + (u & ~1);
        return (u > 0 || mbar_try_wait(&q_full[qn % Cfg::QB * 2 + t], (qn / Cfg::QB) & 1)) && mbar_try_wait(&kv_full[at % Cfg::RING], (at / Cfg::RING) & 1);
      };
      auto issue_qk = [&](uint32_t kv, int kv_len, int u, int n) {
        const uint32_t at = kv + (u & ~1), st = at % Cfg::RING, buf = qn % Cfg::QB * 2 + t;
        if (u == 0 && !ready(&q_full[buf], (qn / Cfg::QB) & 1)) return false;
        if (!ready(&kv_full[st], (at / Cfg::RING) & 1)) return false;
        tc_fence_after_sync();
        const uint32_t idesc = make_idesc_bf16(128, width(kv_len, u), false, false);
        const uint64_t q = make_smem_desc_sw128(smem_u32(sQ + buf * Cfg::TILE), 0, 1024),
                       k = make_smem_desc_sw128(smem_u32(sKV + st * Cfg::TILE + (u & 1) * (64 * 128)), 0, 1024);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = ((kk / 4) * (128 * 128) + (kk % 4) * 32) >> 4;
          umma_f16_ss(s_col + (sn & 1) * 64, q + off, k + off, idesc, kk > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[t * 2 + (sn & 1)]);
        ++sn;
        if (u + 1 == n) {
          umma_commit(&q_empty[buf]);
          ++qn;
        }
        if ((u & 1) || u + 1 == n) umma_commit(&kv_empty[st]);
        return true;
      };
      auto issue_pv = [&](uint32_t kv, int kv_len, int u, int n) {
        const uint32_t at = kv + (u & ~1) + 1, st = at % Cfg::RING, steps = width(kv_len, u) / 16;
        if (!ready(&kv_full[st], (at / Cfg::RING) & 1) || !ready(&p_full[t * 2 + (pn & 1)], (pn >> 1) & 1)) return false;
        tc_fence_after_sync();
        const uint64_t v = make_smem_desc_sw128(smem_u32(sKV + st * Cfg::TILE + (u & 1) * (64 * 128)), 128 * 128, 1024);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          if (kk < steps) umma_f16_ts(o_col, s_col + (pn & 1) * 64 + kk * 8, v + ((kk * 2048) >> 4), idesc_pv, (u > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&o_full[t * 2 + (pn & 1)]);
        ++pn;
        if ((u & 1) || u + 1 == n) umma_commit(&kv_empty[st]);
        return true;
      };
      bool fine = true;
      FaItem w = fa_item(p, blockIdx.x);
      uint32_t kv = 0;
      int pre = 0;                                            // units of this work item whose scores were issued with the item before
      for (uint32_t it = 0; fine; ++it) {
        const int n = fa_units(w, t), blocks = fa_blocks(w), kv_len = w.kv_len;
        bool known = false, more = false;                     // is the next work item known; is there one
        int pre_next = 0;
        auto fetch = [&]() {
          const int idx = clc_answer(answers + (it & 1) * 16);
          mbar_arrive(&next_empty[it & 1]);
          known = true;
          more = idx >= 0;
          if (more) w = fa_item(p, idx);
        };
        for (int u = pre; fine && u < min(2, n); ++u) fine = issue_qk(kv, kv_len, u, n);
        for (int u = 0; fine && u < n; ++u) {
          fine = issue_pv(kv, kv_len, u, n);
          if (!fine) break;
          if (u + 2 < n) {
            fine = issue_qk(kv, kv_len, u + 2, n);
          } else {                                            // a buffer is free: scores of the next work item, if they need no wait
            if (!known && mbar_try_wait(&next_full[it & 1], (it >> 1) & 1)) fetch();
            if (more && pre_next < fa_units(w, t) && qk_ready(kv + 2 * blocks, pre_next)) {
              fine = issue_qk(kv + 2 * blocks, w.kv_len, pre_next, fa_units(w, t));
              ++pre_next;
            }
          }
        }
        for (int j = (n + 1) / 2 * 2; fine && j < 2 * blocks; ++j) {   // keys and values of the other tile alone
          const uint32_t at = kv + j, st = at % Cfg::RING;
          fine = ready(&kv_full[st], (at / Cfg::RING) & 1);
          if (fine) mbar_arrive(&kv_empty[st]);
        }
        if (fine && !known) {
          fine = ready(&next_full[it & 1], (it >> 1) & 1);
          if (fine) fetch();
        }
        if (!more) break;
        kv += 2 * blocks;
        pre = pre_next;
      }
    }
    __syncwarp();
  } else {
    const int t = (warp_idx - 4) / 4, quad = warp_idx % 4;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_tile = tmem_base + lane_off + t * 128, o_addr = tmem_base + lane_off + Cfg::O_COL + t * D;
    uint32_t sn = 0;                                          // units so far
    int idx = blockIdx.x;
    for (uint32_t it = 0; idx >= 0; ++it) {
      const FaItem w = fa_item(p, idx);
      const int q_warp = w.q0 + t * 128 + quad * 32, q_idx = q_warp + lane, n = fa_units(w, t);
      // keys [0, key_lim) are visible to this row, [0, lim_lo) to all rows of this warp
      const int key_lim = p.causal ? min(w.kv_len, q_idx + 1) : w.kv_len, lim_lo = p.causal ? min(w.kv_len, q_warp + 1) : w.kv_len;
      float m_run = -INFINITY, l_run = 0.f;
      // The first reference is the maximum of 128 keys: the largest probability is 1 and not rounded (with that of 64, results of 100 to 200 keys
      // are 2 to 4 % further off; 1.7 us of [64, 197, 16, 64]).
      if (n > 1) {
        uint32_t x[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t b = (sn + c / 2) & 1;
          if (c % 2 == 0) {
            ready(&s_full[t * 2 + b], ((sn + c / 2) >> 1) & 1);
            __syncwarp();
            tc_fence_after_sync();
          }
          tmem_ld_32x32b_x32(s_tile + b * 64 + c % 2 * 32, x[c]);
        }
        tmem_ld_wait();
        float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (lim_lo >= 128) {
#pragma unroll
          for (int i = 0; i < 128; i += 2) top[(i >> 1) & 3] = max3(top[(i >> 1) & 3], __uint_as_float(x[i / 32][i % 32]), __uint_as_float(x[i / 32][i % 32 + 1]));
        } else {
#pragma unroll
          for (int i = 0; i < 128; ++i) top[i & 3] = fmaxf(top[i & 3], i < key_lim ? __uint_as_float(x[i / 32][i % 32]) : -INFINITY);
        }
        m_run = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * p.scale_log2;
      }
      bool fine = true;
      for (int u = 0; u < n; ++u, ++sn) {
        fine = ready(&s_full[t * 2 + (sn & 1)], (sn >> 1) & 1);
        __syncwarp();
        if (__any_sync(0xffffffffu, !fine)) break;
        tc_fence_after_sync();
        const uint32_t s_addr = s_tile + (sn & 1) * 64;
        uint32_t s[2][32];
        tmem_ld_32x32b_x32(s_addr, s[0]);
        tmem_ld_32x32b_x32(s_addr + 32, s[1]);
        tmem_ld_wait();
        if (u * 64 + 64 > lim_lo) {
#pragma unroll
          for (int i = 0; i < 64; ++i) s[i / 32][i % 32] = u * 64 + i < key_lim ? s[i / 32][i % 32] : __float_as_uint(-INFINITY);
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 64; i += 2) mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], __uint_as_float(s[i / 32][i % 32]), __uint_as_float(s[i / 32][i % 32 + 1]));
        const float m_cand = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
        const bool bump = (m_cand - m_run > 8.0f) || (m_run == -INFINITY && m_cand != -INFINITY);
        float alpha = 1.0f;
        if (bump) {
          alpha = fast_exp2(m_run - m_cand);                  // 0 on the first unit
          m_run = m_cand;
        }
        if (__any_sync(0xffffffffu, bump && u > 0)) {
          fine = ready(&o_full[t * 2 + ((sn - 1) & 1)], ((sn - 1) >> 1) & 1);             // P·V of the unit before is done
          __syncwarp();
          if (__any_sync(0xffffffffu, !fine)) break;
          tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(o_addr + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x32b_x16(o_addr + c * 16, o);
          }
        }
        const float neg_m = (m_run == -INFINITY) ? 0.f : -m_run;
        float sum[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        uint32_t packed[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          float x, y;
          fma2(x, y, __uint_as_float(s[i / 32][i % 32]), __uint_as_float(s[i / 32][i % 32 + 1]), p.scale_log2, neg_m);
          x = fast_exp2(x);                                   // (masked: 2^-inf = 0)
          y = fast_exp2(y);
          add2(sum[(i >> 1) & 1][0], sum[(i >> 1) & 1][1], x, y);
          packed[i / 2] = pack_bf16(x, y);
        }
        tmem_st_32x32b_x32(s_addr, packed);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t * 2 + (sn & 1)]);
        l_run = l_run * alpha + ((sum[0][0] + sum[0][1]) + (sum[1][0] + sum[1][1]));
      }
      // the next work item's index, while the last P·V runs
      const uint32_t slot = it & 1;
      fine = ready(&next_full[slot], (it >> 1) & 1) && fine;
      __syncwarp();
      if (__any_sync(0xffffffffu, !fine)) break;
      idx = clc_answer(answers + slot * 16);
      __syncwarp();
      if (lane == 0) mbar_arrive(&next_empty[slot]);
      if (n > 0) {
        fine = ready(&o_full[t * 2 + ((sn - 1) & 1)], ((sn - 1) >> 1) & 1);
        __syncwarp();
        tc_fence_after_sync();
        const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
        __nv_bfloat16* orow = p.o + ((static_cast<size_t>(w.batch) * p.S + q_idx) * p.A + w.head) * D;
        const bool store = __all_sync(0xffffffffu, fine) && q_idx < p.S;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          __syncwarp();                                       // whole warps read tensor memory: the stores below are per lane
          tmem_ld_32x32b_x32(o_addr + c * 32, o);
          tmem_ld_wait();
          if (store) {
#pragma unroll
            for (int i = 0; i < 32; i += 16) {
              uint32_t b[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) b[e] = pack_bf16(__uint_as_float(o[i + 2 * e]) * inv, __uint_as_float(o[i + 2 * e + 1]) * inv);
              asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(orow + c * 32 + i), "r"(b[0]), "r"(b[1]), "r"(b[2]),
                           "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7])
                           : "memory");
            }
          }
        }
        if (store)
          p.lse[static_cast<size_t>(w.bh) * p.S + q_idx] = (m_run == -INFINITY) ? -INFINITY : (m_run + log2f(l_run)) * 0.6931471805599453f;
        tc_fence_before_sync();
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*stop) {                                                // copies in flight land before the shared memory goes away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) { *const_cast<volatile int*>(p.err) = 1; __threadfence_system(); }
    __syncthreads();
  }
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc<512>(tmem_base);
  }
}

}  // namespace lb

namespace {
template <int D>
int launch_fwd_pair(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const lb::FaParams& p, cudaStream_t s) {
  auto kern = lb::attn_fwd_pair_kernel<D>;
  static std::atomic<unsigned long long> done{0};             // the limit on shared memory is per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (!(done.load(std::memory_order_relaxed) & bit)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lb::FaCfg<D>::SMEM);
    if (e != cudaSuccess) return (int)e;
    done.fetch_or(bit, std::memory_order_relaxed);
  }
  return (int)lb_host::launch_chained(kern, dim3((unsigned)(p.parts * p.BA)), dim3(lb::FA_THREADS), lb::FaCfg<D>::SMEM, s, 0, tq, tk, tv, p);
}
}  // namespace

// Is the kernel the faster one?  Not where a head has a single full tile at head dim 64 (two CTAs of attn_fwd_v2_kernel per SM work on two
// heads, here one tile of two would idle: [64, 128, 16, 64] 22.1 against 27.1 us; up to 64 queries, one unit, 37.2 against 35.6), and not at head
// dim 128 where every tile has an SM of its own, the chain of one tile counts and that one has two threads per row: [1, 1024, 8, 128] 14.5
// against 16.3, [1, 384, 8, 128] 8.4 against 9.2; up to 192 queries 6.7 against 6.4.
extern "C" int lb_attn_fwd_pair_rule(int B, int A, int S, int D) {
  if (B > 65535 || A > 65535) return 0;
  if (D == 64) return S <= 64 || S > 128;
  return S <= 192 || (long)B * A * ((S + 127) / 128) > 148;
}

// o [B, S, A, D] (32-byte aligned), lse [B, A, S].  Returns 0, a cudaError_t or a negative code.
extern "C" int lb_attn_fwd_pair(const void* q, const void* k, const void* v, void* o, float* lse, int B, int A, int S, int D, const long* qs,
                                const long* ks, const long* vs, int causal, float scale, const int* kv_lens, int* err, cudaStream_t s) {
  if ((D != 64 && D != 128) || B <= 0 || A <= 0 || S <= 0 || B > 65535 || A > 65535) return -1;
  for (int i = 0; i < 3; ++i)
    if ((qs[i] % 8) || (ks[i] % 8) || (vs[i] % 8)) return -3;
  if (reinterpret_cast<uintptr_t>(o) & 31) return -3;
  lb::FaParams p{};
  p.o = (__nv_bfloat16*)o;
  p.lse = lse;
  const long heads = (long)B * A;
  if (heads * ((S + 127) / 128) > 0x7fffffffL) return -1;
  p.A = A; p.S = S; p.BA = (int)heads; p.causal = causal;
  // one tile per CTA where every tile gets an SM of its own
  p.rows = (long)((S + 127) / 128) * p.BA <= 148 ? 128 : 256;
  p.parts = (S + p.rows - 1) / p.rows;
  // 32 MB of keys and values at a time: the heads in flight share L2 with Q and O
  const long head_bytes = (long)S * D * 4;
  long group = (32L << 20) / head_bytes;
  p.group = (int)(group < 1 ? 1 : (group > p.BA ? p.BA : group));
  p.scale_log2 = scale * 1.4426950408889634f;
  p.kv_lens = kv_lens;
  p.err = err;
  CUtensorMap tq, tk, tv;
  auto map = [&](CUtensorMap* m, const void* ptr, const long* st) {
    uint64_t dims[4] = {(uint64_t)D, (uint64_t)S, (uint64_t)A, (uint64_t)B};
    uint64_t strides[4] = {2, (uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
    uint32_t box[4] = {64, 128, 1, 1};
    return lb_host::make_tmap_bf16(m, ptr, 4, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  if (!map(&tq, q, qs) || !map(&tk, k, ks) || !map(&tv, v, vs)) return -2;
  return D == 64 ? launch_fwd_pair<64>(tq, tk, tv, p, s) : launch_fwd_pair<128>(tq, tk, tv, p, s);
}

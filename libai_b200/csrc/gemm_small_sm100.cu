// y[M, N] = x[M, K] · w[N, K]ᵀ (+ bias, activation or residual) for few rows of x: the linear layers of a generation step or of a
// short prompt.  Where it is the better kernel: lb_gemm_small_rule below.
//
// Bounded by reading w once, so the tensor core's roles are swapped against gemm_sm100.cu: 128 rows of w are the M side of the MMA
// (they fill it whatever M is) and NT = 16, 32, 64 or 128 rows of x the N side (zero-filled by TMA behind M).  The K range of a tile is split over
// the CTAs of a cluster (1, 2, 4 or 8), each streaming its own part of w, so that even a [1024, 1024] weight is read by 64 SMs; the
// partial sums meet in distributed shared memory in a fixed order (no atomics, no workspace, the same bits in every run), every CTA
// finishing its share of the columns.  Two CTAs per SM: one streams while the other reduces and stores.  Measured, 4 rows:
// [1024, 4096] 19.8 -> 6.7 us, [3072, 1024] 8.8 -> 5.6 us, [4096, 11008] 49.5 -> 19 us, [12288, 4096] 34 -> 19.8 us (5.1 TB/s of w).
// Every wait on an mbarrier is bounded (attention_tc.cuh).
#include "attention_tc.cuh"

#include <mutex>

namespace lb {

constexpr int GS_THREADS = 192;                   // TMA warp, MMA warp, 4 epilogue warps
constexpr int GS_W_BYTES = 128 * 64 * 2;

template <int NT>
struct GsCfg {
  static constexpr int X_BYTES = NT * 64 * 2;
  static constexpr int STAGE = GS_W_BYTES + X_BYTES;
  static constexpr int PART_BYTES = NT * 128 * 4; // partial sums [NT][128], over the pipeline's memory once it has run dry
  static constexpr uint32_t TMEM = NT < 32 ? 32 : NT;
  static_assert(PART_BYTES <= 2 * STAGE, "partial sums fit the pipeline");
};
constexpr int GS_SMEM = 104000;                   // of pipeline: two CTAs per SM (one with twice the stages leaves no room for clusters of 8 in some GPCs)
constexpr int GS_NORM_BLOCKS = 11;                // k-blocks per CTA with a norm in front: their rows of x beside four stages of w (five up to ten k-blocks)
// K-blocks of w that a CTA sends to L2 ahead of chain_wait(): memory stands still while the small kernel before (a norm, a rotation) ends.  128 KB per CTA are what
// comes in 3 us.  Llama block, one token of 4 sequences on 2046: 151.5 -> 147.5 us (16 k-blocks 148.4); GPT-2 block of 8 sequences on 511: 38.1 -> 37.2.  The same for the first keys
// and values of the decode attention gave nothing.  Not for small matrices, which are in L2 more often than not: [200, 384] x [384, 384] out of L2 4.56 us, 4.91 with it.
constexpr int GS_AHEAD = 8;
constexpr long GS_AHEAD_BYTES = 4 << 20;
constexpr int GS_MAX_STAGES = GS_SMEM / GsCfg<16>::STAGE, GS_TAIL = 1024 + 512;   // alignment, barriers, statistics

struct GemmSmallParams {
  int M, N, K, kb_per_cta, stages, ahead;
  const __nv_bfloat16* bias;      // [N] or nullptr
  const __nv_bfloat16* residual;  // [M, ldo] or nullptr
  __nv_bfloat16 *out, *pre_out;   // [M, ldo]; pre_out (optional): before the activation
  int ldo, act;
  int* err;
};
// with a norm in front: rows of x as they are, its weight and bias (or nullptr)
struct alignas(64) GemmSmallNormParams : GemmSmallParams {
  const __nv_bfloat16 *x, *gamma, *beta;
  int ldx, rms;
  float eps;
};
template <bool NORM> using GemmSmallArgs = std::conditional_t<NORM, GemmSmallNormParams, GemmSmallParams>;
// (two tensor maps and these: what a launch costs the host depends on the bytes, see GemmReduce; 376 for both kinds took 3.7 us, 328 and 384 take 3.5)
static_assert((sizeof(GemmSmallParams) + 7) % 64 < 16 && (sizeof(GemmSmallNormParams) + 7) % 64 < 16, "bytes of the arguments");

// count, mean and sum of squared deviations of two sets of numbers together
LB_DEVICE void merge_moments(float& n, float& mean, float& m2, float n2, float mean2, float m22) {
  const float all = n + n2, d = mean2 - mean, f = all > 0.f ? n2 / all : 0.f;
  mean = fmaf(d, f, mean);
  m2 += m22 + d * d * n * f;
  n = all;
}

// four partial sums of CTA `rank` of the cluster (its own through the same window)
LB_DEVICE float4 gs_ld_remote(uint32_t addr, uint32_t rank) {
  uint32_t ra;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
  return v;
}

// grid (cluster, tiles of 128 columns of y, tiles of NT rows of y).  NORM: x are the rows before a layer or RMS norm; the epilogue's warps read them, take their
// statistics (every CTA those of all its rows) and write the normalised bf16 rows of each k-block where TMA would have put them, while w is on its way.
template <int NT, int RANKS, bool NORM>
__global__ void __launch_bounds__(GS_THREADS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, GemmSmallArgs<NORM> p) {
  using Cfg = GsCfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int STAGE = NORM ? GS_W_BYTES : Cfg::STAGE;             // NORM: all of the CTA's rows of x behind the stages of w
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * STAGE + (NORM ? p.kb_per_cta * Cfg::X_BYTES : 0));
  uint64_t* empty_bar = full_bar + GS_MAX_STAGES;
  uint64_t* acc_full = empty_bar + GS_MAX_STAGES;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* stop = reinterpret_cast<volatile int*>(acc_full + 2);
  [[maybe_unused]] uint64_t* x_full = acc_full + 3;
  [[maybe_unused]] float* row_mean = reinterpret_cast<float*>(full_bar + 20);       // 16, then 16 reciprocal deviations (NORM: NT = 16)
  static_assert(!NORM || (NT == 16 && 2 * GS_MAX_STAGES + 4 <= 20), "statistics lie behind the barriers");
  static_assert(!NORM || (GS_SMEM - GS_NORM_BLOCKS * Cfg::X_BYTES) / GS_W_BYTES == 4, "stages of w beside the most rows of x");
  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int rank = blockIdx.x;
  const int n0 = blockIdx.y * 128, m0 = blockIdx.z * NT;
  const int kb_total = (p.K + 63) / 64, kb0 = min(kb_total, rank * p.kb_per_cta), kb1 = min(kb_total, kb0 + p.kb_per_cta);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    if constexpr (!NORM) tma_prefetch_desc(&tmap_x);
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
    if constexpr (NORM) mbar_init(x_full, 4);
    mbar_init(acc_full, 1);
    *stop = 0;
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 1) tmem_alloc<Cfg::TMEM>(tmem_ptr_smem);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  if (threadIdx.x == 32)                     // on its way to L2 while the kernel before this one ends; the warp whose own work begins last
    for (int kb = kb0; kb < min(kb1, kb0 + p.ahead); ++kb) tma_prefetch_2d(&tmap_w, kb * 64, n0);
  [[maybe_unused]] const __nv_bfloat16 *xg = nullptr, *gamma = nullptr, *beta = nullptr;
  if constexpr (NORM) { xg = p.x; gamma = p.gamma; beta = p.beta; }
  chain_wait(xg, gamma, beta);
  chain_next();

  if (warp_idx == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 1;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!tc_wait(&empty_bar[s], phase, stop)) break;
        uint8_t* sw = smem + s * STAGE;
        mbar_arrive_expect_tx(&full_bar[s], STAGE);
        tma_load_2d(sw, &tmap_w, &full_bar[s], kb * 64, n0);
        if constexpr (!NORM) tma_load_2d(sw + GS_W_BYTES, &tmap_x, &full_bar[s], kb * 64, m0);
        if (++s == p.stages) { s = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(128, NT, false, false);
    bool ok = true;
    if constexpr (NORM) ok = __all_sync(0xffffffffu, tc_wait(x_full, 0, stop));
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = __all_sync(0xffffffffu, ok && tc_wait(&full_bar[s], phase, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        const uint32_t sw = smem_u32(smem + s * STAGE), sx = NORM ? smem_u32(smem + p.stages * STAGE + (kb - kb0) * Cfg::X_BYTES) : sw + GS_W_BYTES;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ss(tmem_base, make_smem_desc_sw128(sw + k * 32, 0, 1024), make_smem_desc_sw128(sx + k * 32, 0, 1024), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
        if (kb == kb1 - 1) umma_commit(acc_full);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; phase ^= 1; }
    }
  }
  if constexpr (NORM) {
    if (warp_idx >= 2) {
      const int tid = static_cast<int>(threadIdx.x) - 64, rows = min(16, p.M - m0);
      auto unpack8 = [](const uint4& q, float (&v)[8]) {
        const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), c = unpack_bf16(q.z), d = unpack_bf16(q.w);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
      };
      // 16 bytes of a row of a k-block; those of the first two k-blocks are on their way while the statistics are taken
      const int row = tid / 8, chunk = tid % 8;
      const bool live = row < rows;
      const __nv_bfloat16* xr = xg + static_cast<size_t>(m0 + (live ? row : 0)) * p.ldx;
      uint4 first[2][3];
      auto fetch = [&](int kb, uint4 (&q)[3]) {
        const int k = kb * 64 + chunk * 8;
        q[0] = q[1] = q[2] = make_uint4(0u, 0u, 0u, 0u);
        if (live && kb < kb1 && k < p.K) {
          q[0] = *reinterpret_cast<const uint4*>(xr + k);
          q[1] = *reinterpret_cast<const uint4*>(gamma + k);
          if (beta != nullptr) q[2] = *reinterpret_cast<const uint4*>(beta + k);
        }
      };
      fetch(kb0, first[0]);
      fetch(kb0 + 1, first[1]);
      {                                             // statistics: a power of two of threads per row, as many as there are
        int lanes = 8;
        while (lanes < 128 && rows * lanes * 2 <= 128) lanes *= 2;
        const int srow = tid / lanes, sub = tid % lanes;
        float n = 0.f, mean = 0.f, m2 = 0.f;
        if (srow < rows) {
          const __nv_bfloat16* sr = xg + static_cast<size_t>(m0 + srow) * p.ldx;
          for (int k = sub * 8; k < p.K; k += lanes * 32) {          // up to 32 numbers at a time: their mean, then their deviations from it
            uint4 q[4];
            float cnt = 0.f, sum = 0.f, sq = 0.f;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              const bool in = k + a * lanes * 8 < p.K;
              q[a] = in ? *reinterpret_cast<const uint4*>(sr + k + a * lanes * 8) : make_uint4(0u, 0u, 0u, 0u);
              cnt += in ? 8.f : 0.f;
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              float v[8];
              unpack8(q[a], v);
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                sum += v[e];
                if (p.rms) sq = fmaf(v[e], v[e], sq);
              }
            }
            if (p.rms) {
              m2 += sq;
              continue;
            }
            const float c = sum / cnt;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              float v[8];
              unpack8(q[a], v);
              float part = 0.f;
#pragma unroll
              for (int e = 0; e < 8; ++e) part = fmaf(v[e] - c, v[e] - c, part);
              sq += 8.f * a < cnt ? part : 0.f;
            }
            merge_moments(n, mean, m2, cnt, c, sq);
          }
        }
        for (int m = 1; m < min(lanes, 32); m <<= 1) {
          const float n2 = __shfl_xor_sync(0xffffffffu, n, m), mean2 = __shfl_xor_sync(0xffffffffu, mean, m), m22 = __shfl_xor_sync(0xffffffffu, m2, m);
          if (p.rms) m2 += m22;
          else merge_moments(n, mean, m2, n2, mean2, m22);
        }
        float* over = row_mean + 32;                // sums of whole warps, where a row has several: [warp][3]
        if (lanes > 32) {
          if (lane == 0) {
            over[(warp_idx - 2) * 3] = n;
            over[(warp_idx - 2) * 3 + 1] = mean;
            over[(warp_idx - 2) * 3 + 2] = m2;
          }
          asm volatile("bar.sync 1, 128;\n" ::: "memory");
          const int per = lanes / 32, first = (warp_idx - 2) / per * per;
          n = over[first * 3];
          mean = over[first * 3 + 1];
          m2 = over[first * 3 + 2];
          for (int w = first + 1; w < first + per; ++w) {
            if (p.rms) m2 += over[w * 3 + 2];
            else merge_moments(n, mean, m2, over[w * 3], over[w * 3 + 1], over[w * 3 + 2]);
          }
        }
        if (sub == 0 && srow < rows) {
          row_mean[srow] = p.rms ? 0.f : mean;
          row_mean[16 + srow] = rsqrtf(m2 / p.K + p.eps);
        }
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
      }
      const float mean = live ? row_mean[row] : 0.f, rstd = live ? row_mean[16 + row] : 0.f;
      uint8_t* xs = smem + p.stages * STAGE;        // the CTA's k-blocks one behind the other
      auto put = [&](int kb, const uint4 (&q)[3]) {
        float v[8], g[8], b[8];
        unpack8(q[0], v);
        unpack8(q[1], g);
        unpack8(q[2], b);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = fmaf((v[e] - mean) * rstd, g[e], b[e]);          // (zeros behind the rows and columns there are)
        *reinterpret_cast<uint4*>(xs + (kb - kb0) * Cfg::X_BYTES + row * 128 + ((chunk ^ (row & 7)) << 4)) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
      };
      if (kb0 < kb1) put(kb0, first[0]);
      if (kb0 + 1 < kb1) put(kb0 + 1, first[1]);
#pragma unroll 2
      for (int kb = kb0 + 2; kb < kb1; ++kb) {
        fetch(kb, first[0]);
        put(kb, first[0]);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(x_full);
    }
  }
  // the pipeline has run dry once acc_full has come (every full stage was consumed): its memory holds the partial sums [NT][128] now
  float* part = reinterpret_cast<float*>(smem);
  if (warp_idx >= 2) {
    const int quad = warp_idx % 4, n_local = quad * 32 + lane;
    if (kb0 < kb1) {
      tc_wait(acc_full, 0, stop);
      __syncwarp();
      tc_fence_after_sync();
    }
    const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll
    for (int c = 0; c < NT; c += 16) {
      if (m0 + c >= p.M) break;                    // rows that do not exist are not read below
      uint32_t r[16];
      if (kb0 < kb1) {
        tmem_ld_32x32b_x16(t_addr + c, r);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c + j) * 128 + n_local] = __uint_as_float(r[j]);
    }
  }
  if constexpr (RANKS > 1) cluster_sync_all();
  else __syncthreads();
  if (warp_idx >= 2) {
    // a warp finishes one row at a time, four columns per lane; the cluster's CTAs take the rows in turn
    const int n = n0 + lane * 4;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias != nullptr && n < p.N) {
      const uint2 q = *reinterpret_cast<const uint2*>(p.bias + n);
      const float2 b0 = unpack_bf16(q.x), b1 = unpack_bf16(q.y);
      bias[0] = b0.x; bias[1] = b0.y; bias[2] = b1.x; bias[3] = b1.y;
    }
#pragma unroll 2
    for (int j = rank + (warp_idx - 2) * RANKS; j < NT; j += 4 * RANKS) {
      if (m0 + j >= p.M || n >= p.N) break;
      const uint32_t at = smem_u32(part + j * 128 + lane * 4);
      float4 f[RANKS];
#pragma unroll
      for (int r = 0; r < RANKS; ++r) f[r] = RANKS > 1 ? gs_ld_remote(at, r) : *reinterpret_cast<const float4*>(part + j * 128 + lane * 4);
      float v[4] = {bias[0], bias[1], bias[2], bias[3]};
#pragma unroll
      for (int r = 0; r < RANKS; ++r) { v[0] += f[r].x; v[1] += f[r].y; v[2] += f[r].z; v[3] += f[r].w; }
      const size_t o = static_cast<size_t>(m0 + j) * p.ldo + n;
      if (p.pre_out != nullptr) *reinterpret_cast<uint2*>(p.pre_out + o) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
      if (p.residual != nullptr) {
        const uint2 q = *reinterpret_cast<const uint2*>(p.residual + o);
        const float2 r0 = unpack_bf16(q.x), r1 = unpack_bf16(q.y);
        v[0] += r0.x; v[1] += r0.y; v[2] += r1.x; v[3] += r1.y;
      } else if (p.act == ACT_GELU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = gelu_fast(v[e]);
      } else if (p.act != ACT_NONE) {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = act_fwd(v[e], p.act);
      }
      *reinterpret_cast<uint2*>(p.out + o) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
    }
  }
  __syncwarp();                                    // lanes behind column N left the loop early; the cluster's barrier takes whole warps
  if constexpr (RANKS > 1) cluster_sync_all();     // nobody leaves while its partial sums are read
  tc_fence_before_sync();
  __syncthreads();
  if (*stop) {
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0) { *const_cast<volatile int*>(p.err) = 1; __threadfence_system(); }
    __syncthreads();
  }
  if (warp_idx == 1) {
    tc_fence_after_sync();
    tmem_dealloc<Cfg::TMEM>(tmem_base);
  }
}

template <int NT, int RANKS, bool NORM = false>
cudaError_t launch_gemm_small_r(const CUtensorMap& tw, const CUtensorMap& tx, GemmSmallArgs<NORM> p, cudaStream_t s) {
  auto kern = gemm_small_kernel<NT, RANKS, NORM>;
  const int stage = NORM ? GS_W_BYTES : GsCfg<NT>::STAGE, rows = NORM ? p.kb_per_cta * GsCfg<NT>::X_BYTES : 0;
  const int fit = (GS_SMEM - rows) / stage;
  p.ahead = (long)p.N * p.K * 2 >= GS_AHEAD_BYTES ? GS_AHEAD : 0;
  p.stages = p.kb_per_cta < 2 ? 2 : p.kb_per_cta;
  if (p.stages > fit) p.stages = fit;
  const int smem = p.stages * stage + rows + GS_TAIL;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM + GS_TAIL);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  return lb_host::launch_chained(kern, dim3((unsigned)RANKS, (unsigned)((p.N + 127) / 128), (unsigned)((p.M + NT - 1) / NT)), dim3(GS_THREADS), (size_t)smem, s,
                                 (unsigned)RANKS, tw, tx, p);
}
template <int NT>
cudaError_t launch_gemm_small(const CUtensorMap& tw, const CUtensorMap& tx, const GemmSmallParams& p, int ranks, cudaStream_t s) {
  switch (ranks) {
    case 1: return launch_gemm_small_r<NT, 1>(tw, tx, p, s);
    case 2: return launch_gemm_small_r<NT, 2>(tw, tx, p, s);
    case 4: return launch_gemm_small_r<NT, 4>(tw, tx, p, s);
    default: return launch_gemm_small_r<NT, 8>(tw, tx, p, s);
  }
}

}  // namespace lb

namespace {
// mapped host word that a kernel sets when one of its bounded waits ran out; nullptr: it could not be had, or is set
int* small_wait_word() {
  static std::mutex lock;
  static int* host = nullptr;
  std::lock_guard<std::mutex> guard(lock);
  if (host == nullptr) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;       // the first call may come inside a capture
    cudaThreadExchangeStreamCaptureMode(&mode);
    int* word = nullptr;
    const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&word), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return nullptr;
    *word = 0;
    host = word;
  }
  if (*static_cast<volatile int*>(host) != 0) return nullptr;
  int* dev = nullptr;
  return cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev), host, 0) == cudaSuccess ? dev : nullptr;
}
}  // namespace

// Whether this kernel is the better one, with `nt` rows of x per tile and `ranks` CTAs per tile.
//   this kernel:     3.4 us + 0.03 us per row of the tile + the merge of a cluster (0.1 us of 2, 0.2 us of 4 CTAs, 8 ns per row of the tile
//                    of 8) + the larger of: the k-blocks of a CTA (0.28 us each with 16 rows, 0.34 with 32 and 64, 0.38 with 128; up to 1.8
//                    times that where two CTAs share an SM), w at 6 TB/s
//   gemm_sm100.cu:   lb_gemm_tile_us
// Fitted over 350 products, M = 1 .. 2048 and w from [384, 384] to [50304, 1024] and [4096, 11008] (7 % and 3 % rms).  Up to 32 rows this
// kernel was the better one everywhere (nearest: [32, 1024] x [50304, 1024] 24.8 against 25.3 us); above that it is taken where the estimate
// is 4 % and 0.5 us ahead: few tiles and a long K ([128, 4096] x [1024, 4096] 9.3 against 19.9 us, [200, 11008] x [4096, 11008] 28.6 against
// 46.6), not many tiles ([64, 1024] x [50304, 1024] 27.3 against 23.4 us, [2048, 5120] x [1280, 5120] 39.6 against 29.3) and not a short K
// ([256, 384] x [1536, 384] 6.2 against 5.8).  Near the line, 414 products with 33 to 2048 rows, it is 0.2 % from the better kernel on average; 0.45 us instead of 0.5 would win
// [136 .. 152, 384] x [1152, 384] (4.9 against 5.2) and lose [512, 768] x [768, 768] and [128, 768] x [3072, 768] (6.8 against 6.6).  Clusters of 4 and 8 are kept to 264 CTAs: the SMs of a GPC do not divide by them, and 72
// clusters of 4 with two CTAs per SM ran in two waves ([96, 1024] x [3072, 1024] 10.2 against 8.2 us).
// More than 2048 rows only against one tile of 16 to 128 columns (the gates of a mixer), where the other kernel walks all of K in one CTA:
// [2560, 2048] x [16, 2048] 9.6 against 11.1 us, x [128, 2048] 9.2 against 11.4, [4096, 4096] x [32, 4096] 9.8 against 18.6, [8192, 4096] x [64, 4096]
// 14.0 against 19.3; with 8 columns [8192, 4096] 19.7 against 18.9, and [16384, 2048] x [64, 2048] 15.5 against 12.1.
extern "C" double lb_gemm_tile_us(int M, int N, int K);
extern "C" int lb_gemm_small_rule(int M, int N, int K, int* nt, int* ranks) {
  if (M > (N < 16 || N > 128 ? 2048 : 8192)) return 0;
  const int kb = (K + 63) / 64, tiles_n = (N + 127) / 128;
  const double w_us = (double)N * K * 2 / 6e6;
  const double block_us[4] = {0.28, 0.34, 0.34, 0.38};
  double best = 1e30;
  for (int i = 0; i < 4; ++i) {
    const int t = 16 << i;
    if (t < 128 && M > 8 * t) continue;                       // tiles of few rows would read w over and over
    if (t > 16 && M <= t / 2) break;
    const long tiles = (long)tiles_n * ((M + t - 1) / t);
    for (int lg = 0; lg < 4; ++lg) {
      const int r = 1 << lg;
      if (r > 1 && (tiles * r > (r > 2 ? 264 : 296) || kb < r)) break;
      const int per = (kb + r - 1) / r;
      const long ctas = tiles * r, waves = (ctas + 295) / 296;
      const double load = (ctas < 296 ? ctas : 296) / 148.0;
      double us = waves * per * block_us[i] * (load > 1 ? 1 + 0.8 * (load - 1) : 1);
      if (w_us > us) us = w_us;
      us += 3.4 + 0.03 * t + (r < 8 ? 0.1 * lg : 0.008 * t) + 1.5 * (waves - 1);
      if (us < best - 1e-9) {
        best = us;
        *nt = t;
        *ranks = r;
      }
    }
  }
  if (M <= 32) return 1;
  const double old_us = lb_gemm_tile_us(M, N, K);
  return best * 1.04 < old_us && best + 0.5 < old_us;
}

// Returns 0, a cudaError_t, or a negative code for unsupported arguments (-20: an earlier launch's wait ran out).
extern "C" int lb_gemm_small(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldo, const void* bias, int act,
                             void* pre_out, const void* residual, int nt, int ranks, cudaStream_t s) {
  const uintptr_t vec = reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(pre_out) | reinterpret_cast<uintptr_t>(residual);
  if (M <= 0 || N <= 0 || K <= 0 || N % 4 || ldo % 4 || (vec & 7) || ldx % 8 || ldw % 8 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
    return -1;
  if ((M + nt - 1) / nt > 65535 || (N + 127) / 128 > 65535) return -1;
  lb::GemmSmallParams p{};
  p.err = small_wait_word();
  if (p.err == nullptr) return -20;
  p.M = M; p.N = N; p.K = K;
  p.kb_per_cta = ((K + 63) / 64 + ranks - 1) / ranks;
  p.bias = (const __nv_bfloat16*)bias;
  p.residual = (const __nv_bfloat16*)residual;
  p.out = (__nv_bfloat16*)out;
  p.pre_out = (__nv_bfloat16*)pre_out;
  p.ldo = ldo;
  p.act = act;
  auto map = [&](CUtensorMap* m, const void* ptr, int rows, int ld, int box_rows) {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)rows};
    uint64_t strides[2] = {2, (uint64_t)ld * 2};
    uint32_t box[2] = {64u, (uint32_t)box_rows};
    return lb_host::make_tmap_bf16(m, ptr, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  CUtensorMap tw, tx;
  if (!map(&tw, w, N, ldw, 128) || !map(&tx, x, M, ldx, nt)) return -2;
  cudaError_t e = nt == 16 ? lb::launch_gemm_small<16>(tw, tx, p, ranks, s) : nt == 32 ? lb::launch_gemm_small<32>(tw, tx, p, ranks, s)
                  : nt == 64 ? lb::launch_gemm_small<64>(tw, tx, p, ranks, s) : lb::launch_gemm_small<128>(tw, tx, p, ranks, s);
  return (int)e;
}

// The same for up to 16 rows with a layer norm (without beta, `rms`: an RMS norm) of x in front: y = act(norm(x) · wᵀ + bias), two launches in one.  [8, 1024] x
// [3072, 1024] and [4096, 1024] 6.8 us each, where norm and product took 2.4 + 4.9; what counts is the launch that the host does not make: a step of GPT-2 against a cache
// (5 launches in place of 7) 44.5 -> 39.3 us.  Not where a CTA has more than 11 k-blocks ([4, 4096] x [12288, 4096], 32 of them): their rows do not fit beside the stages
// of w, and normalised k-block by k-block behind w they hold it up (three products of Llama-2 7B 63 + 5 us for the norms, 83 so).
extern "C" int lb_gemm_small_norm(const void* x, const void* gamma, const void* beta, float eps, int rms, const void* w, void* out, int M, int N, int K, int ldx,
                                  int ldw, int ldo, const void* bias, int act, cudaStream_t s) {
  const uintptr_t vec = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta) | reinterpret_cast<uintptr_t>(w);
  if (M <= 0 || M > 16 || N <= 0 || K <= 0 || N % 4 || K % 8 || ldo % 4 || ldx % 8 || ldw % 8 || (vec & 15) ||
      ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(bias)) & 7) || (N + 127) / 128 > 65535)
    return -1;
  int nt = 0, ranks = 0;
  if (!lb_gemm_small_rule(M, N, K, &nt, &ranks) || nt != 16) return -1;
  if (((K + 63) / 64 + ranks - 1) / ranks > lb::GS_NORM_BLOCKS) return -1;
  lb::GemmSmallNormParams p{};
  p.err = small_wait_word();
  if (p.err == nullptr) return -20;
  p.M = M; p.N = N; p.K = K;
  p.kb_per_cta = ((K + 63) / 64 + ranks - 1) / ranks;
  p.bias = (const __nv_bfloat16*)bias;
  p.out = (__nv_bfloat16*)out;
  p.ldo = ldo;
  p.act = act;
  p.x = (const __nv_bfloat16*)x; p.gamma = (const __nv_bfloat16*)gamma; p.beta = (const __nv_bfloat16*)beta;
  p.ldx = ldx; p.rms = rms; p.eps = eps;
  CUtensorMap tw;
  const uint64_t dims[2] = {(uint64_t)K, (uint64_t)N}, strides[2] = {2, (uint64_t)ldw * 2};
  const uint32_t box[2] = {64u, 128u};
  if (!lb_host::make_tmap_bf16(&tw, w, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -2;
  switch (ranks) {
    case 1: return (int)lb::launch_gemm_small_r<16, 1, true>(tw, tw, p, s);
    case 2: return (int)lb::launch_gemm_small_r<16, 2, true>(tw, tw, p, s);
    case 4: return (int)lb::launch_gemm_small_r<16, 4, true>(tw, tw, p, s);
    default: return (int)lb::launch_gemm_small_r<16, 8, true>(tw, tw, p, s);
  }
}

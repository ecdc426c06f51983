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
constexpr int GS_MAX_STAGES = GS_SMEM / GsCfg<16>::STAGE, GS_TAIL = 1024 + 256;   // alignment, barriers

struct GemmSmallParams {
  int M, N, K, kb_total, kb_per_cta, stages;
  const __nv_bfloat16* bias;      // [N] or nullptr
  const __nv_bfloat16* residual;  // [M, ldo] or nullptr
  __nv_bfloat16 *out, *pre_out;   // [M, ldo]; pre_out (optional): before the activation
  int ldo, act;
  int* err;
};

// four partial sums of CTA `rank` of the cluster (its own through the same window)
LB_DEVICE float4 gs_ld_remote(uint32_t addr, uint32_t rank) {
  uint32_t ra;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
  return v;
}

// grid (cluster, tiles of 128 columns of y, tiles of NT rows of y)
template <int NT, int RANKS>
__global__ void __launch_bounds__(GS_THREADS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, GemmSmallParams p) {
  using Cfg = GsCfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * Cfg::STAGE);
  uint64_t* empty_bar = full_bar + GS_MAX_STAGES;
  uint64_t* acc_full = empty_bar + GS_MAX_STAGES;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* stop = reinterpret_cast<volatile int*>(acc_full + 2);
  const int warp_idx = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int rank = blockIdx.x;
  const int n0 = blockIdx.y * 128, m0 = blockIdx.z * NT;
  const int kb0 = min(p.kb_total, rank * p.kb_per_cta), kb1 = min(p.kb_total, kb0 + p.kb_per_cta);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int i = 0; i < p.stages; ++i) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
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
  chain_wait();
  chain_next();

  if (warp_idx == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t phase = 1;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!tc_wait(&empty_bar[s], phase, stop)) break;
        uint8_t* sw = smem + s * Cfg::STAGE;
        mbar_arrive_expect_tx(&full_bar[s], Cfg::STAGE);
        tma_load_2d(sw, &tmap_w, &full_bar[s], kb * 64, n0);
        tma_load_2d(sw + GS_W_BYTES, &tmap_x, &full_bar[s], kb * 64, m0);
        if (++s == p.stages) { s = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp_idx == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(128, NT, false, false);
    bool ok = true;
    int s = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = __all_sync(0xffffffffu, ok && tc_wait(&full_bar[s], phase, stop));
      tc_fence_after_sync();
      if (ok && elect_one()) {
        const uint32_t sw = smem_u32(smem + s * Cfg::STAGE), sx = sw + GS_W_BYTES;
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

template <int NT, int RANKS>
cudaError_t launch_gemm_small_r(const CUtensorMap& tw, const CUtensorMap& tx, GemmSmallParams p, cudaStream_t s) {
  auto kern = gemm_small_kernel<NT, RANKS>;
  const int fit = GS_SMEM / GsCfg<NT>::STAGE;
  p.stages = p.kb_per_cta < 2 ? 2 : p.kb_per_cta;
  if (p.stages > fit) p.stages = fit;
  const int smem = p.stages * GsCfg<NT>::STAGE + GS_TAIL;
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
// ([256, 384] x [1536, 384] 6.2 against 5.8).  Clusters of 4 and 8 are kept to 264 CTAs: the SMs of a GPC do not divide by them, and 72
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
  p.kb_total = (K + 63) / 64;
  p.kb_per_cta = (p.kb_total + ranks - 1) / ranks;
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

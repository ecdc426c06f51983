// Persistent warp-specialised bf16 GEMM for sm_100a: TMA -> shared (128B swizzle) -> tcgen05.mma
// (accumulators in TMEM, double buffered) -> tcgen05.ld epilogue with fused bias / activation.
//
//   D[M,N] = A · Bᵀ   with three operand layouts (all row-major tensors in global memory):
//     NT: A[M,K], B[N,K]   (forward  : y  = x · Wᵀ)
//     NN: A[M,K], B[K,N]   (dgrad    : dx = dy · W,   B is "MN-major")
//     TN: A[K,M], B[K,N]   (wgrad    : dW = dyᵀ · x,  both "MN-major"; split-K + fp32 TMA reductions)
//
// Replaces the cuBLAS matmuls behind libai/layers/linear.py:123-157 and the separate
// fused_bias_add_gelu kernel (libai/layers/mlp.py:95) of the reference.
//
// Warp roles (320 threads): warp 0 = TMA producer, warp 1 = MMA issuer (+TMEM alloc),
// warps 2..9 = epilogue (TMEM lane quadrant = warp_idx % 4, column half = (warp_idx - 2) / 4: two warps per
// scheduler keep the elementwise epilogue math (bias, GELU, GELU') off the critical path).  One CTA per SM,
// static round-robin tile scheduler over (m_blk, n_blk, k_split).
#include "common.cuh"

#include <cmath>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace lb {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;  // 64 bf16 = 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr int NUM_THREADS = 320;
constexpr int NUM_EPI_THREADS = 256;

enum Epi : int { EPI_BF16 = 0, EPI_F32 = 1, EPI_ATOMIC_F32 = 2 };

struct GemmParams {
  int M, N, K;
  int k_splits;        // number of K partitions (atomic epilogue only when > 1)
  int group_m;         // row blocks per band of the tile order (1: row by row)
  int k_per_split;     // in units of BLOCK_K blocks
  const __nv_bfloat16* bias;  // [N] or nullptr
  int act;                    // Act enum
  void* out;                  // bf16 or fp32 [M, ldo]
  __nv_bfloat16* pre_out;     // optional pre-activation copy (bf16)
  const __nv_bfloat16* pre_in;  // optional [M, ldo]: out = acc * act'(pre_in)  (dgrad fused with the activation backward)
  int ldo;                    // leading dimension of out (elements)
  int rmw;                    // EPI_F32: out += acc (plain read-modify-write; a tile is owned by one CTA)
  // fp8 (E4M3) operands, K-major only.  The byte layout of a [rows, K] e4m3 matrix equals that of a [rows, K/2] bf16
  // matrix, so the TMA maps, the 128-byte swizzle rows and the 32-byte descriptor advance per MMA are unchanged (K
  // above is in bf16-equivalent units = bytes / 2); only the MMA kind (kind::f8f6f4, 32 elements of K per instruction)
  // and the dequantisation scale in the epilogue differ.
  // optional fp32 [N] vector receiving the column sums of the bf16 output (`red.add`): the bias gradient of the layer
  // whose output gradient this GEMM produces (dgrad fused with the activation backward), without a second pass
  float* colsum;
  int fp8;
  const float* deq_a;         // per-tensor dequantisation scales (device scalars): out = acc * deq_a[0] * deq_b[0]
  const float* deq_b;
  // grouped mode (NT layout, single-CTA tiles, no split-K): B is a stack of matrices [groups * N, K] and every BLOCK_M-row
  // block of A belongs to one of them — tile_group[m_blk] = its group, < 0 = the block holds no rows (skipped by all
  // roles alike).  The list lives in device memory, so the row counts of the groups never reach the host.
  const int* tile_group;
};

// Fused collective modes (tensor parallel): peer pointers refer to NVLink peer-mapped symmetric memory.
//   COMM_AG : all-gather -> GEMM.  One operand is the concatenation over ranks of [rows_per_rank, K] shards along its
//             row dimension: A for NT/NN (row blocks of the output), B for TN (`gathered_is_b`: the shards lie along
//             the REDUCTION dimension of the wgrad dW = dyᵀ · all_gather(x)).  Tiles / k-blocks that only need the local
//             shard read it through its own tensor map and start at once; `n_comm` dedicated CTAs push the local shard
//             into every peer's gathered buffer (TMA bulk copies over NVLink) meanwhile; per-row-block arrival counters
//             (bumped by the pushing peer) gate the TMA loads of the remote rows.
//   COMM_RS : GEMM -> reduce-scatter.  Each rank computes the full [M, N] partial product; the epilogue stores
//             row block tiles straight into the owner's staging slot (P2P stores) and bumps the owner's arrival
//             counter; after its tiles every CTA helps reducing the local rows (sum over sources + bias + residual).
// All handshake state lives in DEVICE memory and is advanced by the kernel itself (`state[0]` = number of completed
// calls on this buffer set): the launch parameters of a call site never change, so transformer blocks containing these
// kernels are captured into CUDA graphs and replayed.  Write-after-read safety of the symmetric buffers does not rely
// on any call-order convention: a rank publishes "finished call c" into every peer's `done` row when its kernel
// retires, and nobody writes call c+1 data into a peer's buffer before having seen that peer's "finished call c".
enum CommMode : int { COMM_NONE = 0, COMM_AG = 1, COMM_RS = 2 };
struct CommParams {
  int mode, world, rank;
  int rows_per_rank;            // rows of one shard, multiple of BLOCK_M
  int n_comm;                   // COMM_AG: number of copy CTAs
  int gathered_is_b;            // COMM_AG with the TN layout: the gathered operand is B, gated per k-block
  int fill_local;               // COMM_AG: the copy CTAs also write the local shard into the local gathered buffer
  int copy_rings;               // COMM_AG: independent copy engines (threads with their own smem ring) per copy CTA
  uint32_t arrivals;            // arrivals per row block and call (AG: 1; RS: world * n_blocks)
  uint32_t* state;              // local: [0] completed calls on this buffer set, [1] CTA exit counter
  __nv_bfloat16* peer_buf[8];   // AG: gathered buffers of all ranks; RS: staging buffers of all ranks
  uint32_t* peer_flags[8];      // per-row-block arrival counters of all ranks (AG: M/128 entries; RS: rows_per_rank/128)
  uint32_t* peer_done[8];       // [world] words on every rank: peer_done[q][r] = calls rank r has finished (written by r)
  const __nv_bfloat16* local_shard;  // AG: this rank's shard [rows_per_rank, K] (source of the pushes)
  const __nv_bfloat16* residual;  // RS: optional [rows_per_rank, N]
  __nv_bfloat16* rs_out;        // RS: [rows_per_rank, N]
  long staging_parity_off;      // RS: element offset of the staging half used by this call
  unsigned long long timeout_ns;  // bound of every cross-GPU flag wait (0 = default)
};

// streaming (non-volatile, L1 no-allocate) 128-bit load: many of these stay in flight per thread over NVLink
LB_DEVICE uint4 ld_stream_u4(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
LB_DEVICE uint32_t ld_acquire_gpu_u32(const uint32_t* a) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(a) : "memory");
  return v;
}

template <int BLOCK_N, int CTAS = 1, bool REDUCE = false, bool B_MN = false>
struct StageCfg {
  static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;
  // CTA pair: each CTA stages half of the B tile (where that lies along rows, in whole boxes of 64 columns, of which the last may hold more than the half)
  static constexpr int B_COLS = B_MN ? (BLOCK_N / CTAS + 63) / 64 * 64 : BLOCK_N / CTAS;
  static constexpr int B_BYTES = B_COLS * BLOCK_K * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int NUM_STAGES = CTAS == 2 ? (BLOCK_N == 128 ? 8 : (B_COLS == 96 ? 7 : 6))
                                              : ((BLOCK_N == 256) ? 4 : (BLOCK_N == 192 ? (REDUCE ? 4 : 5) : (BLOCK_N == 128 ? 6 : 8)));
  static constexpr int STAGING_SLOT = REDUCE ? 4096 : 2048;   // per epilogue warp: a 32 x 32 chunk in fp32 (box of a TMA reduction) or bf16
  static constexpr int STAGING_BYTES = 8 * STAGING_SLOT;
  static constexpr int SMEM_BYTES = NUM_STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/ + STAGING_BYTES;
  static_assert(SMEM_BYTES <= 232448, "shared memory of one CTA");
  static constexpr uint32_t TMEM_COLS = (2 * BLOCK_N <= 32) ? 32 : (2 * BLOCK_N <= 64 ? 64 : (2 * BLOCK_N <= 128 ? 128 : (2 * BLOCK_N <= 256 ? 256 : 512)));
};

// ---- epilogue staging: row-per-lane (TMEM layout) <-> 4-lanes-per-row (coalesced global layout) ----------------
// A 32x32 bf16 chunk is 32 rows x 64 B.  `tcgen05.ld.32x32b` gives every lane one ROW, so a direct 16-byte global
// access per lane touches 32 different 128-byte lines per instruction (the L1/LSU wavefront count, not the tensor
// pipe, bounded the K=1024 GEMMs: ncu l1tex 63 %, tensor pipe 39 %).  Staging the chunk through 2 KB of shared
// memory per warp turns that into 8 rows x 64 contiguous bytes per instruction.  16-byte slots are XOR-swizzled with
// (row >> 1) & 3 so both the row-wise and the transposed access are bank-conflict free.
LB_DEVICE uint32_t stg_off(int row, int slot) { return static_cast<uint32_t>(row * 64 + ((slot ^ ((row >> 1) & 3)) << 4)); }
// lane holds its row as 4 x uint4 -> after the call lane holds slot (lane & 3) of rows 8j + (lane >> 2), j = 0..3
LB_DEVICE void stg_rows_to_quads(uint8_t* stg, int lane, const uint4 (&rowv)[4], uint4 (&quad)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(stg + stg_off(lane, i)) = rowv[i];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) quad[j] = *reinterpret_cast<const uint4*>(stg + stg_off(8 * j + (lane >> 2), lane & 3));
  __syncwarp();
}
LB_DEVICE void stg_quads_to_rows(uint8_t* stg, int lane, const uint4 (&quad)[4], uint4 (&rowv)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(stg + stg_off(8 * j + (lane >> 2), lane & 3)) = quad[j];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) rowv[i] = *reinterpret_cast<const uint4*>(stg + stg_off(lane, i));
  __syncwarp();
}
// store a staged chunk: slab = pointer to (first row of this warp's 32-row slab, first column of the chunk)
// colsum_dst (optional): fp32 pointer to the chunk's first column; receives the sums over the chunk's valid rows of
// the bf16-rounded values (4 rows in-register, then the 8 lanes that share a 16-byte column slot, then one red.add.v4
// pair per slot)
LB_DEVICE void stg_store_chunk(uint8_t* stg, int lane, const float (&v)[32], __nv_bfloat16* slab, size_t ld,
                               int rows_valid, int cols_valid, float* colsum_dst = nullptr) {
  uint4 rowv[4], quad[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    rowv[i] = make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                         pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
  stg_rows_to_quads(stg, lane, rowv, quad);
  const int sub = lane & 3;
  if (sub * 8 < cols_valid) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int rr = 8 * j + (lane >> 2);
      if (rr < rows_valid) *reinterpret_cast<uint4*>(slab + static_cast<size_t>(rr) * ld + sub * 8) = quad[j];
    }
  }
  if (colsum_dst != nullptr) {  // warp-uniform
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (8 * j + (lane >> 2) < rows_valid) {
        const float2 a = unpack_bf16(quad[j].x), b = unpack_bf16(quad[j].y), c = unpack_bf16(quad[j].z), d = unpack_bf16(quad[j].w);
        s[0] += a.x; s[1] += a.y; s[2] += b.x; s[3] += b.y; s[4] += c.x; s[5] += c.y; s[6] += d.x; s[7] += d.y;
      }
    }
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
#pragma unroll
      for (int k = 0; k < 8; ++k) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
    }
    if ((lane >> 2) == 0 && sub * 8 < cols_valid) {
      float* dst = colsum_dst + sub * 8;
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst), "f"(s[0]), "f"(s[1]), "f"(s[2]), "f"(s[3]) : "memory");
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst + 4), "f"(s[4]), "f"(s[5]), "f"(s[6]), "f"(s[7]) : "memory");
    }
  }
}

// What only some kinds of the kernel take lies behind the collectives' parameters in one argument, so that the others pass nothing for it.  What a launch costs the host depends on the
// bytes of its arguments: with 57 to 72 beyond a multiple of 64 it is 0.25 us less (776 bytes and 56 more 3.5 us, 8 to 48 more 3.7 to 3.8; an empty struct as an argument of its own had made
// 776 bytes 777).
struct GemmReduce : CommParams { CUtensorMap map; };      // EPI_ATOMIC_F32: the output in boxes of 32 x 32
// MULTI: B is several matrices [n[i], K] in memory of their own, one after the other along the columns of the output (NT, CTA pairs, bf16 results)
constexpr int GEMM_MAX_B = 8;
struct GemmMultiB : CommParams {
  CUtensorMap map[GEMM_MAX_B];
  int count;
  int n[GEMM_MAX_B], first[GEMM_MAX_B + 1], col[GEMM_MAX_B];   // columns; first tile along N; first column of the output
};
template <int EPI, bool MULTI> struct GemmMore { using type = CommParams; };
template <> struct GemmMore<EPI_ATOMIC_F32, false> { using type = GemmReduce; };
template <> struct GemmMore<EPI_BF16, true> { using type = GemmMultiB; };
constexpr int cheap_args(int bytes) { return (bytes + 7) % 64 < 16; }
static_assert(cheap_args(3 * sizeof(CUtensorMap) + sizeof(GemmParams) + sizeof(CommParams)) && cheap_args(sizeof(GemmReduce)) && cheap_args(sizeof(GemmMultiB)),
              "bytes of the arguments (those of the last two begin on a multiple of 64)");

// CTAS == 2: `cta_group::2` — clusters of two CTAs (one TPC) compute 256 x BLOCK_N tiles; no fused collectives, bf16 only.
template <int BLOCK_N, bool A_MN, bool B_MN, int EPI, bool FP8 = false, int CTAS = 1, bool MULTI = false>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
            const __grid_constant__ CUtensorMap tmap_g /* COMM_AG: the local shard of the gathered operand */,
            GemmParams p, const __grid_constant__ typename GemmMore<EPI, MULTI>::type cp) {
  using Cfg = StageCfg<BLOCK_N, CTAS, EPI == EPI_ATOMIC_F32, B_MN>;
  constexpr int NS = Cfg::NUM_STAGES;
  static_assert(CTAS == 1 || (CTAS == 2 && BLOCK_N >= 128 && !FP8), "CTA-pair mode: bf16 tiles of 128 columns and more");
  const int cta_rank = CTAS == 2 ? static_cast<int>(cluster_ctarank()) : 0;   // 0 = leader of the pair
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + NS * Cfg::STAGE_BYTES;        // one slot per epilogue warp (on 1024 bytes: swizzled boxes)
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + Cfg::STAGING_BYTES);
  uint64_t* empty_bar = full_bar + NS;
  uint64_t* tmem_full = empty_bar + NS;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp_idx = threadIdx.x / 32;
  const int lane = threadIdx.x % 32;

  // (CTA pair: `m_blocks` counts 256-row blocks = one per pair; this CTA works on rows [256 m + 128 rank, +128))
  const int m_blocks = (p.M + BLOCK_M * CTAS - 1) / (BLOCK_M * CTAS);
  static_assert(!MULTI || (CTAS == 2 && !A_MN && !B_MN && EPI == EPI_BF16), "several B: NT products on CTA pairs, bf16 results");
  int n_blocks = (p.N + BLOCK_N - 1) / BLOCK_N;
  if constexpr (MULTI) n_blocks = cp.first[cp.count];
  [[maybe_unused]] auto segment = [&](int n_blk) {          // MULTI: which matrix a column tile belongs to
    int i = 0;
    if constexpr (MULTI)
      while (n_blk >= cp.first[i + 1]) ++i;
    return i;
  };
  const int k_blocks_total = (p.K + BLOCK_K - 1) / BLOCK_K;
  const int num_tiles = m_blocks * n_blocks * p.k_splits;
  // CTAs [0, n_comm) are copy CTAs in COMM_AG mode; the rest run the GEMM roles
  const int n_comm = (cp.mode == COMM_AG) ? cp.n_comm : 0;
  const int cta = (static_cast<int>(blockIdx.x) - n_comm) / CTAS;
  const int cta_stride = (static_cast<int>(gridDim.x) - n_comm) / CTAS;
  const int mbpr = cp.mode != COMM_NONE ? cp.rows_per_rank / BLOCK_M : m_blocks;
  const bool ag_b = cp.mode == COMM_AG && cp.gathered_is_b != 0;   // TN wgrad: shards along the reduction dimension
  // row blocks are visited owner by owner: AG starts with the local rows (already resident), RS ends with them
  // (in units of one CTA tile row = BLOCK_M * CTAS rows; a shard holds mbpr / CTAS of them)
  auto map_m = [&](int m_seq) -> int {
    if (cp.mode == COMM_NONE || ag_b) return m_seq;
    const int upr = mbpr / CTAS;
    const int shift = (cp.mode == COMM_AG) ? 0 : 1;
    const int owner = (cp.rank + shift + m_seq / upr) % cp.world;
    return owner * upr + m_seq % upr;
  };
  // work item -> (output tile, K partition).  Default: partitions of one tile are neighbours (their reductions hit L2
  // together).  Gathered-B wgrad: partition-major, starting with the partitions that lie in the local shard (the host
  // makes k_splits a multiple of world and partitions never straddle a shard boundary), so every CTA has local work
  // while the remote shards are still in flight.
  const int mn_tiles = m_blocks * n_blocks;
  auto decode_tile = [&](int tile, int& mn, int& split) {
    if (ag_b) {
      mn = tile % mn_tiles;
      split = (tile / mn_tiles + cp.rank * (p.k_splits / cp.world)) % p.k_splits;
    } else {
      mn = tile / p.k_splits;
      split = tile % p.k_splits;
      if (p.group_m > 1) {                    // bands of group_m row blocks, row blocks fastest
        const int band = mn / (p.group_m * n_blocks), first = band * p.group_m, r = mn - first * n_blocks;
        const int rows = min(p.group_m, m_blocks - first);
        mn = (first + r % rows) * n_blocks + r / rows;
      }
    }
  };
  // handshake epoch of this call: number of calls already completed on this buffer set (identical on all ranks; the
  // last CTA to leave advances it, i.e. nobody modifies it while any CTA of this launch may still read it)
  const uint32_t call_idx = cp.mode != COMM_NONE ? *reinterpret_cast<volatile const uint32_t*>(cp.state) : 0u;
  const uint32_t arrive_target = (call_idx + 1u) * cp.arrivals;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_a);
    if constexpr (MULTI) {
      for (int i = 0; i < cp.count; ++i) tma_prefetch_desc(&cp.map[i]);
    } else {
      tma_prefetch_desc(&tmap_b);
    }
    if (cp.mode == COMM_AG) tma_prefetch_desc(&tmap_g);
    if constexpr (EPI == EPI_ATOMIC_F32) tma_prefetch_desc(&cp.map);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full_bar[i], CTAS);   // pair: the leader's barrier collects one arrival per CTA (+ both CTAs' bytes)
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&tmem_full[0], 1);
    mbar_init(&tmem_full[1], 1);
    // (pair: one arrival per epilogue WARP of both CTAs on the leader's barrier — 256 remote arrivals per tile would
    // be needless cluster traffic)
    mbar_init(&tmem_empty[0], CTAS == 2 ? 16 : NUM_EPI_THREADS);
    mbar_init(&tmem_empty[1], CTAS == 2 ? 16 : NUM_EPI_THREADS);
    fence_barrier_init();
    fence_proxy_async();
  }
  if (warp_idx == 1) {
    if constexpr (CTAS == 2) tmem_alloc_2cta<Cfg::TMEM_COLS>(tmem_ptr_smem);
    else tmem_alloc<Cfg::TMEM_COLS>(tmem_ptr_smem);
  }
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (CTAS == 2) cluster_sync_all();   // the peer's barriers must be initialised before anything targets them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  if (cp.mode == COMM_NONE) {
    chain_wait();
    chain_next();
  }

  if (n_comm > 0 && static_cast<int>(blockIdx.x) < n_comm) {
    // ======================= COMM_AG copy CTA: push the local row blocks to the peers over NVLink ==============
    // Push, not pull: P2P stores are posted (no NVLink round trip per request) and the data is ready by stream
    // order, so no "shard ready" handshake is needed.  The copy itself is done by the TMA engine: one thread streams
    // 32 KB chunks  local global -> smem ring (cp.async.bulk + mbarrier)  ->  peer global (cp.async.bulk store),
    // keeping the whole ring (6 x 32 KB = the GEMM pipeline's smem, idle in this CTA) in flight, instead of
    // 16-byte register round trips.  Row blocks (128 rows x K, contiguous in both buffers) are taken round-robin,
    // destination by destination in the order the peers consume them (the peer right "below" needs our rows
    // first); after a row block has fully landed the peer's arrival counter is bumped with a system-scope release.
    // WAR safety: the gathered buffers are double-buffered by call parity; a peer only finishes call n-1 after our
    // pushes of call n-1, which we issue after our call n-2 kernel ended, so nobody still reads parity (n-2).
    // `copy_rings` independent engines per copy CTA (lane 0 of the first warps), each with its own slice of the
    // (otherwise idle) pipeline smem as a 6-slot ring and its own mbarriers: one engine alone is latency bound
    // (~1.6 us per 32 KB chunk, ~20 GB/s).
    const int n_rings = cp.copy_rings > 0 ? cp.copy_rings : 1;
    if (lane == 0 && warp_idx < n_rings) {
      // 12 slots; at most LOADS_AHEAD loads (local, L2-resident source: fast) and up to NSLOT - LOADS_AHEAD stores (the
      // slow side: remote writes) are in flight
      constexpr int NSLOT = 12, LOADS_AHEAD = 3, STORES_PENDING = NSLOT - LOADS_AHEAD;
      const int ring = warp_idx;
      const uint32_t ring_bytes = static_cast<uint32_t>(NS * Cfg::STAGE_BYTES) / n_rings;
      const uint32_t CHUNK = (ring_bytes / NSLOT) & ~1023u;
      uint8_t* ring_smem = smem + ring * ring_bytes;
      uint64_t* bars = reinterpret_cast<uint64_t*>(staging) + ring * 16;   // (the epilogue staging area is idle here)
#pragma unroll
      for (int b = 0; b < NSLOT; ++b) mbar_init(&bars[b], 1);
      fence_barrier_init();
      fence_proxy_async();
      const size_t blk_bytes = static_cast<size_t>(BLOCK_M) * (ag_b ? p.N : p.K) * 2;  // 128 rows of the gathered operand
      const int n_chunks = static_cast<int>((blk_bytes + CHUNK - 1) / CHUNK);
      // destinations in the order the peers consume our rows (the rank right "below" first); with `fill_local` the
      // local gathered buffer is one more destination, served last (q / mbpr == world - 1 -> dst == rank)
      const int n_remote = (cp.world - 1 + (cp.fill_local ? 1 : 0)) * mbpr;
      auto dst_of = [&](int q) { return (cp.rank - 1 - q / mbpr + 2 * cp.world) % cp.world; };
      auto blk_of = [&](int q) { return cp.rank * mbpr + q % mbpr; };
      // write-after-read: before the first byte of this call goes into peer d's buffer, d must have retired its
      // previous call on this buffer (it read what we pushed then).  Checked once per destination.
      uint32_t dst_ok_mask = 1u << cp.rank;
      auto chunk_bytes = [&](int c) {
        const size_t off = static_cast<size_t>(c) * CHUNK;
        return static_cast<uint32_t>(blk_bytes - off < CHUNK ? blk_bytes - off : CHUNK);
      };
      auto signal = [&](uint32_t* flag) {
        // the bulk stores of the row block have completed (wait_group): order them (async proxy) before the
        // generic-proxy release that publishes the arrival
        asm volatile("fence.proxy.async.global;\n" ::: "memory");
        asm volatile("red.release.sys.global.add.u32 [%0], 1;\n" ::"l"(flag) : "memory");
      };
      // One flat stream of chunks over all row blocks of this engine: the load cursor runs up to NSLOT-1 chunks ahead
      // of the store cursor, and a finished row block is signalled two stores later (so the completion wait never
      // drains the pipe).
      const int engine = static_cast<int>(blockIdx.x) * n_rings + ring, n_engines = n_comm * n_rings;
      int q_ld = engine, c_ld = 0, q_st = engine, c_st = 0;
      uint32_t issued = 0, stored = 0, pend_at = 0;
      uint32_t* pend_flag = nullptr;
      while (q_st < n_remote) {
        while (q_ld < n_remote && issued - stored < static_cast<uint32_t>(LOADS_AHEAD)) {
          const uint32_t slot = issued % NSLOT;
          // the slot was last read by store #(issued - NSLOT); at least STORES_PENDING newer stores exist (fill bound)
          if (issued >= static_cast<uint32_t>(NSLOT)) tma_store_wait_read<STORES_PENDING>();
          const uint8_t* sp = reinterpret_cast<const uint8_t*>(cp.local_shard) +
                              static_cast<size_t>(q_ld % mbpr) * blk_bytes + static_cast<size_t>(c_ld) * CHUNK;
          const uint32_t bytes = chunk_bytes(c_ld);
          mbar_arrive_expect_tx(&bars[slot], bytes);
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                           smem_u32(ring_smem + slot * CHUNK)),
                       "l"(sp), "r"(bytes), "r"(smem_u32(&bars[slot]))
                       : "memory");
          ++issued;
          if (++c_ld == n_chunks) {
            c_ld = 0;
            q_ld += n_engines;
          }
        }
        const uint32_t slot = stored % NSLOT;
        mbar_wait(&bars[slot], (stored / NSLOT) & 1);
        const int dst = dst_of(q_st);
        if (!((dst_ok_mask >> dst) & 1u)) {
          spin_wait_ge_sys(cp.peer_done[cp.rank] + dst, call_idx, cp.timeout_ns, /*what=*/3, dst);
          dst_ok_mask |= 1u << dst;
        }
        uint8_t* dp = reinterpret_cast<uint8_t*>(cp.peer_buf[dst]) + static_cast<size_t>(blk_of(q_st)) * blk_bytes +
                      static_cast<size_t>(c_st) * CHUNK;
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dp),
                     "r"(smem_u32(ring_smem + slot * CHUNK)), "r"(chunk_bytes(c_st))
                     : "memory");
        tma_store_commit();
        ++stored;
        if (++c_st == n_chunks) {
          if (pend_flag != nullptr) {  // (tiny row blocks) the previous one is still unsignalled: complete everything
            tma_store_wait<0>();
            signal(pend_flag);
          }
          // (the local fill needs no arrival: its consumers are later kernels of this stream)
          pend_flag = dst == cp.rank ? nullptr : cp.peer_flags[dst] + blk_of(q_st);
          pend_at = stored + 6;
          c_st = 0;
          q_st += n_engines;
        }
        if (pend_flag != nullptr && stored >= pend_at) {
          tma_store_wait<6>();  // all but the six newest stores are complete -> the pending row block has landed
          signal(pend_flag);
          pend_flag = nullptr;
        }
      }
      tma_store_wait<0>();   // nothing may still read the ring (or be in flight to the local buffer) when the CTA exits
      if (pend_flag != nullptr) signal(pend_flag);
    }
  } else if (warp_idx == 0) {
    // ======================= TMA producer =======================
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      int waited_blk = -1;
      for (int tile = cta; tile < num_tiles; tile += cta_stride) {
        int split, mn;
        decode_tile(tile, mn, split);
        const int m_blk = map_m(mn / n_blocks) * CTAS + cta_rank, n_blk = mn % n_blocks;   // this CTA's 128-row block
        int grp_row = 0;                                          // grouped mode: first row of this block's matrix in B
        if (p.tile_group) {
          const int grp = p.tile_group[m_blk];
          if (grp < 0) continue;
          grp_row = grp * p.N;
        }
        // gathered A: rows of the local shard come straight from the shard's own tensor map, rows owned by a peer
        // from the gathered buffer once that peer's copy CTAs have pushed the row block (arrival counter)
        const bool a_local = cp.mode == COMM_AG && !ag_b && m_blk / mbpr == cp.rank;
        if (cp.mode == COMM_AG && !ag_b && !a_local) {
          spin_wait_ge_sys(cp.peer_flags[cp.rank] + m_blk, arrive_target, cp.timeout_ns, /*what=*/1, m_blk / mbpr);
          asm volatile("fence.proxy.async.global;\n" ::: "memory");
        }
        const CUtensorMap* map_a = a_local ? &tmap_g : &tmap_a;
        const int m_row = a_local ? (m_blk - cp.rank * mbpr) * BLOCK_M : m_blk * BLOCK_M;
        int n_row = grp_row + n_blk * BLOCK_N + cta_rank * (BLOCK_N / CTAS);   // pair: this CTA's half of the B tile
        const CUtensorMap* map_nt = &tmap_b;
        if constexpr (MULTI) {
          const int seg = segment(n_blk);
          map_nt = &cp.map[seg];
          n_row -= cp.first[seg] * BLOCK_N;
        }
        const int kb0 = split * p.k_per_split;
        const int kb1 = min(kb0 + p.k_per_split, k_blocks_total);
        for (int kb = kb0; kb < kb1; ++kb) {
          // gathered B (TN): k-block kb = token rows [64 kb, 64 kb + 64) = half of row block kb / 2
          bool b_local = false;
          if (ag_b) {
            const int blk = (kb * BLOCK_K) / BLOCK_M;
            b_local = blk / mbpr == cp.rank;
            if (!b_local && blk != waited_blk) {
              spin_wait_ge_sys(cp.peer_flags[cp.rank] + blk, arrive_target, cp.timeout_ns, /*what=*/1, blk / mbpr);
              asm volatile("fence.proxy.async.global;\n" ::: "memory");
              waited_blk = blk;
            }
          }
          mbar_wait(&empty_bar[stage], phase ^ 1);
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          const CUtensorMap* map_b = b_local ? &tmap_g : &tmap_b;
          const int k_row = b_local ? kb * BLOCK_K - cp.rank * cp.rows_per_rank : kb * BLOCK_K;
          if constexpr (CTAS == 2) {
            // both CTAs' loads complete on the LEADER's barrier: the leader arms it with the bytes of both, the peer
            // contributes its arrival remotely
            if (cta_rank == 0) mbar_arrive_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES * 2);
            else mbar_arrive_cluster(&full_bar[stage], 0);
            if constexpr (!A_MN) {
              tma_load_2d_2cta(sa, map_a, &full_bar[stage], kb * BLOCK_K, m_row);
            } else {
#pragma unroll
              for (int a = 0; a < BLOCK_M / 64; ++a)
                tma_load_2d_2cta(sa + a * (BLOCK_K * 128), &tmap_a, &full_bar[stage], m_row + a * 64, kb * BLOCK_K);
            }
            if constexpr (!B_MN) {
              tma_load_2d_2cta(sb, map_nt, &full_bar[stage], kb * BLOCK_K, n_row);
            } else {
#pragma unroll
              for (int a = 0; a < Cfg::B_COLS / 64; ++a)
                tma_load_2d_2cta(sb + a * (BLOCK_K * 128), map_b, &full_bar[stage], n_row + a * 64, k_row);
            }
            if (++stage == NS) {
              stage = 0;
              phase ^= 1;
            }
            continue;
          }
          mbar_arrive_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES);
          if constexpr (!A_MN) {
            tma_load_2d(sa, map_a, &full_bar[stage], kb * BLOCK_K, m_row);
          } else {
#pragma unroll
            for (int a = 0; a < BLOCK_M / 64; ++a)
              tma_load_2d(sa + a * (BLOCK_K * 128), &tmap_a, &full_bar[stage], m_blk * BLOCK_M + a * 64, kb * BLOCK_K);
          }
          if constexpr (!B_MN) {
            tma_load_2d(sb, &tmap_b, &full_bar[stage], kb * BLOCK_K, grp_row + n_blk * BLOCK_N);
          } else {
#pragma unroll
            for (int a = 0; a < BLOCK_N / 64; ++a)
              tma_load_2d(sb + a * (BLOCK_K * 128), map_b, &full_bar[stage], n_blk * BLOCK_N + a * 64, k_row);
          }
          if (++stage == NS) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp_idx == 1) {
    // ======================= MMA issuer =======================
    // (FP8 is a template parameter so the bf16 instantiations carry no trace of it)
    constexpr uint32_t idesc = FP8 ? make_idesc_e4m3(BLOCK_M, BLOCK_N) : make_idesc_bf16(BLOCK_M * CTAS, BLOCK_N, A_MN, B_MN);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = cta; tile < num_tiles && cta_rank == 0; tile += cta_stride) {   // (pair: the leader issues for both)
      int split, mn_unused;
      decode_tile(tile, mn_unused, split);
      if (p.tile_group && p.tile_group[mn_unused / n_blocks] < 0) continue;   // grouped mode: an empty row block
      const int kb0 = split * p.k_per_split;
      const int kb1 = min(kb0 + p.k_per_split, k_blocks_total);
      mbar_wait(&tmem_empty[acc], acc_phase ^ 1);
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + acc * BLOCK_N;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(&full_bar[stage], phase);
        tc_fence_after_sync();
        if (elect_one()) {
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
            // K-major: 8-row groups are 1024B apart (SBO), advance 32B per UMMA_K inside the swizzle row.
            // MN-major: 64-element MN atoms are BLOCK_K*128B apart (LBO), 8-k-row groups 1024B apart (SBO),
            //           advance 16 k-rows = 2048B per UMMA_K.
            const uint64_t da = A_MN ? make_smem_desc_sw128(sa + k * (UMMA_K * 128), BLOCK_K * 128, 1024)
                                     : make_smem_desc_sw128(sa + k * (UMMA_K * 2), 0, 1024);
            const uint64_t db = B_MN ? make_smem_desc_sw128(sb + k * (UMMA_K * 128), BLOCK_K * 128, 1024)
                                     : make_smem_desc_sw128(sb + k * (UMMA_K * 2), 0, 1024);
            if constexpr (FP8) umma_f8_ss(d_tmem, da, db, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            else if constexpr (CTAS == 2) umma_f16_ss_2cta(d_tmem, da, db, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            else umma_f16_ss(d_tmem, da, db, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          }
          if constexpr (CTAS == 2) {
            umma_commit_2cta(&empty_bar[stage]);                    // frees the slot in BOTH CTAs
            if (kb == kb1 - 1) umma_commit_2cta(&tmem_full[acc]);   // both CTAs' epilogues
          } else {
            umma_commit(&empty_bar[stage]);                    // smem slot reusable once these MMAs retire
            if (kb == kb1 - 1) umma_commit(&tmem_full[acc]);   // accumulator complete
          }
        }
        __syncwarp();
        if (++stage == NS) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ======================= epilogue (8 warps) =======================
    const int quad = warp_idx % 4;          // TMEM lanes [32*quad, 32*quad+32)
    const int half = (warp_idx - 2) / 4;    // column half of the tile
    constexpr int CHUNKS_PER_HALF = BLOCK_N / 64;
    int acc = 0;
    uint32_t acc_phase = 0;
    float alpha = 1.0f;
    if constexpr (FP8) alpha = *p.deq_a * *p.deq_b;       // (written by the launches before: ordinary loads behind chain_wait)
    if (cp.mode == COMM_RS) {
      // write-after-read on the owners' staging buffers: every owner must have retired its previous call on this
      // buffer set (its reduce phase read what we stored then) before the first partial tile of this call lands
      if (lane == 0) {
        for (int q = 0; q < cp.world; ++q)
          if (q != cp.rank) spin_wait_ge_sys(cp.peer_done[cp.rank] + q, call_idx, cp.timeout_ns, /*what=*/4, q);
      }
      __syncwarp();
    }
    for (int tile = cta; tile < num_tiles; tile += cta_stride) {
      int mn, split_unused;
      decode_tile(tile, mn, split_unused);
      const int m_blk = map_m(mn / n_blocks) * CTAS + cta_rank, n_blk = mn % n_blocks;   // this CTA's 128-row block
      if (p.tile_group && p.tile_group[m_blk] < 0) continue;                  // grouped mode: an empty row block
      mbar_wait(&tmem_full[acc], acc_phase);
      tc_fence_after_sync();
      const int row = m_blk * BLOCK_M + quad * 32 + lane;
      const bool row_ok = row < p.M;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + acc * BLOCK_N;
      int tile_col = n_blk * BLOCK_N, tile_cols = p.N - tile_col;        // first column of the tile in the output, columns that there are from there
      if constexpr (MULTI) {
        const int seg = segment(n_blk), local = (n_blk - cp.first[seg]) * BLOCK_N;
        tile_col = cp.col[seg] + local;
        tile_cols = cp.n[seg] - local;
      }
#pragma unroll 1
      for (int c = half * CHUNKS_PER_HALF; c < (half + 1) * CHUNKS_PER_HALF; ++c) {
        const int col0 = tile_col + c * 32;
        if (c * 32 >= tile_cols) break;  // warp-uniform
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_row + c * 32, r);
        if constexpr (EPI == EPI_BF16) {
          // ---- bf16 output: all global traffic of the chunk goes through the per-warp staging slot, so every
          // load/store instruction covers 8 rows x 64 contiguous bytes (see stg_* above).  All 32 lanes take part
          // (rows >= M hold garbage that is never stored).
          uint8_t* stg = staging + (warp_idx - 2) * 2048;
          const int slab_row0 = m_blk * BLOCK_M + quad * 32;
          const int rows_valid = p.M - slab_row0;  // <= 0: nothing of this slab exists
          const int cols_valid = tile_cols - c * 32;   // > 0, multiple of 8 (enforced on the host)
          const int sub = lane & 3, rsel = lane >> 2;
          const bool use_bias = p.bias != nullptr && cp.mode != COMM_RS;  // RS: bias added once, in the reduce phase
          const bool use_pre = p.pre_in != nullptr;
          // operands fetched while the TMEM load is in flight: bias slice (same address for the whole warp =
          // broadcast) and the pre-activation tile for the fused activation backward (coalesced, 4 lanes per row)
          uint4 bq[4], pquad[4], pq[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            bq[i] = (use_bias && i * 8 < cols_valid) ? *reinterpret_cast<const uint4*>(p.bias + col0 + i * 8) : make_uint4(0, 0, 0, 0);
          if (use_pre) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int rr = 8 * j + rsel;
              pquad[j] = (rr < rows_valid && sub * 8 < cols_valid)
                             ? *reinterpret_cast<const uint4*>(p.pre_in + static_cast<size_t>(slab_row0 + rr) * p.ldo + col0 + sub * 8)
                             : make_uint4(0, 0, 0, 0);
            }
          }
          tmem_ld_wait();
          if (use_pre) stg_quads_to_rows(stg, lane, pquad, pq);
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          if constexpr (FP8) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] *= alpha;
          }
          if (use_bias) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 a = unpack_bf16(bq[i].x), b = unpack_bf16(bq[i].y), c2 = unpack_bf16(bq[i].z), d = unpack_bf16(bq[i].w);
              v[i * 8] += a.x; v[i * 8 + 1] += a.y; v[i * 8 + 2] += b.x; v[i * 8 + 3] += b.y;
              v[i * 8 + 4] += c2.x; v[i * 8 + 5] += c2.y; v[i * 8 + 6] += d.x; v[i * 8 + 7] += d.y;
            }
          }
          if (p.pre_out != nullptr)
            stg_store_chunk(stg, lane, v, p.pre_out + static_cast<size_t>(slab_row0) * p.ldo + col0, p.ldo, rows_valid, cols_valid);
          if (use_pre) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              const uint4 q = pq[i / 8];
              const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), c2 = unpack_bf16(q.z), d = unpack_bf16(q.w);
              if (p.act == ACT_RESADD) {  // row-parallel output projection: y = x·Wᵀ + bias + residual in one pass
                v[i] += a.x; v[i + 1] += a.y; v[i + 2] += b.x; v[i + 3] += b.y;
                v[i + 4] += c2.x; v[i + 5] += c2.y; v[i + 6] += d.x; v[i + 7] += d.y;
              } else if (p.act == ACT_GELU) {  // hot case without the per-element switch
                v[i] *= gelu_grad_fast(a.x); v[i + 1] *= gelu_grad_fast(a.y);
                v[i + 2] *= gelu_grad_fast(b.x); v[i + 3] *= gelu_grad_fast(b.y);
                v[i + 4] *= gelu_grad_fast(c2.x); v[i + 5] *= gelu_grad_fast(c2.y);
                v[i + 6] *= gelu_grad_fast(d.x); v[i + 7] *= gelu_grad_fast(d.y);
              } else {
                v[i] *= act_grad(a.x, p.act); v[i + 1] *= act_grad(a.y, p.act);
                v[i + 2] *= act_grad(b.x, p.act); v[i + 3] *= act_grad(b.y, p.act);
                v[i + 4] *= act_grad(c2.x, p.act); v[i + 5] *= act_grad(c2.y, p.act);
                v[i + 6] *= act_grad(d.x, p.act); v[i + 7] *= act_grad(d.y, p.act);
              }
            }
          } else if (p.act == ACT_GELU) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = gelu_fast(v[i]);
          } else if (p.act != ACT_NONE) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = act_fwd(v[i], p.act);
          }
          __nv_bfloat16* slab = reinterpret_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(slab_row0) * p.ldo + col0;
          size_t ld = static_cast<size_t>(p.ldo);
          if (cp.mode == COMM_RS) {
            // partial tile -> this rank's OWN partial-product buffer [M, N] (peer-mapped): the epilogue runs at local
            // HBM speed; the owners pull the rows they own during their reduce phase with wide coalesced loads and the
            // whole GPU's memory-level parallelism (P2P stores of 64-byte row segments from the epilogue throttled the
            // GEMM itself)
            slab = cp.peer_buf[cp.rank] + cp.staging_parity_off + static_cast<size_t>(slab_row0) * p.N + col0;
            ld = static_cast<size_t>(p.N);
          }
          stg_store_chunk(stg, lane, v, slab, ld, rows_valid, cols_valid,
                          (p.colsum != nullptr && cp.mode != COMM_RS) ? p.colsum + col0 : nullptr);
        } else if constexpr (EPI == EPI_ATOMIC_F32) {
          // ---- accumulation into fp32 (wgrad into main_grad, split-K): the chunk goes through shared memory and one TMA reduction.
          // One instruction per 4 KB and none that waits: the 8 rows x 64 bytes of red.global.add.v4 per instruction that this took before
          // cost [2048, 22016]ᵀ x [2048, 4096] 290 us, now 280 (bf16 results 232: the difference is 540 MB more to and from HBM), [2048, 4096]ᵀ x [2048, 11008]
          // 149.6 -> 145.7, [8192, 50304]ᵀ x [8192, 1024] 582 -> 570, [8192, 1024]ᵀ x [8192, 3072] 39.7 -> 38.4.  The output ahead into L2
          // (cp.async.bulk.prefetch) makes it slower, 283 and 158 us; an evict-first policy changes nothing.
          uint8_t* stg = staging + (warp_idx - 2) * Cfg::STAGING_SLOT;
          if (lane == 0) tma_store_wait_read<0>();          // the reduction before has read the slot
          tmem_ld_wait();
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i)                       // row `lane` of the box, its 16-byte pieces where the 128-byte swizzle has them
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
          fence_proxy_async();
          __syncwarp();
          const int row0 = m_blk * BLOCK_M + quad * 32;
          if (lane == 0 && row0 < p.M) {                    // (rows and columns behind the end are left out by the map)
            tma_reduce_add_2d(&cp.map, stg, col0, row0);
            tma_store_commit();
          }
        } else {
          // ---- fp32 outputs (plain store or read-modify-write): the
          // same staging slot, 16 columns (64 B per row) at a time, so every global instruction covers 8 rows x 64
          // contiguous bytes instead of 32 rows x 16 B.
          tmem_ld_wait();
          uint8_t* stg = staging + (warp_idx - 2) * 2048;
          const int slab_row0 = m_blk * BLOCK_M + quad * 32;
          const int rows_valid = p.M - slab_row0;
          const int sub = lane & 3, rsel = lane >> 2;
          float* slab = reinterpret_cast<float*>(p.out) + static_cast<size_t>(slab_row0) * p.ldo + col0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint4 rowv[4], quadv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) rowv[i] = make_uint4(r[16 * h + 4 * i], r[16 * h + 4 * i + 1], r[16 * h + 4 * i + 2], r[16 * h + 4 * i + 3]);
            stg_rows_to_quads(stg, lane, rowv, quadv);
            const int c = 16 * h + 4 * sub;  // first of this lane's 4 columns inside the chunk
            if (col0 + c < p.N) {           // N % 8 == 0
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const int rr = 8 * j + rsel;
                if (rr < rows_valid) {
                  float* dst = slab + static_cast<size_t>(rr) * p.ldo + c;
                  float4 o4 = make_float4(__uint_as_float(quadv[j].x), __uint_as_float(quadv[j].y), __uint_as_float(quadv[j].z),
                                          __uint_as_float(quadv[j].w));
                  if (p.rmw) {
                    const float4 old = *reinterpret_cast<const float4*>(dst);
                    o4.x += old.x; o4.y += old.y; o4.z += old.z; o4.w += old.w;
                  }
                  *reinterpret_cast<float4*>(dst) = o4;
                }
              }
            }
          }
        }    // fp32 epilogues
      }      // chunk loop
      tc_fence_before_sync();
      if constexpr (CTAS == 2) {
        __syncwarp();
        if (lane == 0) {
          if (cta_rank == 0) mbar_arrive(&tmem_empty[acc]);
          else mbar_arrive_cluster(&tmem_empty[acc], 0);   // the leader's MMA thread waits for both epilogues
        }
      } else {
        mbar_arrive(&tmem_empty[acc]);
      }
      if (cp.mode == COMM_RS) {
        // all 256 epilogue threads have issued their P2P stores -> one release-increment on the owner's counter
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (threadIdx.x == 64) {
          // (release at system scope is cumulative over the stores of all 256 epilogue threads ordered before it by
          // the bar.sync above: no separate fence.sc.sys — that one drained this warp's store queue once per tile)
          const int owner = m_blk / mbpr;
          // one arrival per (source rank, column tile): world * n_blocks per row block and call
          asm volatile("red.release.sys.global.add.u32 [%0], 1;\n" ::"l"(cp.peer_flags[owner] + (m_blk % mbpr)) : "memory");
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if constexpr (EPI == EPI_ATOMIC_F32) {
      if (lane == 0) tma_store_wait<0>();
      __syncwarp();
    }
  }

  if (cp.mode == COMM_RS) {
    // ---------------- reduce phase: out[r, :] = sum_src staging[src][r, :] (+ bias) (+ residual) ----------------
    // Bandwidth bound (world + 2 streams of rows_per_rank x N bf16), one CTA per SM: every thread keeps UNR row
    // vectors x (sources + residual) 16-byte loads in flight — with one vector at a time this phase was latency bound
    // and cost more than the GEMM it follows.
    constexpr int UNR = 4;
    const int col_groups = (p.N + 255) / 256;
    const int units = mbpr * col_groups;
    auto acc_add = [](float (&a)[8], const uint4& q) {
      const float2 x = unpack_bf16(q.x), y = unpack_bf16(q.y), z = unpack_bf16(q.z), w = unpack_bf16(q.w);
      a[0] += x.x; a[1] += x.y; a[2] += y.x; a[3] += y.y; a[4] += z.x; a[5] += z.y; a[6] += w.x; a[7] += w.y;
    };
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const int lm = u / col_groups, cg = u % col_groups;
      if (threadIdx.x == 0) spin_wait_ge_sys(cp.peer_flags[cp.rank] + lm, arrive_target, cp.timeout_ns, /*what=*/2, lm);
      __syncthreads();
      const int c_lo = cg * 256;
      const int c_n = min(256, p.N - c_lo) / 8;  // vectors of 8 per row in this column group
      const int total_v = BLOCK_M * c_n;
      for (int v0 = threadIdx.x; v0 < total_v; v0 += NUM_THREADS * UNR) {
        float acc8[UNR][8];
        size_t off[UNR];
        int cc[UNR];
        bool ok[UNR];
#pragma unroll
        for (int j = 0; j < UNR; ++j) {
          const int v = v0 + j * NUM_THREADS;
          ok[j] = v < total_v;
          const int vv = ok[j] ? v : 0;
          cc[j] = c_lo + (vv % c_n) * 8;
          off[j] = static_cast<size_t>(lm * BLOCK_M + vv / c_n) * p.N + cc[j];
#pragma unroll
          for (int e = 0; e < 8; ++e) acc8[j][e] = 0.f;
        }
        uint4 q[UNR], rq[UNR], bq[UNR];
        if (cp.residual != nullptr) {
#pragma unroll
          for (int j = 0; j < UNR; ++j) rq[j] = ld_stream_u4(reinterpret_cast<const uint4*>(cp.residual + off[j]));
        }
        if (p.bias != nullptr) {
#pragma unroll
          for (int j = 0; j < UNR; ++j) bq[j] = *reinterpret_cast<const uint4*>(p.bias + cc[j]);
        }
        for (int s0 = 0; s0 < cp.world; ++s0) {
          // every rank's partial product of MY rows (peers over NVLink, starting with the next rank so that the ranks
          // do not all pull from the same peer at the same time)
          const int src = (cp.rank + 1 + s0) % cp.world;
          const __nv_bfloat16* sp = cp.peer_buf[src] + cp.staging_parity_off + static_cast<size_t>(cp.rank) * cp.rows_per_rank * p.N;
#pragma unroll
          for (int j = 0; j < UNR; ++j) q[j] = ld_stream_u4(reinterpret_cast<const uint4*>(sp + off[j]));
#pragma unroll
          for (int j = 0; j < UNR; ++j) acc_add(acc8[j], q[j]);
        }
#pragma unroll
        for (int j = 0; j < UNR; ++j) {
          if (p.bias != nullptr) acc_add(acc8[j], bq[j]);
          if (cp.residual != nullptr) acc_add(acc8[j], rq[j]);
          if (ok[j])
            *reinterpret_cast<uint4*>(cp.rs_out + off[j]) =
                make_uint4(pack_bf16(acc8[j][0], acc8[j][1]), pack_bf16(acc8[j][2], acc8[j][3]),
                           pack_bf16(acc8[j][4], acc8[j][5]), pack_bf16(acc8[j][6], acc8[j][7]));
        }
      }
      __syncthreads();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if constexpr (CTAS == 2) cluster_sync_all();   // nobody may still target the peer's barriers / TMEM
  if (warp_idx == 1) {
    tc_fence_after_sync();
    if constexpr (CTAS == 2) tmem_dealloc_2cta<Cfg::TMEM_COLS>(tmem_base);
    else tmem_dealloc<Cfg::TMEM_COLS>(tmem_base);
  }
  if (cp.mode != COMM_NONE && threadIdx.x == 0) {
    // retire: the last CTA to get here advances the call counter and tells every peer that this rank is done reading
    // (AG: its gathered buffer, RS: its staging buffer) for call `call_idx`
    __threadfence();
    const uint32_t prev = atomicAdd(cp.state + 1, 1u);
    if (prev == gridDim.x - 1) {
      cp.state[1] = 0;
      cp.state[0] = call_idx + 1u;
      __threadfence_system();
      for (int q = 0; q < cp.world; ++q) {
        if (q == cp.rank) continue;
        asm volatile("st.release.sys.global.u32 [%0], %1;\n" ::"l"(cp.peer_done[q] + cp.rank), "r"(call_idx + 1u) : "memory");
      }
    }
  }
}

}  // namespace lb

// =================================================================================================
// host side
// =================================================================================================
namespace lb_host {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres);
    if (e == cudaSuccess && qres == cudaDriverEntryPointSuccess) fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

bool make_tmap_typed(CUtensorMap* out, CUtensorMapDataType dtype, const void* base, int rank, const uint64_t* dims,
                     const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_tiled();
  if (fn == nullptr) return false;
  // the driver entry point needs a current context: threads that have not touched the runtime yet (the autograd
  // engine's) bind the primary context once (otherwise the first call returns CUDA_ERROR_INVALID_CONTEXT — handled by
  // the retry below, but reported as an API error by compute-sanitizer)
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  cuuint64_t gdim[5];
  cuuint64_t gstride[5];
  cuuint32_t gbox[5];
  cuuint32_t estr[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    gbox[i] = box[i];
    estr[i] = 1;
    if (i > 0) gstride[i - 1] = strides_bytes[i];
  }
  CUresult r = fn(out, dtype, rank, const_cast<void*>(base), gdim, gstride, gbox, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // driver entry point called on a thread (e.g. the autograd engine's) that has not touched the runtime yet:
    // bind the primary context to this thread and retry
    cudaFree(nullptr);
    r = fn(out, dtype, rank, const_cast<void*>(base), gdim, gstride, gbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "[libai_b200] cuTensorMapEncodeTiled failed (%d): base=%p rank=%d dims=", (int)r, base, rank);
    for (int i = 0; i < rank; ++i) fprintf(stderr, "%llu ", (unsigned long long)gdim[i]);
    fprintf(stderr, "strides(B)=");
    for (int i = 0; i + 1 < rank; ++i) fprintf(stderr, "%llu ", (unsigned long long)gstride[i]);
    fprintf(stderr, "box=");
    for (int i = 0; i < rank; ++i) fprintf(stderr, "%u ", gbox[i]);
    fprintf(stderr, "\n");
  }
  return r == CUDA_SUCCESS;
}

bool make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box, CUtensorMapSwizzle swizzle) {
  return make_tmap_typed(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, rank, dims, strides_bytes, box, swizzle);
}

}  // namespace lb_host

namespace {

int g_num_sms = 0;
int num_sms() {                                   // (without a device the rules below answer for the chip they are fitted on)
  if (g_num_sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    g_num_sms = n;
  }
  return g_num_sms;
}

// operand tensor map: K-major [rows, K] -> box {64, rows_box}; MN-major [K, cols] -> box {64, 64}
bool operand_tmap(CUtensorMap* m, const void* ptr, bool mn_major, int rows_or_cols, int K, int ld, int block_mn) {
  if (!mn_major) {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)rows_or_cols};
    uint64_t strides[2] = {2, (uint64_t)ld * 2};
    uint32_t box[2] = {(uint32_t)lb::BLOCK_K, (uint32_t)block_mn};
    return lb_host::make_tmap_bf16(m, ptr, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  }
  uint64_t dims[2] = {(uint64_t)rows_or_cols, (uint64_t)K};
  uint64_t strides[2] = {2, (uint64_t)ld * 2};
  uint32_t box[2] = {64u, (uint32_t)lb::BLOCK_K};
  return lb_host::make_tmap_bf16(m, ptr, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Not where the epilogue multiplies by the derivative of the activation: [12608, 1024] x [1024, 4096] with it 138 us in order, 142 us chained (CTAs that
// start one by one take the tiles in another order, and rows of the two inputs are read twice); without it the chain is 2 to 3 us ahead.
bool chained(const lb::GemmParams& p, const lb::CommParams& cp) { return cp.mode == lb::COMM_NONE && (p.pre_in == nullptr || p.act == lb::ACT_RESADD); }

// CTA-pair (cta_group::2) variant: clusters of 2, 256 x BN tiles
template <int BN, bool AMN, bool BMN, int EPI>
cudaError_t launch_2cta(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tg, const CUtensorMap& to, const lb::GemmParams& p,
                        const lb::CommParams& cp, int grid, cudaStream_t stream) {
  using Cfg = lb::StageCfg<BN, 2, EPI == lb::EPI_ATOMIC_F32, BMN>;
  auto kern = lb::gemm_kernel<BN, AMN, BMN, EPI, false, 2>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  typename lb::GemmMore<EPI, false>::type more;
  static_cast<lb::CommParams&>(more) = cp;
  if constexpr (EPI == lb::EPI_ATOMIC_F32) more.map = to;
  if (chained(p, cp)) return lb_host::launch_chained(kern, dim3((unsigned)grid), dim3(lb::NUM_THREADS), Cfg::SMEM_BYTES, stream, 2, ta, tb, tg, p, more);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(lb::NUM_THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, ta, tb, tg, p, more);
}

template <int BN, bool AMN, bool BMN, int EPI, bool FP8 = false>
cudaError_t launch_cfg(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tg, const CUtensorMap& to, const lb::GemmParams& p,
                       const lb::CommParams& cp, int grid, cudaStream_t stream) {
  using Cfg = lb::StageCfg<BN, 1, EPI == lb::EPI_ATOMIC_F32, BMN>;
  auto kern = lb::gemm_kernel<BN, AMN, BMN, EPI, FP8>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  typename lb::GemmMore<EPI, false>::type more;
  static_cast<lb::CommParams&>(more) = cp;
  if constexpr (EPI == lb::EPI_ATOMIC_F32) more.map = to;
  if (chained(p, cp)) return lb_host::launch_chained(kern, dim3((unsigned)grid), dim3(lb::NUM_THREADS), Cfg::SMEM_BYTES, stream, 0, ta, tb, tg, p, more);
  kern<<<grid, lb::NUM_THREADS, Cfg::SMEM_BYTES, stream>>>(ta, tb, tg, p, more);
  return cudaGetLastError();
}

template <bool AMN, bool BMN, int EPI, bool FP8 = false>
cudaError_t launch_bn(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tg, const CUtensorMap& to, const lb::GemmParams& p,
                      const lb::CommParams& cp, int grid, cudaStream_t s) {
  switch (bn) {
    case 256:
      return launch_cfg<256, AMN, BMN, EPI, FP8>(ta, tb, tg, to, p, cp, grid, s);
    case 192:
      return launch_cfg<192, AMN, BMN, EPI, FP8>(ta, tb, tg, to, p, cp, grid, s);
    case 128:
      return launch_cfg<128, AMN, BMN, EPI, FP8>(ta, tb, tg, to, p, cp, grid, s);
    default:
      return launch_cfg<64, AMN, BMN, EPI, FP8>(ta, tb, tg, to, p, cp, grid, s);
  }
}

}  // namespace

// layout: 0 = NT (A[M,K], B[N,K]); 1 = NN (A[M,K], B[K,N]); 2 = TN (A[K,M], B[K,N])
// epi:    0 = bf16 store (+bias, act, optional pre-activation copy); 1 = fp32 store; 2 = fp32 atomic accumulate
// Returns 0 on success, a negative code for unsupported arguments, or a cudaError_t (> 0).
static bool wgrad_rmw() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("LIBAI_B200_WGRAD_RMW");
    v = (e != nullptr && e[0] == '1') ? 1 : 0;
  }
  return v == 1;
}

static int gemm_allow_2cta() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("LIBAI_B200_GEMM_2CTA");
    // 0: off; 1: plain GEMMs only; 2 (default): also the fused-collective GEMMs (AG->GEMM / GEMM->RS / gathered-B wgrad)
    v = (e == nullptr) ? 2 : (e[0] == '0' ? 0 : (e[0] == '1' ? 1 : 2));
  }
  return v;
}

// Time of a product with bf16 results by its tiles, in us: fixed + waves x (per wave + k-blocks x per k-block), but not below w at 6 TB/s.  Measured: 150 products each NT and NN
// (and 48 TN, below), M = 256 .. 12608, N and K = 384 .. 5120; fitted over both together without NT of 256 rows, which the few-row kernel takes, 290 in all (3 to 5 % rms per kind),
// the 192 wide pair's by layout.  A pair's tile takes half of B from L2 per SM: 256 x 192 a k-block in 0.235 us on two SMs where two single 128 x 192 tiles take 0.29.  B along rows
// comes in boxes of 64 columns, of which the 96 of a pair's half take two: 192 wide tiles are dearer there.  Single and pair, us: [8192, 768] x K = 3072 34.8 -> 30.4,
// [2560, 2048] x 2048 24.9 -> 20.9 (NN 21.8), [2048, 1024] x 4096 21.8 -> 18.1, [12608, 512] x 2048 31.3 -> 25.8.
// The numbers of the 192 and 128 wide pairs are the fit's times 1.04, so that they have to be 4 % ahead: they leave more SMs without work where tiles are few ([180, 1912] x [1912, 1712]
// 12.0 us in 54 single tiles, 13.3 in 14 of pairs).  Against one tile of columns single CTAs are kept ([5997, 2040] x [104, 2040] 13.4 against 14.7).  Beyond four waves the last one
// matters less than the traffic and power per product ([2048, 4096] x [12288, 4096] 135.8 us 256 wide in six waves, 139.7 192 wide in seven).  256 wide single tiles are for up to 128 rows
// against much of w.  Of kinds that are even the one with less to do per SM is taken (`order`: it decides 8 of 2128 sizes tried, 0.2 % apart by the estimate; [6300, 4096] x
// [4096, 1024] 45.5 us 128 wide, 44.7 256 wide).
struct TileKind {
  int bn;
  bool pair;
  double fixed, wave, block;
};
static const TileKind kTileKinds[2][7] = {
    {{256, true, 5.50, 0.78, 0.302}, {192, true, 5.22, 0.76, 0.239}, {128, true, 5.06, 0.62, 0.202}, {256, false, 4.20, 1.20, 0.360}, {192, false, 4.16, 0.87, 0.293},
     {128, false, 4.39, 0.47, 0.261}, {64, false, 3.96, 0.43, 0.237}},
    {{256, true, 5.50, 0.78, 0.302}, {192, true, 4.70, 1.25, 0.249}, {128, true, 5.06, 0.62, 0.202}, {256, false, 4.20, 1.20, 0.360}, {192, false, 4.16, 0.87, 0.293},
     {128, false, 4.39, 0.47, 0.261}, {64, false, 3.96, 0.43, 0.237}}};
static double tile_choice(int M, int N, int K, bool nn, int* bn, bool* pair) {
  const int sms = num_sms(), kb = (K + lb::BLOCK_K - 1) / lb::BLOCK_K;
  const bool pairs = M > lb::BLOCK_M && gemm_allow_2cta();
  const double w_us = (double)N * K * 2 / 6e6;
  double best = 1e30, time = 1e30;
  for (const TileKind& t : kTileKinds[nn]) {
    if ((t.bn > 64 && N <= t.bn / 2) || (t.pair ? !pairs || N <= 128 : t.bn == 256 && pairs)) continue;
    const int rows = t.pair ? 2 * lb::BLOCK_M : lb::BLOCK_M, slots = t.pair ? sms / 2 : sms;
    const int tiles = (M + rows - 1) / rows * ((N + t.bn - 1) / t.bn), waves = (tiles + slots - 1) / slots;
    if (t.pair && t.bn < 256 && waves > 4) continue;
    const double us = waves * (t.wave + kb * t.block), all = t.fixed + (us > w_us ? us : w_us), order = all + 0.06 * us;
    if (order < best - 1e-9) {
      best = order;
      time = all;
      *bn = t.bn;
      *pair = t.pair;
    }
  }
  return time;
}
extern "C" double lb_gemm_tile_us(int M, int N, int K) {
  int bn;
  bool pair;
  return tile_choice(M, N, K, false, &bn, &pair);
}

// Partitions of K for an accumulation with tiles of bn columns: persistent CTAs take work items round-robin, so the kernel lasts ceil(items / SMs) rounds of one K partition
// each; the count that minimises rounds x (k-blocks per partition + a fixed per-item cost for pipeline fill and the epilogue).  (A plain ceil(SMs / tiles)
// overshoots into a second round: 32 tiles x 5 splits = 160 items on 148 SMs took 2 x 26 k-blocks where 4 splits take 1 x 32.)
static int split_choice(long tiles, int k_blocks, int sms) {
  double best = 1e30;
  int splits = 1;
  for (int c = 1; c <= 16 && c <= k_blocks; ++c) {
    if (c > 1 && k_blocks / c < 4) break;  // keep at least 4 k-blocks per split so the pipeline fills
    const long rounds = (tiles * c + sms - 1) / sms;
    const int kps = (k_blocks + c - 1) / c;
    const double cost = (double)rounds * (kps + (c > 1 ? 6.0 : 3.0));
    if (cost < best - 1e-9) {
      best = cost;
      splits = c;
    }
  }
  return splits;
}
// Width of the pair tiles of an accumulation (weight gradients): fixed + rounds x (per round + k-blocks x per k-block) + bytes added.  Fitted over 48 products of up to
// [3072, 1024], K = 512 .. 8192 (2.5 to 5 % rms; the numbers of the narrow ones are the fit's times 1.03: they have to be 3 % ahead).  256 wide and the chosen width, us: [1152, 384] x K = 2048 9.9 -> 8.1, [1536, 384] x 2048 9.1 -> 7.4,
// [2304, 768] x 5000 19.2 -> 16.7, [1280, 1280] x 5000 19.3 -> 16.2, [1024, 1024] x 512 8.4 -> 6.8; [3072, 1024] x 8192 and larger keep 256 (the fit's bytes are up to 13 MB, and a
// MB costs all three the same: [21128, 768] x 1304 took 68 us 128 wide, 50 us 256 wide).
static int wgrad_tile_choice(int M, int N, int K, int sms) {
  static const struct { int bn; double fixed, round, block, mb; } kinds[3] = {{256, 6.56, 0.0, 0.322, 0.061}, {192, 5.25, 0.90, 0.273, 0.061}, {128, 6.10, 0.0, 0.207, 0.061}};
  const int kb = (K + lb::BLOCK_K - 1) / lb::BLOCK_K, m_blocks = (M + lb::BLOCK_M - 1) / lb::BLOCK_M;
  double best = 1e30;
  int bn = 256;
  for (const auto& t : kinds) {
    const long cols = (N + t.bn - 1) / t.bn;
    const int c = split_choice(m_blocks * cols, kb, sms), kps = (kb + c - 1) / c, splits = (kb + kps - 1) / kps;
    const long rounds = ((m_blocks + 1) / 2 * cols * splits + sms / 2 - 1) / (sms / 2);
    const double us = t.fixed + rounds * (t.round + kps * t.block) + t.mb * splits * ((double)M * N * 4e-6);
    if (us < best - 1e-9) {
      best = us;
      bn = t.bn;
    }
  }
  return bn;
}

extern "C" int lb_gemm_small_rule(int M, int N, int K, int* nt, int* ranks);
extern "C" int lb_gemm_small(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int ldw, int ldo, const void* bias, int act,
                             void* pre_out, const void* residual, int nt, int ranks, cudaStream_t s);

static int gemm_impl(const void* a, const void* b, void* out, int M, int N, int K, int lda, int ldb, int ldo, int layout,
                     int epi, const void* bias, int act, void* pre_out, const void* pre_in, int force_bn,
                     int force_splits, const lb::CommParams& cp_in, cudaStream_t stream, const float* deq_a = nullptr,
                     const float* deq_b = nullptr, float* colsum = nullptr, const int* tile_group = nullptr, int groups = 1) {
  lb::CommParams cp = cp_in;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (tile_group && (layout != 0 || epi == 2 || cp_in.mode != lb::COMM_NONE || deq_a || groups < 1)) return -8;
  if ((lda % 8) || (ldb % 8) || (N % 8) || (ldo % 4)) return -1;
  if (layout == 0 && epi == 0 && cp.mode == lb::COMM_NONE && deq_a == nullptr && !tile_group && colsum == nullptr && force_bn == 0 &&
      force_splits == 0 && (pre_in == nullptr || act == lb::ACT_RESADD)) {
    int nt = 0, ranks = 0;      // few rows: w is streamed by clusters of CTAs (gemm_small_sm100.cu)
    if (lb_gemm_small_rule(M, N, K, &nt, &ranks)) {
      const int rc = lb_gemm_small(a, b, out, M, N, K, lda, ldb, ldo, bias, act, pre_out, pre_in, nt, ranks, stream);
      if (rc != -1) return rc;
    }
  }
  if (epi == 0 && ((reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(pre_in) | reinterpret_cast<uintptr_t>(pre_out)) & 15)) return -8;   // vectors of the bf16 epilogue
  const bool a_mn = (layout == 2);
  const bool b_mn = (layout != 0);
  const int sms = num_sms();
  const int m_blocks = (M + lb::BLOCK_M - 1) / lb::BLOCK_M;
  // ---- tiles: a CTA pair's 256 x bn or one CTA's 128 x bn
  const bool pairs_ok = gemm_allow_2cta() && M > lb::BLOCK_M && deq_a == nullptr && !tile_group;
  const bool plain = cp.mode == lb::COMM_NONE && deq_a == nullptr && !tile_group;
  int bn = force_bn;
  bool pair = force_bn == 256;
  const int forced = force_bn < 0 ? -force_bn : force_bn;
  if (force_bn != 0 && forced != 256 && forced != 192 && forced != 128 && force_bn != 64) return -1;
  if (force_bn < 0) {                       // (timing: a pair's tile of that width)
    bn = forced;
    pair = true;
  } else if (force_bn == 0 && epi == 2) {
    // split-K fills the machine for the accumulate (wgrad) epilogue: the widest tile that fits N, on pairs the width that is estimated best
    bn = N >= 192 ? 256 : (N >= 96 ? 128 : 64);
    const bool narrow_pairs = plain && pairs_ok && layout == 2 && N >= 96 && !wgrad_rmw();       // (read-modify-write: 256 wide only)
    if (narrow_pairs) bn = wgrad_tile_choice(M, N, K, sms);
    pair = bn == 256 || narrow_pairs;
  } else if (force_bn == 0 && plain && epi == 0 && layout != 2) {
    tile_choice(M, N, K, layout == 1, &bn, &pair);
  } else if (force_bn == 0) {
    // collectives, fp8, groups, fp32 results: fewest waves, ties -> wider tile (less smem traffic per flop)
    double best = 1e30;
    const int cands[4] = {256, 192, 128, 64};
    for (int c : cands) {
      if (c > 64 && N <= c / 2) continue;
      long tiles = (long)m_blocks * ((N + c - 1) / c);
      long waves = (tiles + sms - 1) / sms;
      // cost ~ waves * per-tile time (proportional to c, narrower tiles pay more shared-memory traffic per
      // flop, plus a fixed prologue/epilogue overhead per tile)
      double eff = c == 256 ? 1.0 : (c == 192 ? 1.03 : (c == 128 ? 1.08 : 1.2));
      if (c == 256 && plain && pairs_ok) {
        // 256-wide tiles run on CTA pairs (256 x 256 per pair, half the B traffic per SM): measured ~12 % faster per
        // tile row, scheduled over sms / 2 pairs
        tiles = (long)((m_blocks + 1) / 2) * ((N + c - 1) / c);
        waves = (tiles + sms / 2 - 1) / (sms / 2);
        eff = 0.89;
      }
      const double cost = (double)waves * (c * eff + 24.0);
      if (cost < best - 1e-9) {
        best = cost;
        bn = c;
        pair = c == 256;
      }
    }
  }
  const int n_blocks = (N + bn - 1) / bn;
  const int k_blocks = (K + lb::BLOCK_K - 1) / lb::BLOCK_K;
  int splits = 1;
  if (epi == 2) {
    splits = force_splits;
    const bool ag_b = cp.mode == lb::COMM_AG && cp.gathered_is_b;
    if (ag_b) {
      // gathered-B wgrad: the partitions must not straddle a shard boundary and their number must be a multiple of the
      // group size (the kernel starts every rank on the partitions of its own shard)
      const int kb_per_rank = cp.rows_per_rank / lb::BLOCK_K;
      const long tiles = (long)m_blocks * n_blocks;
      const int gemm_ctas = sms - cp.n_comm;
      double best = 1e30;
      splits = cp.world;
      for (int j = 1; j <= 16 && j <= kb_per_rank; ++j) {
        if (kb_per_rank % j) continue;
        if (j > 1 && kb_per_rank / j < 4) break;
        const int c = cp.world * j;
        const long rounds = (tiles * c + gemm_ctas - 1) / gemm_ctas;
        const double cost = (double)rounds * (kb_per_rank / j + 6.0);
        if (cost < best - 1e-9) {
          best = cost;
          splits = c;
        }
      }
    } else if (splits <= 0) {
      splits = split_choice((long)m_blocks * n_blocks, k_blocks, sms);
    }
    if (splits > k_blocks) splits = k_blocks;
  }
  lb::GemmParams p;
  p.M = M;
  p.N = N;
  p.K = K;
  p.k_splits = splits;
  p.k_per_split = (k_blocks + splits - 1) / splits;
  p.k_splits = (k_blocks + p.k_per_split - 1) / p.k_per_split;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.rmw = 0;
  if (epi == 2 && p.k_splits == 1 && wgrad_rmw()) {
    // a single K partition owns the whole tile: accumulate with a plain read-modify-write instead of L2 atomics.
    // Off by default: a reduction is not waited for, while the read of the old
    // tile sits exposed at the end of a one-tile-per-CTA GEMM (4096x1024x8192
    // 2-way split with reductions 50 us vs single partition with rmw 63 us; [22016,4096] 280 vs 367).  LIBAI_B200_WGRAD_RMW=1 restores it.
    epi = 1;
    p.rmw = 1;
  }
  p.act = act;
  p.out = out;
  p.pre_out = reinterpret_cast<__nv_bfloat16*>(pre_out);
  p.pre_in = reinterpret_cast<const __nv_bfloat16*>(pre_in);
  p.ldo = ldo;
  p.colsum = (epi == 0) ? colsum : nullptr;
  p.fp8 = (deq_a != nullptr && deq_b != nullptr) ? 1 : 0;
  p.deq_a = deq_a;
  p.deq_b = deq_b;
  p.tile_group = tile_group;

  // CTA pairs (cta_group::2, 256 rows x bn columns, each CTA stages half of B).  LIBAI_B200_GEMM_2CTA=0 keeps everything on single-CTA tiles.
  // (fused collectives: shards must hold whole 256-row pair tiles and the copy CTAs come in pairs)
  const bool comm_ok = cp.mode == lb::COMM_NONE ||
                       (cp.rows_per_rank % (2 * lb::BLOCK_M) == 0 && cp.n_comm % 2 == 0 && gemm_allow_2cta() >= 2);
  const bool two_cta = pair && pairs_ok && comm_ok;
  // (there is no kernel of narrower pairs for the others, and the boxes of another width would bring fewer bytes than it waits for)
  if (two_cta && bn != 256 && !(layout == 2 ? epi == 2 : epi == 0)) return -1;
  // Order of the tiles.  Row by row, the CTAs in flight hold one or two row blocks of A and up to 74 column blocks of B: a B that does
  // not stay in L2 beside the output is read from HBM again for (nearly) every row block (LM head [8192, 1024] x [50304, 1024]: 32 x
  // 103 MB).  In bands of G row blocks they hold G of A and C / G of B, the least bytes at equal sides: G = sqrt(C * columns / rows of a
  // tile).  Measured, row by row -> bands: LM head 693 -> 585 us, its input gradient 641 -> 575; [2048, 4096] x [12288, 4096] 163 -> 143.
  // The line lies at a B of 48 MB: from 8 to 32 MB the orders are within 1 % of each other for 2048 rows and bands 1 to 3 % behind for 8192
  // ([8192, 1024] x [12288, 1024], 24 MB: 150 against 155 us; x [16384, 1024] 215 against 218); at 48 MB 81 against 78 us (2048 rows) and
  // equal (8192); at 64 MB 109 against 100 and 430 against 396 us.  The fp32 accumulate epilogue writes long rows faster than bands
  // ([2048, 4096]ᵀ x [2048, 11008] 152 against 158 us) and keeps the old order.
  p.group_m = 1;
  if (cp.mode == lb::COMM_NONE && !tile_group && epi == 0 && (long)N * K * 2 >= (48L << 20)) {
    const double in_flight = two_cta ? sms / 2 : sms, side = (double)bn / (two_cta ? 2 * lb::BLOCK_M : lb::BLOCK_M);
    p.group_m = (int)(std::sqrt(in_flight * side) + 0.5);
  }
  CUtensorMap ta, tb, tg, to;
  if (!operand_tmap(&ta, a, a_mn, M, K, lda, lb::BLOCK_M)) return -2;
  if (!operand_tmap(&tb, b, b_mn, tile_group ? N * groups : N, K, ldb, two_cta ? bn / 2 : bn)) return -2;
  tg = to = ta;
  if (epi == 2) {
    if (reinterpret_cast<uintptr_t>(out) & 15) return -8;
    const uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, strides[2] = {4, (uint64_t)ldo * 4};
    const uint32_t box[2] = {32u, 32u};
    if (!lb_host::make_tmap_typed(&to, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -2;
  }
  if (cp.mode == lb::COMM_AG) {
    // tensor map of the local shard of the gathered operand: [rows_per_rank, K] rows of A (NT/NN), or rows_per_rank
    // reduction rows of B (TN)
    const bool ok = cp.gathered_is_b ? operand_tmap(&tg, cp.local_shard, true, N, cp.rows_per_rank, ldb, bn)
                                     : operand_tmap(&tg, cp.local_shard, false, cp.rows_per_rank, K, lda, lb::BLOCK_M);
    if (!ok) return -2;
    cp.arrivals = 1;
  } else if (cp.mode == lb::COMM_RS) {
    cp.arrivals = (uint32_t)(cp.world * n_blocks);
  }
  long num_tiles = (long)m_blocks * n_blocks * p.k_splits;
  int grid = (int)(num_tiles < sms ? num_tiles : sms);
  if (two_cta) {
    num_tiles = (long)((m_blocks + 1) / 2) * n_blocks * p.k_splits;   // 256-row tiles, one per CTA pair
    const long pairs = (sms - (cp.mode == lb::COMM_AG ? cp.n_comm : 0)) / 2;
    grid = 2 * (int)(num_tiles < pairs ? num_tiles : pairs);
  }
  if (cp.mode == lb::COMM_AG) {
    if (two_cta) {
      grid += cp.n_comm;
    } else {
      const long g = num_tiles < (sms - cp.n_comm) ? num_tiles : (sms - cp.n_comm);
      grid = (int)g + cp.n_comm;
    }
  }

  cudaError_t e;
  if (two_cta) {
    if (epi == 0 && layout != 2 && bn != 256) {
      if (layout == 0) e = bn == 192 ? launch_2cta<192, false, false, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream)
                                     : launch_2cta<128, false, false, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream);
      else e = bn == 192 ? launch_2cta<192, false, true, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream)
                         : launch_2cta<128, false, true, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream);
    } else if (layout == 0) {
      if (epi == 0) e = launch_2cta<256, false, false, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream);
      else if (epi == 1) e = launch_2cta<256, false, false, lb::EPI_F32>(ta, tb, tg, to, p, cp, grid, stream);
      else e = launch_2cta<256, false, false, lb::EPI_ATOMIC_F32>(ta, tb, tg, to, p, cp, grid, stream);
    } else if (layout == 1) {
      if (epi == 0) e = launch_2cta<256, false, true, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream);
      else if (epi == 1) e = launch_2cta<256, false, true, lb::EPI_F32>(ta, tb, tg, to, p, cp, grid, stream);
      else e = launch_2cta<256, false, true, lb::EPI_ATOMIC_F32>(ta, tb, tg, to, p, cp, grid, stream);
    } else {
      if (epi == 0) e = launch_2cta<256, true, true, lb::EPI_BF16>(ta, tb, tg, to, p, cp, grid, stream);
      else if (epi == 1) e = launch_2cta<256, true, true, lb::EPI_F32>(ta, tb, tg, to, p, cp, grid, stream);
      else if (bn == 192) e = launch_2cta<192, true, true, lb::EPI_ATOMIC_F32>(ta, tb, tg, to, p, cp, grid, stream);
      else if (bn == 128) e = launch_2cta<128, true, true, lb::EPI_ATOMIC_F32>(ta, tb, tg, to, p, cp, grid, stream);
      else e = launch_2cta<256, true, true, lb::EPI_ATOMIC_F32>(ta, tb, tg, to, p, cp, grid, stream);
    }
    return (int)e;
  }
  if (p.fp8) {
    if (layout != 0 || epi != 0 || cp.mode != lb::COMM_NONE) return -7;
    e = launch_bn<false, false, lb::EPI_BF16, true>(bn, ta, tb, tg, to, p, cp, grid, stream);
  } else if (layout == 0) {
    if (epi == 0) e = launch_bn<false, false, lb::EPI_BF16>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else if (epi == 1) e = launch_bn<false, false, lb::EPI_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else e = launch_bn<false, false, lb::EPI_ATOMIC_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
  } else if (layout == 1) {
    if (epi == 0) e = launch_bn<false, true, lb::EPI_BF16>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else if (epi == 1) e = launch_bn<false, true, lb::EPI_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else e = launch_bn<false, true, lb::EPI_ATOMIC_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
  } else {
    if (epi == 0) e = launch_bn<true, true, lb::EPI_BF16>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else if (epi == 1) e = launch_bn<true, true, lb::EPI_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
    else e = launch_bn<true, true, lb::EPI_ATOMIC_F32>(bn, ta, tb, tg, to, p, cp, grid, stream);
  }
  return (int)e;
}

template <int BN>
static cudaError_t launch_multi(const CUtensorMap& ta, const lb::GemmParams& p, const lb::GemmMultiB& mb, int grid, cudaStream_t stream) {
  using Cfg = lb::StageCfg<BN, 2, false, false>;
  auto kern = lb::gemm_kernel<BN, false, false, lb::EPI_BF16, false, 2, true>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  return lb_host::launch_chained(kern, dim3((unsigned)grid), dim3(lb::NUM_THREADS), Cfg::SMEM_BYTES, stream, 2, ta, ta, ta, p, mb);
}
// x [M, K] against `count` matrices w[i] [n[i], K] at once: out [M, ldo], the results one after the other.  One launch and one last wave in place of a launch each, and
// the first of them put together by a copy: a mixer's projections (1024 + 1024 + 2048, 16, 16 and 2048 columns, K = 2048) of 1600 rows 68.4 -> 37.9 us, 300 rows 46.1 -> 15.2,
// 16 rows 30.8 -> 16.3, 1 row 28.8 -> 21.0, 8192 rows 171.7 -> 144.9; K = 1024 with half the columns, 1 row 18.5 -> 9.9 and 8192 rows 72.1 -> 43.9.  Bounded by the tensor
// cores from some 1000 rows (1600 rows: 1.07 PFLOP/s), below by the chain of k-blocks of one tile.  A matrix's last tile is not shared with the next one's first: a tile of its
// own for 16 columns costs less than moving the matrix.  -1: not of a form that this takes.
extern "C" int lb_gemm_multi(const void* x, const void* const* w, const int* n, int count, void* out, int M, int K, int ldx, int ldo, cudaStream_t stream) {
  if (M <= 0 || K <= 0 || count < 1 || count > lb::GEMM_MAX_B || !gemm_allow_2cta() || K % 8 || ldx % 8 || ldo % 8 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -1;
  int total = 0;
  for (int i = 0; i < count; ++i) {
    if (n[i] <= 0 || n[i] % 8 || (reinterpret_cast<uintptr_t>(w[i]) & 15)) return -1;
    total += n[i];
  }
  if (total > ldo) return -1;
  const int pairs = num_sms() / 2, kb = (K + lb::BLOCK_K - 1) / lb::BLOCK_K, m_blocks = (M + 2 * lb::BLOCK_M - 1) / (2 * lb::BLOCK_M);
  int bn = 256;
  double best = 1e30;
  for (int i = 0; i < 3; ++i) {                  // the pair tiles of tile_choice
    const TileKind& t = kTileKinds[0][i];
    long tiles = 0;
    for (int j = 0; j < count; ++j) tiles += (n[j] + t.bn - 1) / t.bn;
    const long waves = (tiles * m_blocks + pairs - 1) / pairs;
    if (t.bn < 256 && waves > 4) continue;
    const double us = t.fixed + (double)waves * (t.wave + kb * t.block);
    if (us < best - 1e-9) {
      best = us;
      bn = t.bn;
    }
  }
  lb::GemmParams p{};
  p.M = M;
  p.N = total;
  p.K = K;
  p.k_splits = 1;
  p.k_per_split = kb;
  p.group_m = (long)total * K * 2 >= (48L << 20) ? (int)(std::sqrt(pairs * (bn / (2.0 * lb::BLOCK_M))) + 0.5) : 1;   // as for one matrix
  p.out = out;
  p.ldo = ldo;
  lb::GemmMultiB mb{};
  mb.count = count;
  CUtensorMap ta;
  if (!operand_tmap(&ta, x, false, M, K, ldx, lb::BLOCK_M)) return -2;
  for (int i = 0, col = 0; i < count; ++i) {
    if (!operand_tmap(&mb.map[i], w[i], false, n[i], K, K, bn / 2)) return -2;
    mb.n[i] = n[i];
    mb.col[i] = col;
    mb.first[i + 1] = mb.first[i] + (n[i] + bn - 1) / bn;
    col += n[i];
  }
  const long tiles = (long)m_blocks * mb.first[count];
  const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
  return (int)(bn == 256 ? launch_multi<256>(ta, p, mb, grid, stream) : bn == 192 ? launch_multi<192>(ta, p, mb, grid, stream) : launch_multi<128>(ta, p, mb, grid, stream));
}

extern "C" int lb_gemm_bf16(const void* a, const void* b, void* out, int M, int N, int K, int lda, int ldb, int ldo,
                            int layout, int epi, const void* bias, int act, void* pre_out, int force_bn,
                            int force_splits, cudaStream_t stream) {
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  return gemm_impl(a, b, out, M, N, K, lda, ldb, ldo, layout, epi, bias, act, pre_out, nullptr, force_bn, force_splits, cp,
                   stream);
}

// Grouped NT GEMM: out[M, N] rows of 128-row block m = a rows x (b[tile_group[m]] [N, K])ᵀ; blocks with tile_group < 0 are skipped.
extern "C" int lb_gemm_bf16_grouped(const void* a, const void* b, void* out, int M, int N, int K, int lda, int ldo, int epi,
                                    const int* tile_group, int groups, cudaStream_t stream) {
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  if (M % lb::BLOCK_M || !tile_group) return -8;
  return gemm_impl(a, b, out, M, N, K, lda, K, ldo, 0, epi, nullptr, 0, nullptr, nullptr, 0, 0, cp, stream, nullptr, nullptr, nullptr,
                   tile_group, groups);
}

// fp8 forward GEMM: y[M,N] (bf16) = act((xq[M,K] · wq[N,K]ᵀ) * deq_x * deq_w + bias); xq / wq hold E4M3 bytes, K % 16 == 0.
// The operands are handed to the kernel as bf16 matrices with K/2 columns (identical bytes, see GemmParams::fp8).
// With `residual` ([M, N] bf16) the epilogue is bias + residual add instead of an activation.
extern "C" int lb_gemm_fp8(const void* xq, const void* wq, void* out, int M, int N, int K, const void* bias, int act,
                           void* pre_out, const void* residual, const float* deq_x, const float* deq_w,
                           cudaStream_t stream) {
  if ((K % 16) != 0 || deq_x == nullptr || deq_w == nullptr) return -7;
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  if (residual != nullptr) {
    act = lb::ACT_RESADD;
    pre_out = nullptr;
  }
  return gemm_impl(xq, wq, out, M, N, K / 2, K / 2, K / 2, N, 0, 0, bias, act, pre_out, residual, 0, 0, cp, stream, deq_x,
                   deq_w);
}

// dgrad fused with the activation backward: out[M,N] = (A·B) * act'(pre_in[M,N])   (bf16 output, ldo = row stride
// of both `out` and `pre_in`)
// `colsum` (optional, fp32 [N], 16-byte aligned): += column sums of `out` = the bias gradient of the layer that produced
// `pre_in`, accumulated by the epilogue (no separate pass over the [M, N] tensor).
extern "C" int lb_gemm_bf16_actgrad(const void* a, const void* b, void* out, int M, int N, int K, int lda, int ldb,
                                    int ldo, int layout, int act, const void* pre_in, float* colsum, cudaStream_t stream) {
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  if (colsum != nullptr && (reinterpret_cast<uintptr_t>(colsum) & 15)) return -8;
  return gemm_impl(a, b, out, M, N, K, lda, ldb, ldo, layout, 0, nullptr, act, nullptr, pre_in, 0, 0, cp, stream, nullptr,
                   nullptr, colsum);
}

// y[M,N] = x[M,K]·w[N,K]ᵀ + bias[N] + residual[M,N]   (bias+residual add of the transformer block in the GEMM epilogue;
// the residual tile is fetched coalesced through the epilogue staging slot while the TMEM load is in flight)
extern "C" int lb_gemm_bf16_bias_residual(const void* x, const void* w, void* out, int M, int N, int K, int lda, int ldb,
                                          const void* bias, const void* residual, cudaStream_t stream) {
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  return gemm_impl(x, w, out, M, N, K, lda, ldb, N, 0, 0, bias, lb::ACT_RESADD, nullptr, residual, 0, 0, cp, stream);
}

// Tensor-parallel fused collective GEMMs.
//   mode 1 (AG->GEMM), layout 0/1: a = local gathered buffer [M, K] (remote rows are pushed into it by the peers' copy
//           CTAs), local_shard = this rank's [M/world, K] rows, out [M, N] bf16 (+bias, +act with pre-activation copy,
//           or x act'(pre_in) for a dgrad fused with the activation backward, + column sums for the bias gradient)
//   mode 1, layout 2 (gathered-B wgrad): a = dy [T, M] (T tokens), b = local gathered buffer [T, N], local_shard =
//           this rank's [T/world, N] rows of it, out [M, N] fp32: epi 2 accumulates, epi 1 stores
//   mode 2 (GEMM->RS), layout 0/1: a = local [M, K_shard]; partial tiles go to the owners' staging buffers;
//           rs_out [M/world, N] = sum over ranks (+bias +residual)
static unsigned long long spin_timeout_ns() {
  static unsigned long long v = ~0ull;
  if (v == ~0ull) {
    const char* e = getenv("LIBAI_B200_SPIN_TIMEOUT_MS");
    v = (e != nullptr && atoll(e) > 0) ? (unsigned long long)atoll(e) * 1000000ull : 0ull;
  }
  return v;
}

extern "C" int lb_gemm_bf16_comm(const void* a, const void* b, void* out, int M, int N, int K, int layout, int epi,
                                 const void* bias, int act, void* pre_out, const void* pre_in, float* colsum, int mode,
                                 int world, int rank, const long* peer_buf, const long* peer_flags, const long* peer_done,
                                 void* state, const void* local_shard, int fill_local, const void* residual, void* rs_out,
                                 long staging_parity_off, int n_comm, cudaStream_t stream) {
  if (world > 8 || world < 2 || state == nullptr) return -4;
  const int gathered_rows = (mode == 1 && layout == 2) ? K : M;   // extent of the dimension that is split over ranks
  if (gathered_rows % (lb::BLOCK_M * world) != 0) return -4;
  if (layout < 0 || layout > 2 || (layout == 2 && mode != 1)) return -6;
  lb::CommParams cp;
  memset(&cp, 0, sizeof(cp));
  cp.mode = mode;
  cp.world = world;
  cp.rank = rank;
  cp.rows_per_rank = gathered_rows / world;
  cp.n_comm = mode == 1 ? n_comm : 0;
  cp.gathered_is_b = (mode == 1 && layout == 2) ? 1 : 0;
  cp.fill_local = fill_local;
  cp.state = reinterpret_cast<uint32_t*>(state);
  for (int i = 0; i < world; ++i) {
    cp.peer_buf[i] = reinterpret_cast<__nv_bfloat16*>(peer_buf[i]);
    cp.peer_flags[i] = reinterpret_cast<uint32_t*>(peer_flags[i]);
    cp.peer_done[i] = reinterpret_cast<uint32_t*>(peer_done[i]);
  }
  cp.local_shard = reinterpret_cast<const __nv_bfloat16*>(local_shard);
  cp.residual = reinterpret_cast<const __nv_bfloat16*>(residual);
  cp.rs_out = reinterpret_cast<__nv_bfloat16*>(rs_out);
  cp.staging_parity_off = staging_parity_off;
  cp.timeout_ns = spin_timeout_ns();
  {
    static int rings = -1;
    if (rings < 0) {
      const char* e = getenv("LIBAI_B200_COPY_RINGS");
      rings = (e != nullptr && atoi(e) >= 1 && atoi(e) <= 8) ? atoi(e) : 1;   // measured: more engines do not help
    }
    cp.copy_rings = rings;
  }
  // timing experiments only (results are WRONG with these set): keep the handshake but take the NVLink payload out
  {
    static int dbg = -1;
    if (dbg < 0) {
      const char* e = getenv("LIBAI_B200_DEBUG_COMM_NO_PAYLOAD");
      dbg = (e != nullptr && e[0] == '1') ? 1 : 0;
    }
    if (dbg == 1) {
      for (int i = 0; i < world; ++i) cp.peer_buf[i] = cp.peer_buf[rank];   // AG pushes / RS partial tiles stay local
    }
  }
  if (mode == 1 && local_shard == nullptr) return -4;
  if (colsum != nullptr && (reinterpret_cast<uintptr_t>(colsum) & 15)) return -8;
  int lda, ldb, ldo;
  if (layout == 0) { lda = K; ldb = K; ldo = N; }
  else if (layout == 1) { lda = K; ldb = N; ldo = N; }
  else { lda = M; ldb = N; ldo = N; }
  if (mode == 2) epi = 0;
  // the RS epilogue writes into the staging buffers; `out` is unused there (pass any valid pointer)
  return gemm_impl(a, b, mode == 2 ? rs_out : out, M, N, K, lda, ldb, ldo, layout, epi, bias, act, pre_out, pre_in, 0,
                   mode == 1 && layout == 2 ? 0 : 1, cp, stream, nullptr, nullptr, colsum);
}

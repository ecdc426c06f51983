// Fused LayerNorm / RMSNorm forward + backward for sm_100a (bandwidth-bound: one warp per row,
// 128-bit vector accesses, statistics in fp32, row cached in registers between the passes).
// Replaces flow._C.layer_norm_affine / rms_norm (reference libai/layers/layer_norm.py:78-131).
//
//   fwd : y = (x - mean) * rstd * gamma + beta          (rms: y = x * rstd * gamma, mean := 0)
//   bwd : dx = rstd * (g·γ - mean_h(g·γ) - x̂ · mean_h(g·γ·x̂))   (rms: no mean_h(g·γ) term)
//         dγ = Σ_rows g·x̂ ,  dβ = Σ_rows g        (two-stage: per-CTA partials, then column reduce)
#include "common.cuh"
#include <atomic>
#include <type_traits>

namespace lb {

constexpr int NORM_WARPS = 8;

template <typename T>
struct Vec8;
template <>
struct Vec8<__nv_bfloat16> {
  static LB_DEVICE void load(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), c = unpack_bf16(q.z), d = unpack_bf16(q.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
  static LB_DEVICE void store(__nv_bfloat16* p, const float (&v)[8]) {
    *reinterpret_cast<uint4*>(p) =
        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  }
};
template <>
struct Vec8<float> {
  static LB_DEVICE void load(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  static LB_DEVICE void store(float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
};

// H = VPL * 256 elements per row (each lane owns VPL vectors of 8, interleaved for coalescing); with TAIL any H % 8 == 0
// in (256 (VPL - 1), 256 VPL): the lanes behind the row's end hold zeros.  h = 384 and 192 (the shipped GPT / T5 recipes)
// took the one-element-per-lane kernel below before: forward 3.4 -> 2.7 us on [200, 384], backward 27 -> 6.6 us on [2048, 384].
// Whole multiples of 256 keep a compile-time width (the backward of [8192, 1024] is 8 % slower with a run-time one).
template <typename T, typename W, int VPL, bool RMS, bool TAIL>
__global__ void __launch_bounds__(NORM_WARPS * 32)
norm_fwd_kernel(const T* __restrict__ x, const W* __restrict__ gamma, const W* __restrict__ beta, T* __restrict__ y,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, float eps, int h_tail) {
  chain_wait(x, gamma, beta);
  chain_next();
  const int H = TAIL ? h_tail : VPL * 256;
  const float inv_h = 1.0f / static_cast<float>(H);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int row = blockIdx.x * NORM_WARPS + warp; row < rows; row += gridDim.x * NORM_WARPS) {
    const T* xr = x + static_cast<size_t>(row) * H;
    float v[VPL][8];
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (TAIL && (i * 32 + lane) * 8 >= H) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
        continue;
      }
      Vec8<T>::load(xr + (i * 32 + lane) * 8, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += v[i][j];
    }
    float mean = 0.f;
    if (!RMS) mean = warp_sum(s) * inv_h;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (TAIL && (i * 32 + lane) * 8 >= H) continue;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = v[i][j] - mean;
        sq += d * d;
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) * inv_h + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    T* yr = y + static_cast<size_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (TAIL && (i * 32 + lane) * 8 >= H) continue;
      float g[8], b[8], o[8];
      Vec8<W>::load(gamma + (i * 32 + lane) * 8, g);
      if (beta != nullptr) Vec8<W>::load(beta + (i * 32 + lane) * 8, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = (v[i][j] - mean) * rstd * g[j];
        if (beta != nullptr) o[j] += b[j];
      }
      Vec8<T>::store(yr + (i * 32 + lane) * 8, o);
    }
  }
}

template <typename T, typename W, int VPL, bool RMS>
__global__ void __launch_bounds__(NORM_WARPS * 32)
norm_bwd_kernel(const T* __restrict__ gy, const T* __restrict__ x, const W* __restrict__ gamma,
                const float* __restrict__ mean_in, const float* __restrict__ rstd_in, T* __restrict__ gx,
                float* __restrict__ part_dgamma, float* __restrict__ part_dbeta, int rows,
                const T* __restrict__ gadd /* optional [rows, H]: gradient of the residual path, added to gx */) {
  chain_next();
  constexpr int H = VPL * 256;
  __shared__ float red[NORM_WARPS][32 * 8 + 8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  float dg[VPL][8], db[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dg[i][j] = db[i][j] = 0.f;
  float gam[VPL][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i) Vec8<W>::load(gamma + (i * 32 + lane) * 8, gam[i]);

  for (int row = blockIdx.x * NORM_WARPS + warp; row < rows; row += gridDim.x * NORM_WARPS) {
    const float mean = RMS ? 0.f : mean_in[row];
    const float rstd = rstd_in[row];
    const T* xr = x + static_cast<size_t>(row) * H;
    const T* gr = gy + static_cast<size_t>(row) * H;
    float xh[VPL][8], gw[VPL][8];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      float xv[8], gv[8];
      Vec8<T>::load(xr + (i * 32 + lane) * 8, xv);
      Vec8<T>::load(gr + (i * 32 + lane) * 8, gv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[i][j] = (xv[j] - mean) * rstd;
        gw[i][j] = gv[j] * gam[i][j];
        s1 += gw[i][j];
        s2 += gw[i][j] * xh[i][j];
        dg[i][j] += gv[j] * xh[i][j];
        db[i][j] += gv[j];
      }
    }
    s1 = RMS ? 0.f : warp_sum(s1) * (1.0f / H);
    s2 = warp_sum(s2) * (1.0f / H);
    T* gxr = gx + static_cast<size_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rstd * (gw[i][j] - s1 - xh[i][j] * s2);
      if (gadd != nullptr) {  // the skip connection's gradient rides along: saves autograd's separate add kernel
        float a[8];
        Vec8<T>::load(gadd + static_cast<size_t>(row) * H + (i * 32 + lane) * 8, a);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += a[j];
      }
      Vec8<T>::store(gxr + (i * 32 + lane) * 8, o);
    }
  }
  // block-level reduction of the per-warp column partials, one vector slot at a time
  for (int i = 0; i < VPL; ++i) {
    for (int which = 0; which < (part_dbeta != nullptr ? 2 : 1); ++which) {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) red[warp][lane * 8 + j] = which == 0 ? dg[i][j] : db[i][j];
      __syncthreads();
      for (int c = threadIdx.x; c < 256; c += NORM_WARPS * 32) {
        float acc = 0.f;
#pragma unroll
        for (int w = 0; w < NORM_WARPS; ++w) acc += red[w][c];
        float* dst = (which == 0 ? part_dgamma : part_dbeta) + static_cast<size_t>(blockIdx.x) * H + i * 256 + c;
        *dst = acc;
      }
    }
  }
}

// bf16 activations up to 1024 columns: a warp per row like the kernel above (same maths, same outputs), bounded by memory.  Rows go through a ring in shared memory, three
// per warp, filled by cp.async (every lane copies what it reads itself: no barrier), so that loads are in flight while a row is worked on; x, gy and the residual's gradient in
// registers, fetched row by row, took [8192, 1024] 16.0 -> 14.3 us (floor 10.2) and [12608, 1024] 23.0 -> 19.7 (15.8).  12 warps per SM.
// SUMS: the column sums of the residual's gradient and of the result too, which are the gradients of the biases in front of and behind this norm in a block (they would read
// both tensors again: with both 14.3 and 20.5 us, without column sums of 4 to 9 us each behind it).
constexpr int NORM_BWD_WARPS = 4, NORM_BWD_STAGES = 3;
LB_DEVICE void cp_async_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

constexpr int norm_bwd_blocks(int vpl, bool sums) { return sums && vpl == 4 ? 2 : 3; }     // per SM: four column sums of 1024 columns need 190 registers
template <typename W, int VPL, bool RMS, bool TAIL, bool SUMS>
__global__ void __launch_bounds__(NORM_BWD_WARPS * 32, norm_bwd_blocks(VPL, SUMS))
norm_bwd_bf16_kernel(const __nv_bfloat16* __restrict__ gy, const __nv_bfloat16* __restrict__ x, const W* __restrict__ gamma,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ gx,
                     float* __restrict__ part_dgamma, float* __restrict__ part_dbeta, int rows,
                     const __nv_bfloat16* __restrict__ gadd, float* __restrict__ acc_dgamma, float* __restrict__ acc_dbeta,
                     float* __restrict__ sum_add, float* __restrict__ sum_out, int h_tail) {
  chain_next();
  const int H = TAIL ? h_tail : VPL * 256;       // TAIL: lanes behind the row's end neither load nor store
  const float inv_h = 1.0f / static_cast<float>(H);
  extern __shared__ uint4 norm_ring[];           // [warp][stage][x, gy, gadd][vector][lane]
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  uint4* ring = norm_ring + warp * (NORM_BWD_STAGES * 3 * VPL * 32) + lane;
  const int step = gridDim.x * NORM_BWD_WARPS;
  auto fetch = [&](int row, int stage) {
    if (row < rows) {
      const size_t base = static_cast<size_t>(row) * H;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        const int c = (i * 32 + lane) * 8;
        if (TAIL && c >= H) continue;
        uint4* at = ring + (stage * 3 * VPL + i) * 32;
        cp_async_16(at, x + base + c);
        cp_async_16(at + VPL * 32, gy + base + c);
        if (gadd != nullptr) cp_async_16(at + 2 * VPL * 32, gadd + base + c);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  float dg[VPL][8], db[VPL][8];
  [[maybe_unused]] float sa[SUMS ? VPL : 1][8], so[SUMS ? VPL : 1][8];
#pragma unroll
  for (int i = 0; i < VPL; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dg[i][j] = db[i][j] = 0.f;
      if constexpr (SUMS) sa[i][j] = so[i][j] = 0.f;
    }
  auto unpack8 = [](const uint4& q, float (&v)[8]) {
    const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), c = unpack_bf16(q.z), d = unpack_bf16(q.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  };

  int row = blockIdx.x * NORM_BWD_WARPS + warp, stage = 0;
#pragma unroll
  for (int k = 0; k < NORM_BWD_STAGES - 1; ++k) fetch(row + k * step, k);
  float mean_next = 0.f, rstd_next = 0.f;
  auto stats = [&](int r) {
    if (r < rows) {
      mean_next = RMS ? 0.f : mean_in[r];
      rstd_next = rstd_in[r];
    }
  };
  stats(row);
  for (; row < rows; row += step) {
    fetch(row + (NORM_BWD_STAGES - 1) * step, (stage + NORM_BWD_STAGES - 1) % NORM_BWD_STAGES);
    const float mean = mean_next, rstd = rstd_next;
    stats(row + step);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NORM_BWD_STAGES - 1) : "memory");
    const uint4* at = ring + stage * 3 * VPL * 32;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (TAIL && (i * 32 + lane) * 8 >= H) continue;
      float xv[8], gv[8], gm[8];
      unpack8(at[i * 32], xv);
      unpack8(at[(VPL + i) * 32], gv);
      Vec8<W>::load(gamma + (i * 32 + lane) * 8, gm);      // (from L1 in both passes instead of VPL x 8 registers)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean) * rstd;
        const float gw = gv[j] * gm[j];
        s1 += gw;
        s2 += gw * xh;
        dg[i][j] += gv[j] * xh;
        db[i][j] += gv[j];
      }
    }
    s1 = RMS ? 0.f : warp_sum(s1) * inv_h;
    s2 = warp_sum(s2) * inv_h;
    const size_t base = static_cast<size_t>(row) * H;
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (TAIL && (i * 32 + lane) * 8 >= H) continue;
      float xv[8], gv[8], gm[8], o[8];
      unpack8(at[i * 32], xv);
      unpack8(at[(VPL + i) * 32], gv);
      Vec8<W>::load(gamma + (i * 32 + lane) * 8, gm);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean) * rstd;
        o[j] = rstd * (gv[j] * gm[j] - s1 - xh * s2);
      }
      if (gadd != nullptr) {  // the skip connection's gradient rides along: saves autograd's separate add kernel
        float a[8];
        unpack8(at[(2 * VPL + i) * 32], a);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j] += a[j];
          if constexpr (SUMS) sa[i][j] += a[j];
        }
      }
      const uint4 q = make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
      *reinterpret_cast<uint4*>(gx + base + (i * 32 + lane) * 8) = q;
      if constexpr (SUMS) {                      // (of the bf16 numbers that the next layer gets)
        unpack8(q, o);
#pragma unroll
        for (int j = 0; j < 8; ++j) so[i][j] += o[j];
      }
    }
    stage = stage + 1 == NORM_BWD_STAGES ? 0 : stage + 1;
  }
  // the block's column sums, over the ring
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  float* sums = reinterpret_cast<float*>(norm_ring);       // [which][warp][column]
  auto put = [&](int which, const float (*v)[8]) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      float* to = sums + ((which * NORM_BWD_WARPS + warp) * VPL + i) * 256 + lane * 8;
      *reinterpret_cast<float4*>(to) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
      *reinterpret_cast<float4*>(to + 4) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
    }
  };
  put(0, dg);
  put(1, db);
  if constexpr (SUMS) {
    put(2, sa);
    put(3, so);
  }
  __syncthreads();
  for (int which = 0; which < (SUMS ? 4 : 2); ++which) {
    float* part = which == 0 ? part_dgamma : part_dbeta;
    // accumulate mode (training: the parameters' fp32 main_grad buffers): straight into the gradients instead of a [blocks, H] matrix of partial
    // sums and a second reduction kernel
    float* acc = which == 0 ? acc_dgamma : which == 1 ? acc_dbeta : which == 2 ? sum_add : sum_out;
    const bool add = which >= 2 || acc_dgamma != nullptr;
    if (add ? acc == nullptr : part == nullptr) continue;
    for (int c = threadIdx.x * 4; c < H; c += NORM_BWD_WARPS * 128) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < NORM_BWD_WARPS; ++w) {
        const float4 u = *reinterpret_cast<const float4*>(sums + (which * NORM_BWD_WARPS + w) * VPL * 256 + c);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
      }
      float* dst = add ? acc + c : part + static_cast<size_t>(blockIdx.x) * H + c;
      if (add && (reinterpret_cast<uintptr_t>(acc) & 15) == 0) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
      } else if (add) {
        atomicAdd(dst, v.x);
        atomicAdd(dst + 1, v.y);
        atomicAdd(dst + 2, v.z);
        atomicAdd(dst + 3, v.w);
      } else {
        *reinterpret_cast<float4*>(dst) = v;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Wide bf16 rows (1024 < H <= 8192, H % 8 == 0): one 256-thread block per row, V = ceil(H / 2048) 16-byte vectors per
// thread.  Bandwidth-bound.  With a warp per row a lane of a 4096-wide row held 16 vectors, i.e. 2 x 128 fp32 column sums
// next to x̂ and g·γ: it spilled, and [2048, 4096] took 298 us backward (13.6 us forward) where the 50 MB (34 MB) it moves
// take 8 us (5 us).  Spread over a block the column sums are 16 V registers, every row's loads are issued at once and the two
// row sums cost one barrier: 20.6 us backward, 7.6 us forward.  Few rows (a decoding step) gain as well: a row is no longer one
// warp's serial walk (4 rows of 4096: 9.9 -> 2.8 us).
// ---------------------------------------------------------------------------------------------------------------------
constexpr int NORM_WIDE_THREADS = 256;

// sums of two values over the block; `buf` alternates so that one barrier per call is enough
LB_DEVICE float2 norm_block_sum2(float a, float b, float2 (*red)[NORM_WIDE_THREADS / 32], int& buf) {
  a = warp_sum(a);
  b = warp_sum(b);
  if (threadIdx.x % 32 == 0) red[buf][threadIdx.x / 32] = make_float2(a, b);
  __syncthreads();
  float2 t = make_float2(0.f, 0.f);
#pragma unroll
  for (int w = 0; w < NORM_WIDE_THREADS / 32; ++w) {
    const float2 r = red[buf][w];
    t.x += r.x;
    t.y += r.y;
  }
  buf ^= 1;
  return t;
}
LB_DEVICE void norm_unpack8(const uint4& q, float (&v)[8]) {
  const float2 a = unpack_bf16(q.x), b = unpack_bf16(q.y), c = unpack_bf16(q.z), d = unpack_bf16(q.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}

template <typename W, int V, bool RMS>
__global__ void __launch_bounds__(NORM_WIDE_THREADS)
norm_fwd_wide_kernel(const __nv_bfloat16* __restrict__ x, const W* __restrict__ gamma, const W* __restrict__ beta,
                     __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int H,
                     float eps) {
  chain_wait(x, gamma, beta);
  chain_next();
  __shared__ float2 red[2][NORM_WIDE_THREADS / 32];
  int buf = 0;
  const float inv_h = 1.0f / static_cast<float>(H);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 q[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
      q[i] = c < H ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
    }
    float mean = 0.f;
    if (!RMS) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float v[8];
        norm_unpack8(q[i], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j];
      }
      mean = norm_block_sum2(s, 0.f, red, buf).x * inv_h;
    }
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if ((i * NORM_WIDE_THREADS + static_cast<int>(threadIdx.x)) * 8 >= H) continue;
      float v[8];
      norm_unpack8(q[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) sq += (v[j] - mean) * (v[j] - mean);
    }
    const float rstd = rsqrtf(norm_block_sum2(sq, 0.f, red, buf).x * inv_h + eps);
    if (threadIdx.x == 0) {
      if (mean_out) mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
      if (c >= H) continue;
      float v[8], g[8], b[8], o[8];
      norm_unpack8(q[i], v);
      Vec8<W>::load(gamma + c, g);
      if (beta != nullptr) Vec8<W>::load(beta + c, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = (v[j] - mean) * rstd * g[j];
        if (beta != nullptr) o[j] += b[j];
      }
      Vec8<__nv_bfloat16>::store(y + base + c, o);
    }
  }
}

// Column sums: one row of partials per block, which colreduce_kernel adds up in a fixed order (vector reductions from every block straight
// into the fp32 gradients saved that launch, but their order, and with it the last bits of a weight gradient, changed from run to run).
template <typename W, int V, bool RMS>
__global__ void __launch_bounds__(NORM_WIDE_THREADS, V <= 2 ? 3 : 1)
norm_bwd_wide_kernel(const __nv_bfloat16* __restrict__ gy, const __nv_bfloat16* __restrict__ x, const W* __restrict__ gamma,
                     const float* __restrict__ mean_in, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ gx,
                     float* __restrict__ part_dgamma, float* __restrict__ part_dbeta, int rows, int H,
                     const __nv_bfloat16* __restrict__ gadd) {
  chain_next();
  __shared__ float2 red[2][NORM_WIDE_THREADS / 32];
  int buf = 0;
  const float inv_h = 1.0f / static_cast<float>(H);
  float dg[V][8], db[V][8];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dg[i][j] = db[i][j] = 0.f;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 xq[V], gq[V], aq[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
      const bool ok = c < H;
      xq[i] = ok ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
      gq[i] = ok ? *reinterpret_cast<const uint4*>(gy + base + c) : make_uint4(0, 0, 0, 0);
      aq[i] = (ok && gadd != nullptr) ? *reinterpret_cast<const uint4*>(gadd + base + c) : make_uint4(0, 0, 0, 0);
    }
    const float mean = RMS ? 0.f : mean_in[row];
    const float rstd = rstd_in[row];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
      if (c >= H) continue;
      float xv[8], gv[8], gm[8];
      norm_unpack8(xq[i], xv);
      norm_unpack8(gq[i], gv);
      Vec8<W>::load(gamma + c, gm);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean) * rstd, gw = gv[j] * gm[j];
        s1 += gw;
        s2 += gw * xh;
        dg[i][j] += gv[j] * xh;
        db[i][j] += gv[j];
      }
    }
    const float2 t = norm_block_sum2(s1, s2, red, buf);
    s1 = RMS ? 0.f : t.x * inv_h;
    s2 = t.y * inv_h;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
      if (c >= H) continue;
      float xv[8], gv[8], gm[8], av[8], o[8];
      norm_unpack8(xq[i], xv);
      norm_unpack8(gq[i], gv);
      norm_unpack8(aq[i], av);
      Vec8<W>::load(gamma + c, gm);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rstd * (gv[j] * gm[j] - s1 - (xv[j] - mean) * rstd * s2) + av[j];
      Vec8<__nv_bfloat16>::store(gx + base + c, o);
    }
  }
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = (i * NORM_WIDE_THREADS + threadIdx.x) * 8;
    if (c >= H) continue;
#pragma unroll
    for (int which = 0; which < 2; ++which) {
      if (which == 1 && part_dbeta == nullptr) continue;
      const float(&v)[8] = which == 0 ? dg[i] : db[i];
      Vec8<float>::store((which == 0 ? part_dgamma : part_dbeta) + static_cast<size_t>(blockIdx.x) * H + c, v);
    }
  }
}

// out[c] = sum_r part[r, c]   (block = 32 columns x 8 row stripes, smem tree over the stripes)
// blockIdx.y selects (part0 -> out0) / (part1 -> out1): dgamma and dbeta in one launch; `accumulate` adds into `out`
// (each column is owned by exactly one thread, so the fp32 main-grad buffer is updated with a plain read-modify-write)
__global__ void __launch_bounds__(256) colreduce_kernel(const float* __restrict__ part0, float* __restrict__ out0,
                                                        const float* __restrict__ part1, float* __restrict__ out1,
                                                        int nrows, int H, int accumulate) {
  chain_wait(part0, out0, part1, out1);
  chain_next();
  const float* __restrict__ part = blockIdx.y == 0 ? part0 : part1;
  float* __restrict__ out = blockIdx.y == 0 ? out0 : out1;
  __shared__ float sm[8][33];
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  const int c = blockIdx.x * 32 + tx;
  float acc = 0.f;
  if (c < H) {
    int r = ty;
    for (; r + 24 < nrows; r += 32) {
      const float a0 = part[static_cast<size_t>(r) * H + c], a1 = part[static_cast<size_t>(r + 8) * H + c];
      const float a2 = part[static_cast<size_t>(r + 16) * H + c], a3 = part[static_cast<size_t>(r + 24) * H + c];
      acc += (a0 + a1) + (a2 + a3);
    }
    for (; r < nrows; r += 8) acc += part[static_cast<size_t>(r) * H + c];
  }
  sm[ty][tx] = acc;
  __syncthreads();
  if (ty == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) t += sm[j][tx];
    out[c] = accumulate ? out[c] + t : t;
  }
}

// ---------------- generic (any H) fallbacks: one warp per row, strided scalar access ----------------
template <typename T, typename W, bool RMS>
__global__ void norm_fwd_generic(const T* __restrict__ x, const W* __restrict__ gamma, const W* __restrict__ beta,
                                 T* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                                 int rows, int H, float eps) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int row = blockIdx.x * (blockDim.x / 32) + warp;
  if (row >= rows) return;
  const T* xr = x + static_cast<size_t>(row) * H;
  float s = 0.f;
  for (int c = lane; c < H; c += 32) s += static_cast<float>(xr[c]);
  const float mean = RMS ? 0.f : warp_sum(s) / H;
  float sq = 0.f;
  for (int c = lane; c < H; c += 32) {
    const float d = static_cast<float>(xr[c]) - mean;
    sq += d * d;
  }
  const float rstd = rsqrtf(warp_sum(sq) / H + eps);
  if (lane == 0) {
    if (mean_out) mean_out[row] = mean;
    rstd_out[row] = rstd;
  }
  T* yr = y + static_cast<size_t>(row) * H;
  for (int c = lane; c < H; c += 32) {
    float o = (static_cast<float>(xr[c]) - mean) * rstd * static_cast<float>(gamma[c]);
    if (beta != nullptr) o += static_cast<float>(beta[c]);
    yr[c] = static_cast<T>(o);
  }
}

template <typename T, typename W, bool RMS>
__global__ void norm_bwd_generic(const T* __restrict__ gy, const T* __restrict__ x, const W* __restrict__ gamma,
                                 const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                                 T* __restrict__ gx, float* __restrict__ dgamma, float* __restrict__ dbeta, int rows,
                                 int H) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int row = blockIdx.x * (blockDim.x / 32) + warp;
  if (row >= rows) return;
  const float mean = RMS ? 0.f : mean_in[row], rstd = rstd_in[row];
  const T* xr = x + static_cast<size_t>(row) * H;
  const T* gr = gy + static_cast<size_t>(row) * H;
  float s1 = 0.f, s2 = 0.f;
  for (int c = lane; c < H; c += 32) {
    const float xh = (static_cast<float>(xr[c]) - mean) * rstd;
    const float g = static_cast<float>(gr[c]);
    const float gw = g * static_cast<float>(gamma[c]);
    s1 += gw;
    s2 += gw * xh;
    atomicAdd(&dgamma[c], g * xh);
    if (dbeta != nullptr) atomicAdd(&dbeta[c], g);
  }
  s1 = RMS ? 0.f : warp_sum(s1) / H;
  s2 = warp_sum(s2) / H;
  T* gxr = gx + static_cast<size_t>(row) * H;
  for (int c = lane; c < H; c += 32) {
    const float xh = (static_cast<float>(xr[c]) - mean) * rstd;
    const float gw = static_cast<float>(gr[c]) * static_cast<float>(gamma[c]);
    gxr[c] = static_cast<T>(rstd * (gw - s1 - xh * s2));
  }
}

}  // namespace lb

namespace {
int norm_sms() {                                  // (without a device: of the chip that the grids are made for)
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
    sms = n;
  }
  return sms;
}
int norm_grid_of(int rows, int rows_per_block, int blocks_per_sm) {
  const int need = (rows + rows_per_block - 1) / rows_per_block;
  const int cap = norm_sms() * blocks_per_sm;
  return need < cap ? need : cap;
}
int norm_grid(int rows) { return norm_grid_of(rows, lb::NORM_WARPS, 2); }
// forward: 64 registers → four 8-warp blocks per SM
int norm_fwd_grid(int rows) { return norm_grid_of(rows, lb::NORM_WARPS, 4); }
// bf16 backward: up to three 4-warp blocks per SM (one wave), but no more than give every warp up to three rows once there is a block per SM: every block adds or leaves
// a row of column sums, which took longer than the rows ([1812, 256] 453 blocks 5.3 us, 151 blocks 3.3; [2048, 384] 6.2 and 5.1; [200, 384] 50 blocks 2.8, 17 blocks 4.2).
int norm_bwd_bf16_grid(int rows, int H, bool sums) {
  if (rows <= 0) return 0;
  const int per_sm = lb::NORM_BWD_WARPS * norm_sms(), want = (rows + per_sm - 1) / per_sm, each = want < lb::NORM_BWD_STAGES ? want : lb::NORM_BWD_STAGES;
  return norm_grid_of(rows, lb::NORM_BWD_WARPS * each, lb::norm_bwd_blocks((H + 255) / 256, sums));
}
// wide rows: blocks loop over rows; the backward keeps to one wave, and to as few blocks as do it in the same number of rounds, because
// every block leaves a row of column sums at the end
int norm_fwd_wide_grid(int rows) { return norm_grid_of(rows, 1, 6); }
int norm_bwd_wide_grid(int rows, int H) {
  const int cap = norm_sms() * (H <= 4096 ? 3 : 1);
  if (rows <= cap) return rows;
  const int rounds = cap > 0 ? (rows + cap - 1) / cap : rows;
  return (rows + rounds - 1) / rounds;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
// bf16 rows of whole 16-byte vectors: the warp kernels up to 1024 columns (four vectors per lane: beyond that their column sums
// spill), the block kernels up to 8192, but for the rules below
constexpr int NORM_WARP_MAX_H = 1024, NORM_WIDE_MAX_H = 8192;
bool norm_vec_bf16(int H, int dtype) { return dtype == 0 && H % 8 == 0 && H <= NORM_WIDE_MAX_H; }
// Between 1024 and 2560 columns a warp still holds a row, and with enough rows to fill the chip with warps it is ahead of a block per row, whose
// row sums cost barriers.  Forward, warp / block: layer norm [1024, 1280] 3.2 / 3.5, [8192, 1280] 10 / 17, [1024, 2048] 4.1 / 3.7, [1536, 2048]
// 4.4 / 4.7, [8192, 2560] 19 / 31 us, [8192, 3072] equal; RMS norm [1024, 1280] 2.9 / 2.8, [1536, 1280] 2.8 / 3.1, [1536, 2048] 3.9 / 3.5, [8192, 2048]
// 14 / 16 us.  Backward (column sums beside the row: up to 1536): [256, 1280] 6.1 / 5.6, [512, 1280] 6.2 / 8.5, [8192, 1280] 23 / 32, [512, 1536]
// 6.8 / 9.1 us; [8192, 2048] 45 / 38, but [1024, 2048] 10.4 / 11.3 (one round of one block of warps per SM).  (2560 = 10 vectors per lane; 7 and
// 9 are not compiled.)
bool norm_fwd_by_warp(int rows, int H, bool rms) {
  return H % 256 == 0 && H <= 2560 && H != 1792 && H != 2304 && rows >= (H <= 1536 ? 1024 : 1536) + (rms ? 512 : 0);
}
bool norm_bwd_by_warp(int rows, int H) {
  return ((H == 1280 || H == 1536) && rows > 296) || (H == 2048 && rows > 888 && rows <= 148 * lb::NORM_WARPS);
}

// fp32 activations: H = 256 VPL
// Chained where every row has its own warp or block.  Where blocks take several rows in turn, the first SMs to come free would get the blocks with one row
// more: [12608, 1024] 10.9 us in order, 13.0 chained.
template <typename... P, typename... A>
void launch_norm(bool chain, void (*kern)(P...), int grid, int threads, cudaStream_t s, const A&... args) {
  if (chain) lb_host::launch_chained(kern, dim3(grid), dim3(threads), 0, s, 0, args...);
  else kern<<<grid, threads, 0, s>>>(static_cast<P>(args)...);
}
template <bool RMS>
bool fwd_dispatch_f32(int vpl, const float* x, const float* g, const float* b, float* y, float* mean, float* rstd, int rows,
                      float eps, cudaStream_t s) {
  const int grid = norm_fwd_grid(rows);
#define LB_CASE(V)                                                                                                            \
  case V:                                                                                                                     \
    launch_norm(rows <= grid * lb::NORM_WARPS, lb::norm_fwd_kernel<float, float, V, RMS, false>, grid, lb::NORM_WARPS * 32, s, x, g, b, y, mean, rstd, rows, eps, 0); \
    return true;
  switch (vpl) {
    LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) LB_CASE(5) LB_CASE(6) LB_CASE(8) LB_CASE(10) LB_CASE(12) LB_CASE(16)
    LB_CASE(20) LB_CASE(32)
    default:
      return false;
  }
#undef LB_CASE
}

template <typename W, bool RMS>
void fwd_dispatch_bf16(int H, const __nv_bfloat16* x, const W* g, const W* b, __nv_bfloat16* y, float* mean, float* rstd, int rows,
                       float eps, cudaStream_t s) {
  if (H <= NORM_WARP_MAX_H) {
    const int grid = norm_fwd_grid(rows);
#define LB_CASE(V)                                                                                                                  \
  case V:                                                                                                                           \
    if (H % 256 == 0)                                                                                                               \
      launch_norm(rows <= grid * lb::NORM_WARPS, lb::norm_fwd_kernel<__nv_bfloat16, W, V, RMS, false>, grid, lb::NORM_WARPS * 32, s, x, g, b, y, mean, rstd, rows, eps, H); \
    else                                                                                                                            \
      launch_norm(rows <= grid * lb::NORM_WARPS, lb::norm_fwd_kernel<__nv_bfloat16, W, V, RMS, true>, grid, lb::NORM_WARPS * 32, s, x, g, b, y, mean, rstd, rows, eps, H);  \
    break;
    switch ((H + 255) / 256) { LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) }
#undef LB_CASE
    return;
  }
  if (norm_fwd_by_warp(rows, H, RMS)) {
    const int grid = norm_fwd_grid(rows);
#define LB_CASE(V)                                                                                                                  \
  case V:                                                                                                                           \
    launch_norm(rows <= grid * lb::NORM_WARPS, lb::norm_fwd_kernel<__nv_bfloat16, W, V, RMS, false>, grid, lb::NORM_WARPS * 32, s, x, g, b, y, mean, rstd, rows, eps, H); \
    break;
    switch (H / 256) { LB_CASE(5) LB_CASE(6) LB_CASE(8) LB_CASE(10) }
#undef LB_CASE
    return;
  }
  const int grid = norm_fwd_wide_grid(rows);
#define LB_CASE(V)                                                                                                             \
  case V:                                                                                                                      \
    launch_norm(rows <= grid, lb::norm_fwd_wide_kernel<W, V, RMS>, grid, lb::NORM_WIDE_THREADS, s, x, g, b, y, mean, rstd, rows, H, eps);          \
    break;
  switch ((H + 2047) / 2048) { LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) }
#undef LB_CASE
}

template <typename W, int V, bool RMS, bool TAIL, bool SUMS, typename... A>
void launch_norm_bwd(int grid, cudaStream_t s, const A&... args) {
  auto kern = lb::norm_bwd_bf16_kernel<W, V, RMS, TAIL, SUMS>;
  constexpr int smem = lb::NORM_BWD_WARPS * lb::NORM_BWD_STAGES * 3 * V * 512;
  static_assert(smem >= 4 * lb::NORM_BWD_WARPS * V * 1024, "column sums fit the ring");
  if (smem > 48 * 1024) {                        // the limit is per device
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!(done.load(std::memory_order_relaxed) & bit) && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess)
      done.fetch_or(bit, std::memory_order_relaxed);
  }
  kern<<<grid, lb::NORM_BWD_WARPS * 32, smem, s>>>(args...);
}

template <typename W, bool RMS>
void bwd_dispatch_bf16(int H, const __nv_bfloat16* gy, const __nv_bfloat16* x, const W* g, const float* mean, const float* rstd,
                       __nv_bfloat16* gx, float* pdg, float* pdb, int rows, int grid, cudaStream_t s, const __nv_bfloat16* gadd,
                       float* acc_dg, float* acc_db) {
  if (H <= NORM_WARP_MAX_H) {
    float* none = nullptr;
#define LB_CASE(V)                                                                                                                                    \
  case V:                                                                                                                                             \
    if (H % 256 == 0) launch_norm_bwd<W, V, RMS, false, false>(grid, s, gy, x, g, mean, rstd, gx, pdg, pdb, rows, gadd, acc_dg, acc_db, none, none, H); \
    else launch_norm_bwd<W, V, RMS, true, false>(grid, s, gy, x, g, mean, rstd, gx, pdg, pdb, rows, gadd, acc_dg, acc_db, none, none, H);              \
    break;
    switch ((H + 255) / 256) { LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) }
#undef LB_CASE
    return;
  }
  if (norm_bwd_by_warp(rows, H)) {
#define LB_CASE(V)                                                                                                                            \
  case V:                                                                                                                                     \
    lb::norm_bwd_kernel<__nv_bfloat16, W, V, RMS><<<grid, lb::NORM_WARPS * 32, 0, s>>>(gy, x, g, mean, rstd, gx, pdg, pdb, rows, gadd);        \
    break;
    switch (H / 256) { LB_CASE(5) LB_CASE(6) LB_CASE(8) }
#undef LB_CASE
    return;
  }
#define LB_CASE(V)                                                                                                              \
  case V:                                                                                                                       \
    lb::norm_bwd_wide_kernel<W, V, RMS><<<grid, lb::NORM_WIDE_THREADS, 0, s>>>(gy, x, g, mean, rstd, gx, pdg, pdb, rows, H, gadd); \
    break;
  switch ((H + 2047) / 2048) { LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) }
#undef LB_CASE
}

template <bool RMS>
bool bwd_dispatch_f32(int vpl, const float* gy, const float* x, const float* g, const float* mean, const float* rstd, float* gx,
                      float* pdg, float* pdb, int rows, int grid, cudaStream_t s, const float* gadd) {
#define LB_CASE(V)                                                                                                           \
  case V:                                                                                                                    \
    lb::norm_bwd_kernel<float, float, V, RMS><<<grid, lb::NORM_WARPS * 32, 0, s>>>(gy, x, g, mean, rstd, gx, pdg, pdb, rows, gadd); \
    return true;
  switch (vpl) {
    LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) LB_CASE(5) LB_CASE(6) LB_CASE(8) LB_CASE(10) LB_CASE(12) LB_CASE(16)
    default:
      return false;
  }
#undef LB_CASE
}

template <typename W>
void norm_fwd_bf16(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows, int H, float eps,
                   int rms, cudaStream_t s) {
  using T = __nv_bfloat16;
  if (norm_vec_bf16(H, 0) && aligned16(x) && aligned16(y) && aligned16(gamma) && aligned16(beta)) {
    if (rms) fwd_dispatch_bf16<W, true>(H, (const T*)x, (const W*)gamma, (const W*)beta, (T*)y, mean, rstd, rows, eps, s);
    else fwd_dispatch_bf16<W, false>(H, (const T*)x, (const W*)gamma, (const W*)beta, (T*)y, mean, rstd, rows, eps, s);
    return;
  }
  const int wpb = 8, grid = (rows + wpb - 1) / wpb;
  if (rms) lb::norm_fwd_generic<T, W, true><<<grid, wpb * 32, 0, s>>>((const T*)x, (const W*)gamma, (const W*)beta, (T*)y, mean, rstd, rows, H, eps);
  else lb::norm_fwd_generic<T, W, false><<<grid, wpb * 32, 0, s>>>((const T*)x, (const W*)gamma, (const W*)beta, (T*)y, mean, rstd, rows, H, eps);
}
template <typename T, typename W>
void norm_bwd_any(const void* gy, const void* x, const void* gamma, const float* mean, const float* rstd, void* gx, float* dgamma,
                  float* dbeta, int rows, int H, int rms, int accumulate, cudaStream_t s) {
  if (!accumulate) {
    cudaMemsetAsync(dgamma, 0, sizeof(float) * H, s);
    if (dbeta != nullptr) cudaMemsetAsync(dbeta, 0, sizeof(float) * H, s);
  }
  const int wpb = 8, grid = (rows + wpb - 1) / wpb;
  if (rms) lb::norm_bwd_generic<T, W, true><<<grid, wpb * 32, 0, s>>>((const T*)gy, (const T*)x, (const W*)gamma, mean, rstd, (T*)gx, dgamma, dbeta, rows, H);
  else lb::norm_bwd_generic<T, W, false><<<grid, wpb * 32, 0, s>>>((const T*)gy, (const T*)x, (const W*)gamma, mean, rstd, (T*)gx, dgamma, dbeta, rows, H);
}
}  // namespace

// dtype codes: 0 = bf16 activations, 1 = fp32 activations; wdtype: 0 = bf16 params, 1 = fp32 params
extern "C" int lb_norm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd,
                           int rows, int H, float eps, int rms, int dtype, int wdtype, cudaStream_t s) {
  if (rows == 0) return 0;
  if (dtype == 0 && wdtype == 0) {
    norm_fwd_bf16<__nv_bfloat16>(x, gamma, beta, y, mean, rstd, rows, H, eps, rms, s);
  } else if (dtype == 0 && wdtype == 1) {
    norm_fwd_bf16<float>(x, gamma, beta, y, mean, rstd, rows, H, eps, rms, s);
  } else if (dtype == 1 && wdtype == 1) {
    const float *xf = (const float*)x, *gf = (const float*)gamma, *bf = (const float*)beta;
    bool done = false;
    if (H % 256 == 0)
      done = rms ? fwd_dispatch_f32<true>(H / 256, xf, gf, bf, (float*)y, mean, rstd, rows, eps, s)
                 : fwd_dispatch_f32<false>(H / 256, xf, gf, bf, (float*)y, mean, rstd, rows, eps, s);
    if (!done) {
      const int wpb = 8, grid = (rows + wpb - 1) / wpb;
      if (rms) lb::norm_fwd_generic<float, float, true><<<grid, wpb * 32, 0, s>>>(xf, gf, bf, (float*)y, mean, rstd, rows, H, eps);
      else lb::norm_fwd_generic<float, float, false><<<grid, wpb * 32, 0, s>>>(xf, gf, bf, (float*)y, mean, rstd, rows, H, eps);
    }
  } else {
    return -1;
  }
  return (int)cudaGetLastError();
}

// workspace: float[2 * grid_cap * H] where grid_cap = lb_norm_bwd_workspace_rows(); dgamma/dbeta fp32 [H]
extern "C" int lb_norm_bwd_workspace_rows(int rows, int H) {
  const int a = norm_grid(rows), b = norm_bwd_bf16_grid(rows, H, false), c = norm_bwd_wide_grid(rows, H);
  return a > b ? (a > c ? a : c) : (b > c ? b : c);
}
// the fused "+ residual gradient" is implemented by the register-cached kernels only: bf16 rows of whole aligned vectors, fp32
// rows of H = 256 * {1..6, 8, 10, 12, 16}
extern "C" int lb_norm_bwd_supports_gadd(int H, int dtype, const void* gy, const void* x, const void* gamma, const void* gx, const void* gadd) {
  if (dtype == 0) return norm_vec_bf16(H, dtype) && aligned16(gy) && aligned16(x) && aligned16(gamma) && aligned16(gx) && aligned16(gadd);
  if (H % 256 != 0) return 0;
  const int v = H / 256;
  return (v >= 1 && v <= 6) || v == 8 || v == 10 || v == 12 || v == 16;
}

extern "C" int lb_norm_bwd(const void* gy, const void* x, const void* gamma, const float* mean, const float* rstd,
                           void* gx, float* dgamma, float* dbeta, float* workspace, int rows, int H, int rms, int dtype,
                           int wdtype, int accumulate, const void* gadd, cudaStream_t s) {
  if (rows == 0) return 0;
  if (gadd != nullptr && !lb_norm_bwd_supports_gadd(H, dtype, gy, x, gamma, gx, gadd)) return -3;  // caller adds the residual gradient itself
  using B = __nv_bfloat16;
  if (dtype == 0 && (wdtype == 0 || wdtype == 1)) {
    if (!norm_vec_bf16(H, dtype) || !aligned16(gy) || !aligned16(x) || !aligned16(gamma) || !aligned16(gx)) {
      if (wdtype == 0) norm_bwd_any<B, B>(gy, x, gamma, mean, rstd, gx, dgamma, dbeta, rows, H, rms, accumulate, s);
      else norm_bwd_any<B, float>(gy, x, gamma, mean, rstd, gx, dgamma, dbeta, rows, H, rms, accumulate, s);
      return (int)cudaGetLastError();
    }
    const int grid = H <= NORM_WARP_MAX_H ? norm_bwd_bf16_grid(rows, H, false) : norm_bwd_by_warp(rows, H) ? norm_grid(rows) : norm_bwd_wide_grid(rows, H);
    float* pdg = workspace;
    float* pdb = dbeta != nullptr ? workspace + static_cast<size_t>(grid) * H : nullptr;
    // accumulate mode: the warp kernel's blocks add their column sums straight into dgamma / dbeta
    const bool direct = accumulate && H <= NORM_WARP_MAX_H;
    float* adg = direct ? dgamma : nullptr;
    float* adb = direct ? dbeta : nullptr;
#define LB_GO(W, R) bwd_dispatch_bf16<W, R>(H, (const B*)gy, (const B*)x, (const W*)gamma, mean, rstd, (B*)gx, pdg, pdb, rows, grid, s, (const B*)gadd, adg, adb)
    if (wdtype == 0) { if (rms) LB_GO(B, true); else LB_GO(B, false); }
    else { if (rms) LB_GO(float, true); else LB_GO(float, false); }
#undef LB_GO
    if (!direct)
      lb_host::launch_chained(lb::colreduce_kernel, dim3((H + 31) / 32, dbeta != nullptr ? 2 : 1), dim3(256), 0, s, 0, pdg, dgamma, pdb, dbeta, grid, H, accumulate);
  } else if (dtype == 1 && wdtype == 1) {
    const int grid = norm_grid(rows);
    float* pdg = workspace;
    float* pdb = dbeta != nullptr ? workspace + static_cast<size_t>(grid) * H : nullptr;
    bool done = false;
    if (H % 256 == 0 && H / 256 <= 16)
      done = rms ? bwd_dispatch_f32<true>(H / 256, (const float*)gy, (const float*)x, (const float*)gamma, mean, rstd, (float*)gx, pdg, pdb, rows, grid, s, (const float*)gadd)
                 : bwd_dispatch_f32<false>(H / 256, (const float*)gy, (const float*)x, (const float*)gamma, mean, rstd, (float*)gx, pdg, pdb, rows, grid, s, (const float*)gadd);
    if (done)
      lb_host::launch_chained(lb::colreduce_kernel, dim3((H + 31) / 32, dbeta != nullptr ? 2 : 1), dim3(256), 0, s, 0, pdg, dgamma, pdb, dbeta, grid, H, accumulate);
    else
      norm_bwd_any<float, float>(gy, x, gamma, mean, rstd, gx, dgamma, dbeta, rows, H, rms, accumulate, s);
  } else {
    return -1;
  }
  return (int)cudaGetLastError();
}

// Layer norm backward on bf16 rows of up to 1024 columns that adds into fp32 gradients and, beside them, the column sums of gadd into sum_add and those of gx into sum_out
// (either may be nullptr): the gradients of the biases around the norm.  -3: not of this form.
extern "C" int lb_norm_bwd_sums(const void* gy, const void* x, const void* gamma, const float* mean, const float* rstd, void* gx, float* dgamma, float* dbeta, int rows,
                                int H, const void* gadd, float* sum_add, float* sum_out, cudaStream_t s) {
  using B = __nv_bfloat16;
  if (H > NORM_WARP_MAX_H || !norm_vec_bf16(H, 0) || gadd == nullptr || dgamma == nullptr || dbeta == nullptr ||
      !lb_norm_bwd_supports_gadd(H, 0, gy, x, gamma, gx, gadd))
    return -3;
  if (rows == 0) return 0;
  const int grid = norm_bwd_bf16_grid(rows, H, true);
  float* none = nullptr;
#define LB_CASE(V)                                                                                                                                                     \
  case V:                                                                                                                                                              \
    if (H % 256 == 0)                                                                                                                                                  \
      launch_norm_bwd<B, V, false, false, true>(grid, s, (const B*)gy, (const B*)x, (const B*)gamma, mean, rstd, (B*)gx, none, none, rows, (const B*)gadd, dgamma, dbeta, \
                                                sum_add, sum_out, H);                                                                                                  \
    else                                                                                                                                                               \
      launch_norm_bwd<B, V, false, true, true>(grid, s, (const B*)gy, (const B*)x, (const B*)gamma, mean, rstd, (B*)gx, none, none, rows, (const B*)gadd, dgamma, dbeta, \
                                               sum_add, sum_out, H);                                                                                                   \
    break;
  switch ((H + 255) / 256) { LB_CASE(1) LB_CASE(2) LB_CASE(3) LB_CASE(4) }
#undef LB_CASE
  return (int)cudaGetLastError();
}

// One generated token per sequence against a key / value cache: softmax(q Kᵀ) V and the caches grown by the new token, one launch.
//
// The step used to concatenate both caches (torch.cat), convert both to fp32 and run two matrix-vector products and a softmax over
// [b, a, 1, s] on them: at [4, 32, 2047, 128] 531 us of copies, 185 us of conversions and 86 us of products where reading both
// caches once and writing both grown caches once (268 MB) takes 41 us.  Here a CTA streams a range of one head's keys: every 16-byte
// vector that it reads is written to the grown cache and used from the register: 44 us (6.1 TB/s);
// [8, 16, 511, 64] 110 -> 7.9 us.
//
// Bandwidth-bound, so the split is by bytes in flight: LPR lanes hold one row (16 bytes each), a warp 32 / LPR rows, four rows per
// lane group and step (eight 16-byte loads per thread).  A head's keys are split over the CTAs of a cluster (1, 2, 4 or 8: enough
// that the grid has three CTAs per SM, as long as each has 64 keys), which merge through distributed shared memory: no second
// launch, no workspace.  All arithmetic is fp32: products of bf16 numbers, maxima, sums and probabilities.
#include "common.cuh"

namespace lb {

constexpr int ADEC_THREADS = 128, ADEC_WARPS = ADEC_THREADS / 32, ADEC_UNROLL = 4;

struct DecodeParams {
  const __nv_bfloat16 *q, *k_new, *v_new;      // [B, A, 1, d] views: batch and head strides
  long q_st[2], kn_st[2], vn_st[2];
  const __nv_bfloat16 *k_past, *v_past;        // [B, A, past, d] views
  long kp_st[3], vp_st[3];
  __nv_bfloat16 *k_out, *v_out;                // [B, A, past + 1, d] contiguous
  __nv_bfloat16* o;                            // [B, 1, A, d] contiguous
  const uint32_t* mask;                        // optional words [Bm, Am, 1, pitch] and fill [Bm, Am, 1] (log2 domain)
  const float* fill;
  long mask_b, mask_a;
  int pitch;
  int A, past, d;
  float scale_log2;
};

LB_DEVICE float ld_dsmem_f32(uint32_t addr, uint32_t rank) {
  uint32_t ra;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(ra) : "memory");
  return v;
}

// grid (cluster size, A, B), cluster (cluster size, 1, 1); LPR lanes per row, LPR * 8 >= d
template <int LPR, bool MASKED>
__global__ void __launch_bounds__(ADEC_THREADS)
attn_decode_kernel(const DecodeParams p) {
  constexpr int RPW = 32 / LPR;                                   // rows per warp and load
  constexpr int GROUPS = ADEC_WARPS * RPW;
  __shared__ float s_m[GROUPS], s_l[GROUPS];
  __shared__ float s_acc[GROUPS][LPR * 8];
  __shared__ float c_ml[2];                                       // this CTA's merged maximum and sum
  __shared__ float c_acc[LPR * 8];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, sub = lane % LPR, grp = warp * RPW + lane / LPR;
  const int nsplit = gridDim.x, split = blockIdx.x, head = blockIdx.y, batch = blockIdx.z;
  const int S = p.past + 1;
  const int per = ((S + nsplit - 1) / nsplit + GROUPS - 1) / GROUPS * GROUPS;
  const int k_lo = min(S, split * per), k_hi = min(S, k_lo + per);
  const bool col_ok = sub * 8 < p.d;
  auto unpack8 = [](const uint4& w, float (&v)[8]) {
    const float2 a = unpack_bf16(w.x), b = unpack_bf16(w.y), c = unpack_bf16(w.z), e = unpack_bf16(w.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = e.x; v[7] = e.y;
  };
  chain_wait();
  chain_next();
  float q[8];
  unpack8(col_ok ? *reinterpret_cast<const uint4*>(p.q + batch * p.q_st[0] + head * p.q_st[1] + sub * 8) : make_uint4(0, 0, 0, 0), q);
  const __nv_bfloat16* kp = p.k_past + batch * p.kp_st[0] + head * p.kp_st[1] + sub * 8;
  const __nv_bfloat16* vp = p.v_past + batch * p.vp_st[0] + head * p.vp_st[1] + sub * 8;
  const __nv_bfloat16* kn = p.k_new + batch * p.kn_st[0] + head * p.kn_st[1] + sub * 8;
  const __nv_bfloat16* vn = p.v_new + batch * p.vn_st[0] + head * p.vn_st[1] + sub * 8;
  const size_t out0 = (static_cast<size_t>(batch) * p.A + head) * S * p.d + sub * 8;
  [[maybe_unused]] const uint32_t* mrow = nullptr;
  [[maybe_unused]] float fill = 0.f;
  if constexpr (MASKED) {
    const long row = batch * p.mask_b + head * p.mask_a;
    mrow = p.mask + row * p.pitch;
    fill = p.fill[row];
  }
  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  // (the bound is the same for all lanes: the shuffles below need them)
  for (int base = k_lo; base < k_hi; base += GROUPS * ADEC_UNROLL) {
    uint4 kv[ADEC_UNROLL], vv[ADEC_UNROLL];
    float s[ADEC_UNROLL];
#pragma unroll
    for (int u = 0; u < ADEC_UNROLL; ++u) {
      const int key = base + u * GROUPS + grp;
      const bool ok = key < k_hi && col_ok;
      kv[u] = ok ? *reinterpret_cast<const uint4*>(key < p.past ? kp + key * p.kp_st[2] : kn) : make_uint4(0, 0, 0, 0);
      vv[u] = ok ? *reinterpret_cast<const uint4*>(key < p.past ? vp + key * p.vp_st[2] : vn) : make_uint4(0, 0, 0, 0);
    }
    float mx = m;
#pragma unroll
    for (int u = 0; u < ADEC_UNROLL; ++u) {
      const int key = base + u * GROUPS + grp;
      if (key < k_hi && col_ok) {
        *reinterpret_cast<uint4*>(p.k_out + out0 + static_cast<size_t>(key) * p.d) = kv[u];
        *reinterpret_cast<uint4*>(p.v_out + out0 + static_cast<size_t>(key) * p.d) = vv[u];
      }
      float k8[8], t = 0.f;
      unpack8(kv[u], k8);
#pragma unroll
      for (int j = 0; j < 8; ++j) t = fmaf(q[j], k8[j], t);
#pragma unroll
      for (int x = LPR / 2; x >= 1; x >>= 1) t += __shfl_xor_sync(0xffffffffu, t, x);
      t *= p.scale_log2;
      if constexpr (MASKED) {
        if (key < k_hi && !((mrow[key >> 5] >> (key & 31)) & 1u)) t = fill;
      }
      s[u] = key < k_hi ? t : -INFINITY;
      mx = fmaxf(mx, s[u]);
    }
    const float mu = mx == -INFINITY ? 0.f : mx, alpha = fast_exp2(m - mu);
    m = mx;
    l *= alpha;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= alpha;
#pragma unroll
    for (int u = 0; u < ADEC_UNROLL; ++u) {
      if (base + u * GROUPS + grp >= k_hi) continue;              // (a probability of 0 times an infinity would be a NaN)
      const float e = fast_exp2(s[u] - mu);
      l += e;
      float v8[8];
      unpack8(vv[u], v8);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = fmaf(e, v8[j], acc[j]);
    }
  }
  if (sub == 0) { s_m[grp] = m; s_l[grp] = l; }
#pragma unroll
  for (int j = 0; j < 8; ++j) s_acc[grp][sub * 8 + j] = acc[j];
  __syncthreads();
  for (int c = threadIdx.x; c < LPR * 8; c += ADEC_THREADS) {
    float M = -INFINITY;
    for (int g = 0; g < GROUPS; ++g) M = fmaxf(M, s_m[g]);
    const float mu = M == -INFINITY ? 0.f : M;
    float L = 0.f, O = 0.f;
    for (int g = 0; g < GROUPS; ++g) {
      if (s_m[g] == -INFINITY && s_l[g] == 0.f) continue;         // a group without keys
      const float w = fast_exp2(s_m[g] - mu);
      L += s_l[g] * w;
      O += s_acc[g][c] * w;
    }
    c_acc[c] = O;
    if (c == 0) { c_ml[0] = M; c_ml[1] = L; }
  }
  __syncwarp();                                                   // up to 16 columns are merged by a part of warp 0: the barriers take whole warps
  if (nsplit > 1) {
    cluster_sync_all();
    if (split == 0) {
      for (int c = threadIdx.x; c < LPR * 8; c += ADEC_THREADS) {
        float M = -INFINITY, ms[8];
        for (int r = 0; r < nsplit; ++r) {
          ms[r] = ld_dsmem_f32(smem_u32(&c_ml[0]), r);
          M = fmaxf(M, ms[r]);
        }
        const float mu = M == -INFINITY ? 0.f : M;
        float L = 0.f, O = 0.f;
        for (int r = 0; r < nsplit; ++r) {
          const float lr = ld_dsmem_f32(smem_u32(&c_ml[1]), r);
          if (ms[r] == -INFINITY && lr == 0.f) continue;
          const float w = fast_exp2(ms[r] - mu);
          L += lr * w;
          O += ld_dsmem_f32(smem_u32(&c_acc[c]), r) * w;
        }
        if (c < p.d) p.o[(static_cast<size_t>(batch) * p.A + head) * p.d + c] = __float2bfloat16(O / L);
      }
    }
    __syncwarp();
    cluster_sync_all();                                           // nobody leaves while its shared memory is read
  } else {
    __syncthreads();
    for (int c = threadIdx.x; c < p.d; c += ADEC_THREADS)
      p.o[(static_cast<size_t>(batch) * p.A + head) * p.d + c] = __float2bfloat16(c_acc[c] / c_ml[1]);
  }
}

template <int LPR>
cudaError_t launch_attn_decode(const DecodeParams& p, int B, int cluster, cudaStream_t s) {
  const dim3 grid((unsigned)cluster, (unsigned)p.A, (unsigned)B);
  return lb_host::launch_chained(p.mask != nullptr ? attn_decode_kernel<LPR, true> : attn_decode_kernel<LPR, false>, grid, dim3(ADEC_THREADS), 0, s, (unsigned)cluster, p);
}

}  // namespace lb

// strides in elements: q / k_new / v_new (batch, head), k_past / v_past (batch, head, key); every row 16-byte aligned, d % 8 == 0, d <= 256
extern "C" int lb_attn_decode(const void* q, const void* k_new, const void* v_new, const void* k_past, const void* v_past, void* k_out, void* v_out,
                              void* o, int B, int A, int past, int d, const long* q_st, const long* kn_st, const long* vn_st, const long* kp_st,
                              const long* vp_st, float scale, const uint32_t* mask, const float* fill, long mask_b, long mask_a, cudaStream_t s) {
  if (B <= 0 || A <= 0 || past < 0 || d < 8 || d > 256 || d % 8 || B > 65535 || A > 65535 || !(scale > 0.f)) return -1;
  using T = const __nv_bfloat16*;
  lb::DecodeParams p{};
  p.q = (T)q; p.k_new = (T)k_new; p.v_new = (T)v_new; p.k_past = (T)k_past; p.v_past = (T)v_past;
  p.k_out = (__nv_bfloat16*)k_out; p.v_out = (__nv_bfloat16*)v_out; p.o = (__nv_bfloat16*)o;
  long any = 0;
  for (int i = 0; i < 2; ++i) {
    p.q_st[i] = q_st[i]; p.kn_st[i] = kn_st[i]; p.vn_st[i] = vn_st[i];
    any |= q_st[i] | kn_st[i] | vn_st[i];
  }
  for (int i = 0; i < 3; ++i) {
    p.kp_st[i] = kp_st[i]; p.vp_st[i] = vp_st[i];
    any |= kp_st[i] | vp_st[i];
  }
  const uintptr_t ptrs = (uintptr_t)q | (uintptr_t)k_new | (uintptr_t)v_new | (uintptr_t)k_past | (uintptr_t)v_past | (uintptr_t)k_out | (uintptr_t)v_out;
  if ((any & 7) || (ptrs & 15)) return -3;
  p.A = A; p.past = past; p.d = d;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.mask = mask; p.fill = fill; p.mask_b = mask_b; p.mask_a = mask_a;
  p.pitch = (past + 1 + 127) / 128 * 4;
  int cluster = 1;
  while (cluster < 8 && (long)B * A * cluster < 3L * 148 && (past + 1) / (cluster * 2) >= 64) cluster *= 2;
  cudaError_t e;
  if (d <= 8) e = lb::launch_attn_decode<1>(p, B, cluster, s);
  else if (d <= 16) e = lb::launch_attn_decode<2>(p, B, cluster, s);
  else if (d <= 32) e = lb::launch_attn_decode<4>(p, B, cluster, s);
  else if (d <= 64) e = lb::launch_attn_decode<8>(p, B, cluster, s);
  else if (d <= 128) e = lb::launch_attn_decode<16>(p, B, cluster, s);
  else e = lb::launch_attn_decode<32>(p, B, cluster, s);
  return (int)e;
}

// Sequence-mixer kernels for ragged batches with per-sequence state: zero-centred RMS norms on an fp32 residual stream,
// short causal convolutions with carried tails, the gated delta rule (one decay per head or per key channel) with its
// fp32 state, and sliding-window attention over cached low-rank latents (expanded keys/values for prompts, the
// absorbed form for single-token steps).
//
// Conventions.  A step carries B sequences; sequence b brings n_b = seq_off[b+1]-seq_off[b] new tokens that sit
// packed (no padding) at rows seq_off[b]..seq_off[b+1]-1 of every activation matrix, has past[b] tokens already
// folded into the state that lives in slot slots[b], and starts from an all-zero state when past[b] == 0 (the slot's
// old contents are then never read, so a slot can be reused without clearing it).  Activations are `T` (float or
// bf16, `dtype` 0 / 1); everything that enters a norm, a softmax or a recurrence is converted to fp32 first and the
// arithmetic is fp32.  This file is built WITHOUT fast-math: the fp32 mode is meant to be exact to rounding.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"

typedef __nv_bfloat16 bf16;

namespace {

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, m));
  return v;
}
// sum over the block (blockDim.x a multiple of 32, at most 1024); every thread gets the result
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float softplusf_(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// ------------------------------------------------------------------------------------------------------------------
// RMS norm: y = x / sqrt(mean(x^2) + eps) * (offset + w).  One block per row.  Optional gather of the row through
// `ids` (token embedding + norm in one pass).
// ------------------------------------------------------------------------------------------------------------------
template <typename Tin, typename Tw, typename Tout>
__global__ void rmsnorm_kernel(const Tin* __restrict__ x, long ldx, const int64_t* __restrict__ ids, const Tw* __restrict__ w,
                               float offset, float eps, Tout* __restrict__ y, long ldy, int n) {
  __shared__ float red[32];
  const long row = blockIdx.x;
  const Tin* xr = x + (ids ? (long)ids[row] : row) * ldx;
  float ss = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) { float v = ldf(xr + i); ss += v * v; }
  ss = block_sum(ss, red);
  const float r = 1.f / sqrtf(ss / (float)n + eps);
  for (int i = threadIdx.x; i < n; i += blockDim.x) stf(y + row * ldy + i, ldf(xr + i) * r * (offset + ldf(w + i)));
}

// out[row, 0:n] = act(in[row, 0:n]) on column slices; act 0: copy, 1: relu(x)^2, 2: silu, 3: gelu_tanh
template <typename Tin, typename Tout>
__global__ void slice_act_kernel(const Tin* __restrict__ in, long ldi, Tout* __restrict__ out, long ldo, long rows, int n, int act) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * n) return;
  const long r = idx / n; const int c = (int)(idx - r * n);
  float v = ldf(in + r * ldi + c);
  if (act == 1) { v = fmaxf(v, 0.f); v = v * v; }
  else if (act == 2) v = v * sigmoidf_(v);
  else if (act == 3) v = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
  stf(out + r * ldo + c, v);
}

// the same on bf16 with 16-byte accesses: 8 columns per thread (n, both row strides and both base addresses multiples of 8 elements)
__global__ void slice_act_vec8_kernel(const __nv_bfloat16* __restrict__ in, long ldi, __nv_bfloat16* __restrict__ out, long ldo,
                                      long rows, int n8, int act) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * n8) return;
  const long r = idx / n8; const int c = (int)(idx - r * n8) * 8;
  uint4 raw = *reinterpret_cast<const uint4*>(in + r * ldi + c);
  __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 v = __bfloat1622float2(h2[i]);
    if (act == 1) { v.x = fmaxf(v.x, 0.f); v.x *= v.x; v.y = fmaxf(v.y, 0.f); v.y *= v.y; }
    else if (act == 2) { v.x = v.x * sigmoidf_(v.x); v.y = v.y * sigmoidf_(v.y); }
    else if (act == 3) {
      v.x = 0.5f * v.x * (1.f + tanhf(0.7978845608028654f * (v.x + 0.044715f * v.x * v.x * v.x)));
      v.y = 0.5f * v.y * (1.f + tanhf(0.7978845608028654f * (v.y + 0.044715f * v.y * v.y * v.y)));
    }
    h2[i] = __floats2bfloat162_rn(v.x, v.y);
  }
  *reinterpret_cast<uint4*>(out + r * ldo + c) = raw;
}

// ------------------------------------------------------------------------------------------------------------------
// Short causal convolution per channel + SiLU.  in: [tokens, ldi] (C channels from column 0), w: [C, taps] with the
// last tap on the current token, tail: [slots, taps-1, C] = the last taps-1 inputs of every sequence.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void short_conv_kernel(const T* __restrict__ in, long ldi, const T* __restrict__ w, const T* __restrict__ tail,
                                  const int* __restrict__ tok_seq, const int* __restrict__ seq_off, const int* __restrict__ slots,
                                  const int* __restrict__ past, T* __restrict__ out, long ldo, long tokens, int C, int taps) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= tokens * C) return;
  const long tok = idx / C; const int c = (int)(idx - tok * C);
  const int b = tok_seq[tok];
  const int t = (int)(tok - seq_off[b]);
  const bool has_past = past[b] > 0;
  const T* tl = tail + (long)slots[b] * (taps - 1) * C;
  float acc = 0.f;
  for (int k = 0; k < taps; ++k) {
    const int tp = t - k;
    float v;
    if (tp >= 0) v = ldf(in + (tok - k) * ldi + c);
    else v = has_past ? ldf(tl + (long)(taps - 1 + tp) * C + c) : 0.f;
    acc += ldf(w + (long)c * taps + (taps - 1 - k)) * v;
  }
  stf(out + tok * ldo + c, acc * sigmoidf_(acc));
}

// bf16 with 16-byte accesses: a thread owns 8 adjacent channels of one token (C, the row strides and the base addresses are
// multiples of 8 elements); the 8·TAPS weights of its channels are contiguous and come in as TAPS 16-byte loads
template <int TAPS>
__global__ void short_conv_vec8_kernel(const __nv_bfloat16* __restrict__ in, long ldi, const __nv_bfloat16* __restrict__ w,
                                       const __nv_bfloat16* __restrict__ tail, const int* __restrict__ tok_seq,
                                       const int* __restrict__ seq_off, const int* __restrict__ slots, const int* __restrict__ past,
                                       __nv_bfloat16* __restrict__ out, long ldo, long tokens, int C) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int C8 = C >> 3;
  if (idx >= tokens * C8) return;
  const long tok = idx / C8; const int c = (int)(idx - tok * C8) * 8;
  const int b = tok_seq[tok];
  const int t = (int)(tok - seq_off[b]);
  const bool has_past = past[b] > 0;
  const __nv_bfloat16* tl = tail + (long)slots[b] * (TAPS - 1) * C;
  uint4 wraw[TAPS];
#pragma unroll
  for (int k = 0; k < TAPS; ++k) wraw[k] = reinterpret_cast<const uint4*>(w + (long)c * TAPS)[k];
  const __nv_bfloat16* wv = reinterpret_cast<const __nv_bfloat16*>(wraw);      // wv[i * TAPS + j]: channel c + i, tap j
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
  for (int k = 0; k < TAPS; ++k) {
    const int tp = t - k;
    uint4 raw = make_uint4(0u, 0u, 0u, 0u);
    if (tp >= 0) raw = *reinterpret_cast<const uint4*>(in + (tok - k) * ldi + c);
    else if (has_past) raw = *reinterpret_cast<const uint4*>(tl + (long)(TAPS - 1 + tp) * C + c);
    const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __bfloat162float(wv[i * TAPS + (TAPS - 1 - k)]) * __bfloat162float(x[i]);
  }
  uint4 res;
  __nv_bfloat162* r2 = reinterpret_cast<__nv_bfloat162*>(&res);
#pragma unroll
  for (int i = 0; i < 4; ++i) r2[i] = __floats2bfloat162_rn(acc[2 * i] * sigmoidf_(acc[2 * i]), acc[2 * i + 1] * sigmoidf_(acc[2 * i + 1]));
  *reinterpret_cast<uint4*>(out + tok * ldo + c) = res;
}

// The same for strips of STRIP tokens: the weights and the taps - 1 inputs before a token stay in registers, so an input is read 1 + 3 / STRIP
// times instead of four and the weights (64 bytes per 16 of the result) once per strip.  [2560, 4096]: 31 -> 20 us; what is left are the
// sigmoids in IEEE arithmetic (22 of 33 instructions per element; 42 % of the issue slots at [3027, 4096]).  There the strip's inputs ahead of the weights
// where it lies inside one sequence, quotients in 32 bits and six blocks per SM took 26.0 -> 24.5 us, the chained launch 2 us more.
constexpr int CONV_STRIP = 4;
template <int TAPS>
__global__ void __launch_bounds__(128, 6)
short_conv_strip_kernel(const __nv_bfloat16* __restrict__ in, long ldi, const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ tail,
                        const int* __restrict__ tok_seq, const int* __restrict__ seq_off, const int* __restrict__ slots, const int* __restrict__ past,
                        __nv_bfloat16* __restrict__ out, long ldo, long tokens, int C) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int C8 = C >> 3;
  const long strip = idx <= 0xffffffffL ? (unsigned)idx / (unsigned)C8 : idx / C8, tok0 = strip * CONV_STRIP;
  const int c = (int)(idx - strip * C8) * 8;
  lb::chain_wait(in, w, tail, tok_seq, seq_off, slots, past);
  lb::chain_next();
  if (tok0 >= tokens) return;
  float wf[TAPS][8];                         // tap j of channel c + i
  uint4 x[TAPS - 1 + CONV_STRIP];            // the input j - (TAPS - 1) tokens behind the first
  const int last = (int)(tokens - tok0 < CONV_STRIP ? tokens - tok0 : CONV_STRIP), b0 = tok_seq[tok0], t0 = (int)(tok0 - seq_off[b0]);
  const bool inside = last == CONV_STRIP && t0 >= TAPS - 1 && tok_seq[tok0 + CONV_STRIP - 1] == b0;
  if (inside) {                              // one sequence, and nothing from before the call: all loads at once
#pragma unroll
    for (int j = 0; j < TAPS - 1 + CONV_STRIP; ++j) x[j] = *reinterpret_cast<const uint4*>(in + (tok0 + j - (TAPS - 1)) * ldi + c);
  }
  {
    uint4 raw[TAPS];
#pragma unroll
    for (int k = 0; k < TAPS; ++k) raw[k] = reinterpret_cast<const uint4*>(w + (long)c * TAPS)[k];
    const __nv_bfloat16* wv = reinterpret_cast<const __nv_bfloat16*>(raw);
#pragma unroll
    for (int j = 0; j < TAPS; ++j)
#pragma unroll
      for (int i = 0; i < 8; ++i) wf[j][i] = __bfloat162float(wv[i * TAPS + j]);
  }
  auto token = [&](long tok, const uint4* at) {              // at[j]: the input under tap j
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
    for (int k = 0; k < TAPS; ++k) {
      const uint32_t xv[4] = {at[TAPS - 1 - k].x, at[TAPS - 1 - k].y, at[TAPS - 1 - k].z, at[TAPS - 1 - k].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[2 * i] += wf[TAPS - 1 - k][2 * i] * __uint_as_float(xv[i] << 16);
        acc[2 * i + 1] += wf[TAPS - 1 - k][2 * i + 1] * __uint_as_float(xv[i] & 0xffff0000u);
      }
    }
    uint4 res;
    __nv_bfloat162* r2 = reinterpret_cast<__nv_bfloat162*>(&res);
#pragma unroll
    for (int i = 0; i < 4; ++i) r2[i] = __floats2bfloat162_rn(acc[2 * i] * sigmoidf_(acc[2 * i]), acc[2 * i + 1] * sigmoidf_(acc[2 * i + 1]));
    *reinterpret_cast<uint4*>(out + tok * ldo + c) = res;
  };
  if (inside) {
#pragma unroll
    for (int j = 0; j < CONV_STRIP; ++j) token(tok0 + j, x + j);
    return;
  }
  for (int j = 0; j < last; ++j) {
    const long tok = tok0 + j;
    const int b = tok_seq[tok], t = (int)(tok - seq_off[b]);
    const bool has_past = past[b] > 0;
    const __nv_bfloat16* tl = tail + (long)slots[b] * (TAPS - 1) * C;
#pragma unroll
    for (int k = 0; k < TAPS; ++k) {
      uint4 raw = make_uint4(0u, 0u, 0u, 0u);
      if (t - k >= 0) raw = *reinterpret_cast<const uint4*>(in + (tok - k) * ldi + c);
      else if (has_past) raw = *reinterpret_cast<const uint4*>(tl + (long)(TAPS - 1 + t - k) * C + c);
      x[TAPS - 1 - k] = raw;
    }
    token(tok, x);
  }
}

template <typename T>
__global__ void conv_tail_kernel(const T* __restrict__ in, long ldi, T* __restrict__ tail, const int* __restrict__ seq_off,
                                 const int* __restrict__ slots, const int* __restrict__ past, int B, int C, int taps) {
  lb::chain_wait(in, tail, seq_off, slots, past);
  lb::chain_next();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)B * C) return;
  const int b = (int)(idx / C), c = (int)(idx - (long)b * C);
  const int n = seq_off[b + 1] - seq_off[b];
  const bool has_past = past[b] > 0;
  T* tl = tail + (long)slots[b] * (taps - 1) * C;
  for (int i = 0; i < taps - 1; ++i) {          // ascending: new[i] only reads old[i + n], never a rewritten entry
    const int tp = n - (taps - 1) + i;
    float v;
    if (tp >= 0) v = ldf(in + ((long)seq_off[b] + tp) * ldi + c);
    else v = (has_past && i + n < taps - 1) ? ldf(tl + (long)(i + n) * C + c) : 0.f;
    stf(tl + (long)i * C + c, v);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Gated delta rule.  Per head, with S [D, V] in fp32:   S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;
// o = S^T q.  q and k arrive after the convolution, are normalised here to unit length per head (eps inside the
// root) and q is scaled by D^-1/2.  g = exp(-exp(A_log) softplus(a + dt_bias)) per head (chan == 0) or per key channel
// (chan == 1); beta = sigmoid(b).  Columns of S are independent: a block owns `VT` of them for one (sequence, head);
// every column is shared by R lanes (R a power of two, adjacent lanes of one warp) that each keep DPT consecutive rows
// of it in registers, so a token costs 3·DPT fused multiply-adds per lane and log2(R) shuffle rounds.  A first kernel
// prepares the per-token quantities (unit vectors, decays, write strengths) once; the scan stages them
// through shared memory `CT` at a time (rows of lane r at offset r·(DPT+4): 16-byte loads without bank conflicts), so
// the serial part only touches registers and shared memory.
// ------------------------------------------------------------------------------------------------------------------
constexpr int CT = 16;

// Per token: unit-length keys and queries (queries also times D^-1/2) per key head in fp32, their dot product, the write
// strength beta = sigmoid(b) and the decay g per head (or per head and key channel).  One warp per (token, key head);
// the value heads of a group share its work.
template <typename T>
__global__ void delta_prep_kernel(const T* __restrict__ qkv, long ldq, int koff, const T* __restrict__ a, long lda,
                                  const T* __restrict__ bl, long ldb, const T* __restrict__ A_log, const T* __restrict__ dt_bias,
                                  float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ kq, float* __restrict__ g,
                                  float* __restrict__ beta, long tokens, int H, int KH, int D, int chan) {
  const long wid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= tokens * KH) return;
  const long tok = wid / KH; const int kh = (int)(wid - tok * KH);
  const T* qr = qkv + tok * ldq + kh * D; const T* kr = qkv + tok * ldq + koff + kh * D;
  float qq = 0.f, kk = 0.f;
  for (int i = lane; i < D; i += 32) { const float x = ldf(qr + i), y = ldf(kr + i); qq += x * x; kk += y * y; }
  qq = warp_sum(qq); kk = warp_sum(kk);
  const float qsc = (1.f / sqrtf((float)D)) / sqrtf(qq + 1e-6f), ksc = 1.f / sqrtf(kk + 1e-6f);
  float dot = 0.f;
  for (int i = lane; i < D; i += 32) {
    const float x = ldf(qr + i) * qsc, y = ldf(kr + i) * ksc;
    qn[(tok * KH + kh) * D + i] = x; kn[(tok * KH + kh) * D + i] = y; dot += x * y;
  }
  dot = warp_sum(dot);
  if (lane == 0) kq[tok * KH + kh] = dot;
  const int group = H / KH;
  for (int hh = 0; hh < group; ++hh) {
    const int h = kh * group + hh;
    const float rate = expf(ldf(A_log + h));
    if (chan) {
      for (int i = lane; i < D; i += 32)
        g[(tok * H + h) * D + i] = expf(-rate * softplusf_(ldf(a + tok * lda + h * D + i) + ldf(dt_bias + h * D + i)));
    } else if (lane == 0) {
      g[tok * H + h] = expf(-rate * softplusf_(ldf(a + tok * lda + h) + ldf(dt_bias + h)));
    }
    if (lane == 0) beta[tok * H + h] = sigmoidf_(ldf(bl + tok * ldb + h));
  }
}

template <typename T, int DPT>
__global__ void __launch_bounds__(256, DPT <= 16 ? 2 : 1)   // two blocks per SM where 128 registers hold the rows
delta_scan_kernel(const T* __restrict__ qkv, long ldq, int voff, const float* __restrict__ qn, const float* __restrict__ kn,
                  const float* __restrict__ kqs, const float* __restrict__ gs, const float* __restrict__ betas,
                  float* __restrict__ S, const int* __restrict__ seq_off, const int* __restrict__ slots,
                  const int* __restrict__ past, float* __restrict__ out, int H, int KH, int D, int V, int R, int VT, int chan) {
  extern __shared__ __align__(16) float sm[];
  constexpr int PS = DPT + 4;                   // padded stride of one lane's rows
  const int b = blockIdx.x / H, h = blockIdx.x % H, kh = h / (H / KH);
  const int j0 = blockIdx.y * VT;
  const int Dr = R * DPT;                       // rows covered (rows >= D hold zeros)
  const int Dp = R * PS;                        // floats per staged token
  float* sk = sm;                               // [CT][Dp]
  float* sq = sk + CT * Dp;                     // [CT][Dp]
  float* sg = sq + CT * Dp;                     // [CT][Dp] (chan) or [CT]
  float* sv = sg + CT * (chan ? Dp : 4);        // [CT][VT]
  float* sbeta = sv + CT * VT;                  // [CT]
  float* skq = sbeta + CT;                      // [CT]
  const int tid = threadIdx.x, nth = blockDim.x;
  const int r = tid % R, jj = tid / R, j = j0 + jj;
  const bool col_ok = jj < VT && j < V;
  const int n = seq_off[b + 1] - seq_off[b];
  const long tok0 = seq_off[b];
  float* Sg = S + ((long)slots[b] * H + h) * (long)D * V;
  float s[DPT];
#pragma unroll
  for (int d = 0; d < DPT; ++d) {
    const int i = r * DPT + d;
    s[d] = (past[b] > 0 && col_ok && i < D) ? Sg[(long)i * V + j] : 0.f;
  }
  for (int c0 = 0; c0 < n; c0 += CT) {
    const int ct = min(CT, n - c0);
    __syncthreads();
    for (int e = tid; e < ct * Dr; e += nth) {
      const int t = e / Dr, i = e - t * Dr;
      const int pos = t * Dp + (i / DPT) * PS + (i % DPT);
      const long row = tok0 + c0 + t;
      const bool in = i < D;
      sk[pos] = in ? kn[(row * KH + kh) * D + i] : 0.f;
      sq[pos] = in ? qn[(row * KH + kh) * D + i] : 0.f;
      if (chan) sg[pos] = in ? gs[(row * H + h) * D + i] : 1.f;
    }
    for (int e = tid; e < ct * VT; e += nth) {
      const int t = e / VT, c = e - t * VT;
      sv[e] = (j0 + c < V) ? ldf(qkv + (tok0 + c0 + t) * ldq + voff + h * V + j0 + c) : 0.f;
    }
    for (int t = tid; t < ct; t += nth) {
      const long row = tok0 + c0 + t;
      sbeta[t] = betas[row * H + h];
      skq[t] = kqs[row * KH + kh];
      if (!chan) sg[t] = gs[row * H + h];
    }
    __syncthreads();
    // every thread walks the tokens (lanes of idle columns included: the shuffles below name the whole warp)
    for (int t = 0; t < ct; ++t) {
      float kr[DPT];
      float pk[4] = {0.f, 0.f, 0.f, 0.f}, pq[4] = {0.f, 0.f, 0.f, 0.f};
      const float4* k4 = reinterpret_cast<const float4*>(sk + t * Dp + r * PS);
      const float4* q4 = reinterpret_cast<const float4*>(sq + t * Dp + r * PS);
      const float4* g4 = reinterpret_cast<const float4*>(sg + t * Dp + r * PS);
      const float g0 = chan ? 1.f : sg[t];
#pragma unroll
      for (int d4 = 0; d4 < DPT / 4; ++d4) {
        const float4 kx = k4[d4], qx = q4[d4];
        float4 gx = make_float4(g0, g0, g0, g0);
        if (chan) gx = g4[d4];
        kr[4 * d4] = kx.x; kr[4 * d4 + 1] = kx.y; kr[4 * d4 + 2] = kx.z; kr[4 * d4 + 3] = kx.w;
        s[4 * d4] *= gx.x; s[4 * d4 + 1] *= gx.y; s[4 * d4 + 2] *= gx.z; s[4 * d4 + 3] *= gx.w;
        pk[0] += s[4 * d4] * kx.x; pk[1] += s[4 * d4 + 1] * kx.y; pk[2] += s[4 * d4 + 2] * kx.z; pk[3] += s[4 * d4 + 3] * kx.w;
        pq[0] += s[4 * d4] * qx.x; pq[1] += s[4 * d4 + 1] * qx.y; pq[2] += s[4 * d4 + 2] * qx.z; pq[3] += s[4 * d4 + 3] * qx.w;
      }
      float sk_ = (pk[0] + pk[1]) + (pk[2] + pk[3]), sq_ = (pq[0] + pq[1]) + (pq[2] + pq[3]);
      for (int m = R >> 1; m > 0; m >>= 1) { sk_ += __shfl_xor_sync(0xffffffffu, sk_, m); sq_ += __shfl_xor_sync(0xffffffffu, sq_, m); }
      const float u = sbeta[t] * ((jj < VT ? sv[t * VT + jj] : 0.f) - sk_);
#pragma unroll
      for (int d = 0; d < DPT; ++d) s[d] += kr[d] * u;
      if (r == 0 && col_ok) out[(tok0 + c0 + t) * (long)(H * V) + h * V + j] = sq_ + skq[t] * u;
    }
  }
  if (col_ok) {
#pragma unroll
    for (int d = 0; d < DPT; ++d) { const int i = r * DPT + d; if (i < D) Sg[(long)i * V + j] = s[d]; }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// The same scan for one decay per head, two tokens at a time.  With k0, k1, q0, q1 the unit keys and queries of two consecutive
// tokens, all four products with the state are taken on the state before them, and two inner products (k1·k0, q1·k0) carry the
// first token's write over to the second:
//   u0 = b0 (v0 - g0 k0ᵀS);                          o0 = g0 q0ᵀS + (q0·k0) u0
//   u1 = b1 (v1 - g1 (g0 k1ᵀS + (k1·k0) u0));        o1 = g1 (g0 q1ᵀS + (q1·k0) u0) + (q1·k1) u1
//   S <- g0 g1 S + g1 k0 u0ᵀ + k1 u1ᵀ
// Everything stays fp32.  The scan is a serial chain over the tokens, bounded by the latency of one link and by the issue of its
// multiply-adds, so: one reduction and one scaling of the state per two tokens instead of per token; packed pairs of fp32
// (fma.rn.f32x2); four lanes per column with CPT columns each, so that a staged vector is read once for CPT columns (with eight
// lanes and one column per lane the 16-byte shared-memory reads took most of a token's 1370 cycles); the next tokens arrive by
// cp.async meanwhile.  [2560 tokens of 4 sequences up to 1024, 16 heads, 128 x 128]: 755 -> 330 us (one column per lane:
// 434 us).
// Lane r of a column holds rows 16 d + 4 r + 0..3: the four lanes read 64 contiguous bytes.
// ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ void unpack2(unsigned long long a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a)); }
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {        // the rest of the 16 is zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(bytes));
}

constexpr int PAIR_THREADS = 128;
// floats of shared memory: two buffers of k, q, v for CT tokens, and of their scalars (beta, g, q·k, then k1·k0 and q1·k0 per pair)
constexpr int pair_buffer_floats(int rows, int cols) { return CT * rows * 2 + CT * cols; }
constexpr int pair_smem_floats(int rows, int cols) { return 2 * (pair_buffer_floats(rows, cols) + 4 * CT); }

// D <= 16 D4 rows (D % 4 == 0), 32 CPT columns per block; v's rows in whole aligned 16-byte vectors
template <typename T, int D4, int CPT>
__global__ void __launch_bounds__(PAIR_THREADS)
delta_scan_pair_kernel(const T* __restrict__ qkv, long ldq, int voff, const float* __restrict__ qn, const float* __restrict__ kn,
                       const float* __restrict__ kqs, const float* __restrict__ gs, const float* __restrict__ betas,
                       float* __restrict__ S, const int* __restrict__ seq_off, const int* __restrict__ slots,
                       const int* __restrict__ past, float* __restrict__ out, int H, int KH, int D, int V, int shorter_than) {
  constexpr int DP = 16 * D4, VB = 32 * CPT, BUF = pair_buffer_floats(DP, VB), VE = 16 / sizeof(T);
  extern __shared__ __align__(16) float sm[];
  float* scal = sm + 2 * BUF;
  const int tid = threadIdx.x, r = tid & 3, cg = tid >> 2, bit0 = r & 1;
  const int b = blockIdx.x / H, h = blockIdx.x % H, kh = h / (H / KH), j0 = blockIdx.y * VB;
  const int n = seq_off[b + 1] - seq_off[b];
  if (n >= shorter_than) return;
  const long tok0 = seq_off[b];
  float* Sg = S + ((long)slots[b] * H + h) * (long)D * V;
  const int jc = j0 + cg * CPT;
  unsigned long long s[CPT][2 * D4];
#pragma unroll
  for (int d = 0; d < D4; ++d) {
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = d * 16 + r * 4 + e;
        x[e] = (past[b] > 0 && jc + c < V && i < D) ? Sg[(long)i * V + jc + c] : 0.f;
      }
      s[c][2 * d] = pack2(x[0], x[1]);
      s[c][2 * d + 1] = pack2(x[2], x[3]);
    }
  }
  auto stage = [&](int c0, int buf) {
    const int ct = min(CT, n - c0);
    float* sk = sm + buf * BUF;
    float* sq = sk + CT * DP;
    T* sv = reinterpret_cast<T*>(sq + CT * DP);
    float* sc = scal + buf * 4 * CT;
    for (int e = tid; e < CT * DP / 4; e += PAIR_THREADS) {
      const int t = e / (DP / 4), i = (e % (DP / 4)) * 4;
      const bool in = t < ct && i < D;
      const long at = in ? ((tok0 + c0 + t) * KH + kh) * (long)D + i : 0;
      cp_async16(sk + t * DP + i, kn + at, in ? 16 : 0);
      cp_async16(sq + t * DP + i, qn + at, in ? 16 : 0);
    }
    for (int e = tid; e < CT * VB / VE; e += PAIR_THREADS) {
      const int t = e / (VB / VE), c = (e % (VB / VE)) * VE;
      const bool in = t < ct && j0 + c < V;
      cp_async16(sv + t * VB + c, in ? qkv + (tok0 + c0 + t) * ldq + voff + (long)h * V + j0 + c : qkv, in ? 16 : 0);
    }
    if (tid < CT) {
      const bool in = tid < ct;
      const long row = in ? tok0 + c0 + tid : tok0;
      cp_async4(sc + tid, betas + row * H + h, in ? 4 : 0);
      cp_async4(sc + CT + tid, gs + row * H + h, in ? 4 : 0);
      cp_async4(sc + 2 * CT + tid, kqs + row * KH + kh, in ? 4 : 0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  stage(0, 0);
  for (int c0 = 0, buf = 0; c0 < n; c0 += CT, buf ^= 1) {
    const int ct = min(CT, n - c0);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();                              // the tokens are here, and nobody reads the other buffer any more
    if (c0 + CT < n) stage(c0 + CT, buf ^ 1);
    const float* sk = sm + buf * BUF;
    const float* sq = sk + CT * DP;
    const T* sv = reinterpret_cast<const T*>(sq + CT * DP);
    float* sc = scal + buf * 4 * CT;
    for (int p = tid >> 5; p < CT / 2; p += PAIR_THREADS / 32) {     // inner products between the tokens of a pair, one pair per warp
      const int lane = tid & 31;
      float kk = 0.f, qk = 0.f;
      for (int i = lane * 4; i < DP; i += 128) {
        const float4 k0 = *reinterpret_cast<const float4*>(sk + 2 * p * DP + i), k1 = *reinterpret_cast<const float4*>(sk + (2 * p + 1) * DP + i),
                     q1 = *reinterpret_cast<const float4*>(sq + (2 * p + 1) * DP + i);
        kk += (k1.x * k0.x + k1.y * k0.y) + (k1.z * k0.z + k1.w * k0.w);
        qk += (q1.x * k0.x + q1.y * k0.y) + (q1.z * k0.z + q1.w * k0.w);
      }
      kk = warp_sum(kk);
      qk = warp_sum(qk);
      if (lane == 0) { sc[3 * CT + 2 * p] = kk; sc[3 * CT + 2 * p + 1] = qk; }
    }
    __syncthreads();
    auto pair = [&](int t, auto two_tag) {
      const ulonglong2* k0p = reinterpret_cast<const ulonglong2*>(sk + t * DP) + r;
      const ulonglong2* k1p = reinterpret_cast<const ulonglong2*>(sk + (t + 1) * DP) + r;
      const ulonglong2* q0p = reinterpret_cast<const ulonglong2*>(sq + t * DP) + r;
      const ulonglong2* q1p = reinterpret_cast<const ulonglong2*>(sq + (t + 1) * DP) + r;
      unsigned long long acc[CPT][4];
#pragma unroll
      for (int c = 0; c < CPT; ++c)
#pragma unroll
        for (int m = 0; m < 4; ++m) acc[c][m] = 0ull;
      ulonglong2 K0[D4], K1[D4];
#pragma unroll
      for (int d = 0; d < D4; ++d) {
        K0[d] = k0p[d * 4];
        K1[d] = k1p[d * 4];
        const ulonglong2 Q0 = q0p[d * 4], Q1 = q1p[d * 4];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          acc[c][0] = fma2(K0[d].x, s[c][2 * d], acc[c][0]);
          acc[c][1] = fma2(Q0.x, s[c][2 * d], acc[c][1]);
          acc[c][2] = fma2(K1[d].x, s[c][2 * d], acc[c][2]);
          acc[c][3] = fma2(Q1.x, s[c][2 * d], acc[c][3]);
          acc[c][0] = fma2(K0[d].y, s[c][2 * d + 1], acc[c][0]);
          acc[c][1] = fma2(Q0.y, s[c][2 * d + 1], acc[c][1]);
          acc[c][2] = fma2(K1[d].y, s[c][2 * d + 1], acc[c][2]);
          acc[c][3] = fma2(Q1.y, s[c][2 * d + 1], acc[c][3]);
        }
      }
      // sums over the four lanes; with two columns the even lanes end up with the first, the odd ones with the second
      float w[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        float x, y, a0, a1 = 0.f;
        unpack2(acc[0][m], x, y);
        a0 = x + y;
        if constexpr (CPT == 2) {
          unpack2(acc[CPT - 1][m], x, y);
          a1 = x + y;
          const float keep = bit0 ? a1 : a0, send = bit0 ? a0 : a1;
          w[m] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        } else {
          w[m] = a0 + __shfl_xor_sync(0xffffffffu, a0, 1);
        }
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) w[m] += __shfl_xor_sync(0xffffffffu, w[m], 2);
      constexpr bool two = decltype(two_tag)::value;   // the last of an odd number of tokens: no second decay, no second write (0 times what is not finite)
      const float b0 = sc[t], b1 = sc[t + 1], g0 = sc[CT + t], g1 = two ? sc[CT + t + 1] : 1.f, kq0 = sc[2 * CT + t], kq1 = sc[2 * CT + t + 1];
      const float kk = sc[3 * CT + t], qk = sc[3 * CT + t + 1];
      const int vc = cg * CPT + (CPT == 2 ? bit0 : 0);
      const float u0 = b0 * (ldf(sv + t * VB + vc) - g0 * w[0]);
      const float o0 = g0 * w[1] + kq0 * u0;
      const float u1 = b1 * (ldf(sv + (t + 1) * VB + vc) - g1 * (g0 * w[2] + kk * u0));
      const float o1 = g1 * (g0 * w[3] + qk * u0) + kq1 * u1;
      const float gg = g0 * g1, w0 = g1 * u0;
      const unsigned long long G = pack2(gg, gg);
      float U0[CPT], U1[CPT];
      if constexpr (CPT == 2) {
        const float x0 = __shfl_xor_sync(0xffffffffu, w0, 1), x1 = __shfl_xor_sync(0xffffffffu, u1, 1);
        U0[0] = bit0 ? x0 : w0;
        U1[0] = bit0 ? x1 : u1;
        U0[CPT - 1] = bit0 ? w0 : x0;
        U1[CPT - 1] = bit0 ? u1 : x1;
      } else {
        U0[0] = w0;
        U1[0] = u1;
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const unsigned long long p0 = pack2(U0[c], U0[c]);
        [[maybe_unused]] const unsigned long long p1 = pack2(U1[c], U1[c]);
#pragma unroll
        for (int d = 0; d < D4; ++d) {
          s[c][2 * d] = fma2(K0[d].x, p0, mul2(s[c][2 * d], G));
          s[c][2 * d + 1] = fma2(K0[d].y, p0, mul2(s[c][2 * d + 1], G));
          if constexpr (two) {
            s[c][2 * d] = fma2(K1[d].x, p1, s[c][2 * d]);
            s[c][2 * d + 1] = fma2(K1[d].y, p1, s[c][2 * d + 1]);
          }
        }
      }
      if (r < CPT && j0 + vc < V) {
        float* o = out + (tok0 + c0 + t) * (long)(H * V) + (long)h * V + j0 + vc;
        o[0] = o0;
        if (two) o[(long)H * V] = o1;
      }
    };
    int t = 0;
    for (; t + 1 < ct; t += 2) pair(t, std::true_type{});
    if (t < ct) pair(t, std::false_type{});
  }
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    if (jc + c >= V) continue;
#pragma unroll
    for (int d = 0; d < D4; ++d) {
      float x[4];
      unpack2(s[c][2 * d], x[0], x[1]);
      unpack2(s[c][2 * d + 1], x[2], x[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = d * 16 + r * 4 + e;
        if (i < D) Sg[(long)i * V + jc + c] = x[e];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// The same recurrence for long bf16 sequences, CL tokens at a time on the tensor cores.  With G_t the product of the decays from the chunk's
// start, γ(t, s) that of s+1 .. t and S0 the state before the chunk,
//   u_t = β_t (v_t - G_t S0ᵀk_t - Σ_{s<t} γ(t, s) (k_t·k_s) u_s),   that is  U = T Y,  Y = V - G K S0,  T = (I + A)^-1 β,  A_ts = β_t γ(t, s) (k_t·k_s),
//   o_t = G_t S0ᵀq_t + Σ_{s<=t} M_ts u_s,  M_ts = γ(t, s) (q_t·k_s),                        S <- G_L S0 + Σ_s γ(L, s) k_s u_sᵀ.
// A first kernel makes T, M and the decays of all chunks at once, the second walks a sequence's chunks with the state.  There a warp owns 16 columns
// of Sᵀ in registers (accumulator layout of m16n8k16, 16 x 128 fp32), everything is transposed ([16 columns, tokens]) and each result is the
// next product's A operand, so warps share staged operands only and a chunk needs one barrier.
// Precision.  q and k are the bf16 numbers as they came; the state, Y, U, T and M are sums of three bf16 parts (24 bits).  The tensor core cuts
// its sums off at 24 bits instead of rounding them, which in a chain of such sums cost more than the scan's roundings.  So the products of
// first parts leave it step by step and are added in fp32 registers with rounding to nearest, and only those of the smaller parts (2^-8 and below;
// of two matrices in parts the last, 2^-32, is left out) are chained; T's diagonal, the largest term where decays are strong, is a
// product on the FMA pipe.  Lengths, decays, their products, beta and the entries of T and M are made once per chunk in 64 bits (1 / |k_t| is a factor of
// T's row t, so that U can be taken with the keys as they came).  Relative error against 64 bits, decays from strong to
// near one, 100 to 1024 tokens: read-outs 0.8e-7 to 1.4e-7, states 0.5e-7 to 1.4e-7 (pairs 1.0e-7 to 2.6e-6, 0.7e-7 to 3.6e-6).  With the diagonal's
// error and U as two numbers 0.7e-7 to 1.2e-7 and 0.4e-7 to 1.3e-7, but 166 instead of 128 us (registers).
// T and M end at the diagonal: 0 times what is not finite would reach earlier tokens of the column, so columns where Y or U has
// such numbers (or beyond 1e37) take these two products from plain sums over s <= t.
// The scan in pairs is a chain of 1150 cycles per two tokens on one warp per scheduler; here a warp's chunk is 384 products (192 with the state,
// 48 + 48 with T and M, 96 for the update), 6150 cycles on its scheduler's tensor core at 16 each, of 7900 that a chunk takes: the rest are
// the parts, sums and roundings between products that wait for one another, and a sequence's chunks are a chain.
// [2560 tokens of 4 sequences up to 1024, 16 heads, 128 x 128]: 339 -> 165 us with the preparations (25) and inputs from memory; eight sequences of 1024:
// 536 -> 248.  Q S0 with the state's update instead of K S0 was slower (registers).  The same in fp32 on the FMA pipe (the inverse times keys
// and values ahead of the scan, 4 x 4 tiles) took 333: 16-byte reads of shared memory bound it.
// ------------------------------------------------------------------------------------------------------------------
constexpr int CL = 32;                       // tokens per chunk
// Sequences from here on are scanned in chunks: the first length at which they are ahead or level at every size and batch.  Three chunks take what pairs
// take for 81 tokens (one sequence, 16 heads of 128 x 128: 80 tokens 26.7 in pairs, 96 31.2, three chunks 27.0 us) to 88 (8 heads of 64 x 64: 19.6, 22.8 and 21.5).
// Of many the chunks are ahead from 64 on (32 of 64: 71 against 130), but a sequence's result must not depend on the others.
constexpr int CL_MIN = 88;
constexpr int CL_LD = CL + 8;                // row stride of 32 x 32 bf16 matrices in shared memory (ldmatrix without bank conflicts)
constexpr int CL_WARPS = 4;                  // warps (of 16 columns) per block of the scan
constexpr int CL_COLS = 16 * CL_WARPS;
// scratch per (chunk, head), in floats: T and M as three bf16 parts each, then per token the factors of K S0,
// Q S0 and of u in the update and T's diagonal, then G_L
constexpr int CL_SCRATCH = 3 * CL * CL + 4 * CL + 32;

__device__ __forceinline__ uint32_t smem_at(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// a product by itself
__device__ __forceinline__ void mma16816_new(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// added to c with rounding to nearest (the tensor core's accumulator cuts off)
__device__ __forceinline__ void add_mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float y[4];
  mma16816_new(y, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; ++e) c[e] += y[e];
}
// (x, y) as the sum of three pairs of bf16 numbers, largest first
__device__ __forceinline__ void parts3(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(x, y);
    p[i] = *reinterpret_cast<const uint32_t*>(&r);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
// A operand of 16 rows and the 16 columns of two neighbouring accumulator tiles, in three parts
__device__ __forceinline__ void a_parts(const float (&l)[4], const float (&r)[4], uint32_t (&a)[3][4]) {
  uint32_t p[3];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float x = i < 2 ? l[2 * (i & 1)] : r[2 * (i & 1)], y = i < 2 ? l[2 * (i & 1) + 1] : r[2 * (i & 1) + 1];
    parts3(x, y, p);
#pragma unroll
    for (int e = 0; e < 3; ++e) a[e][i] = p[e];
  }
}

// block = (chunk, key head); heads of a group by pairs of warps in turn: one has T, the other M and the factors (both run the decays of the chunk).
// Bounded by the chain over the chunk's tokens.  Six blocks per SM (registers, 36 KB): 98 x 8 blocks are one wave instead of one and a twentieth, 29.7 -> 24 us.
template <int DP>
__global__ void __launch_bounds__(128, 6)
delta_chunk_prep_kernel(const bf16* __restrict__ qkv, long ldq, int koff, const bf16* __restrict__ a, long lda, const bf16* __restrict__ bl, long ldb,
                        const bf16* __restrict__ A_log, const bf16* __restrict__ dt_bias, const int* __restrict__ seq_off, float* __restrict__ scratch,
                        int B, int H, int KH, int D) {
  lb::chain_wait(qkv, a, bl, A_log, dt_bias, seq_off);
  lb::chain_next();
  constexpr int LD = DP + 8;
  __shared__ __align__(16) bf16 sK[CL * LD], sQ[CL * LD];
  __shared__ float sKK[CL][CL + 1], sQK[CL][CL + 1], sA[2][CL][CL + 4];
  __shared__ double ksc[CL], qsc[CL];
  __shared__ int where[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, kh = blockIdx.y;
  if (warp == 0) {                           // the chunk's sequence
    int left = blockIdx.x, found = -1;
    for (int b0 = 0; b0 < B && found < 0; b0 += 32) {
      const int b = b0 + lane, n = b < B ? seq_off[b + 1] - seq_off[b] : 0, c = n >= CL_MIN ? (n + CL - 1) / CL : 0;
      int sum = c;
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, sum, m);
        if (lane >= m) sum += x;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, sum > left);
      if (hit) {
        const int at = __ffs(hit) - 1;
        found = b0 + at;
        left -= __shfl_sync(0xffffffffu, sum - c, at);
      } else {
        left -= __shfl_sync(0xffffffffu, sum, 31);
      }
    }
    if (lane == 0) { where[0] = found; where[1] = left; }
  }
  __syncthreads();
  const int b = where[0];
  if (b < 0) return;
  const long tok0 = seq_off[b] + (long)where[1] * CL;
  const int nt = min(CL, (int)(seq_off[b + 1] - tok0));
  for (int t = tid >> 3; t < CL; t += 16) {  // rows as they are, their lengths apart; eight lanes per row
    double qq = 0.0, kk = 0.0;
    const bf16 *qr = qkv + (tok0 + t) * ldq + (long)kh * D, *kr = qr + koff;
#pragma unroll
    for (int i = (tid & 7) * 4; i < DP; i += 32) {
      uint2 x = make_uint2(0u, 0u), y = x;
      if (t < nt && i < D) { x = *reinterpret_cast<const uint2*>(qr + i); y = *reinterpret_cast<const uint2*>(kr + i); }
      *reinterpret_cast<uint2*>(sQ + t * LD + i) = x;
      *reinterpret_cast<uint2*>(sK + t * LD + i) = y;
      const uint32_t xs[2] = {x.x, x.y}, ys[2] = {y.x, y.y};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double x0 = __uint_as_float(xs[e] << 16), x1 = __uint_as_float(xs[e] & 0xffff0000u);
        const double y0 = __uint_as_float(ys[e] << 16), y1 = __uint_as_float(ys[e] & 0xffff0000u);
        qq += x0 * x0 + x1 * x1;
        kk += y0 * y0 + y1 * y1;
      }
    }
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) {
      qq += __shfl_xor_sync(0xffffffffu, qq, m);
      kk += __shfl_xor_sync(0xffffffffu, kk, m);
    }
    // lengths beyond what fp32 squares hold: such a vector counts as zero, as in the scan token by token (not where an element is infinite)
    const bool q0 = qq > FLT_MAX && qq < INFINITY, k0 = kk > FLT_MAX && kk < INFINITY;
    for (int i = (tid & 7) * 4; i < DP; i += 32) {
      if (q0) *reinterpret_cast<uint2*>(sQ + t * LD + i) = make_uint2(0u, 0u);
      if (k0) *reinterpret_cast<uint2*>(sK + t * LD + i) = make_uint2(0u, 0u);
    }
    if ((tid & 7) == 0) {
      qsc[t] = q0 ? -1.0 : qq;
      ksc[t] = k0 ? -1.0 : kk;
    }
  }
  __syncthreads();
  if (tid < 2 * CL) {                        // -0: counts as zero
    double& sc = tid < CL ? qsc[tid] : ksc[tid - CL];
    sc = sc < 0.0 ? -0.0 : 1.0 / sqrt((tid < CL ? D : 1) * (sc + 1e-6));
  }
  {                                          // K Kᵀ (warps 0, 1) and Q Kᵀ (2, 3), 16 rows per warp
    const bf16* rows = warp < 2 ? sK : sQ;
    const int r0 = (warp & 1) * 16;
    float c[4][4] = {};
#pragma unroll
    for (int k0 = 0; k0 < DP; k0 += 16) {
      uint32_t am[4];
      ldsm4(am, smem_at(rows + (r0 + (lane & 15)) * LD + k0 + (lane >> 4) * 8));
#pragma unroll
      for (int n2 = 0; n2 < 2; ++n2) {
        uint32_t bm[4];
        ldsm4(bm, smem_at(sK + (n2 * 16 + (lane & 7) + (lane >> 4) * 8) * LD + k0 + ((lane >> 3) & 1) * 8));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float x[4] = {};
          mma16816(x, am, bm[2 * i], bm[2 * i + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) c[n2 * 2 + i][e] += x[e];
        }
      }
    }
    float(*dst)[CL + 1] = warp < 2 ? sKK : sQK;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[r0 + (lane >> 2) + (e >> 1) * 8][n * 8 + (lane & 3) * 2 + (e & 1)] = c[n][e];
  }
  __syncthreads();
  const int group = H / KH;
  const bool is_m = warp & 1;                // even warps: T of a head; odd ones: M and the factors
  for (int hh = warp >> 1; hh < group; hh += 2) {
    const int h = kh * group + hh;
    float* mine = scratch + ((long)blockIdx.x * H + h) * CL_SCRATCH;
    bf16* Tp = reinterpret_cast<bf16*>(mine);
    bf16* Mp = Tp + 3 * CL * CL;
    float* fac = mine + 3 * CL * CL;
    double g = 1.0, beta = 0.0;              // of token `lane`
    if (lane < nt) {
      const double z = static_cast<double>(ldf(a + (tok0 + lane) * lda + h)) + ldf(dt_bias + h);
      g = exp(-exp(static_cast<double>(ldf(A_log + h))) * (z > 40.0 ? z : log1p(exp(z))));
      beta = 1.0 / (1.0 + exp(-static_cast<double>(ldf(bl + (tok0 + lane) * ldb + h))));
    }
    double x = 0.0;                          // γ(t, lane)
    const double ks = ksc[lane];
    auto store3 = [&](bf16* p, double v) {
      float x = static_cast<float>(v);
      const float rest = static_cast<float>(v - x);
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const bf16 r = __float2bfloat16_rn(x);
        p[e * CL * CL] = r;
        x -= __bfloat162float(r);
        if (e == 0) x += rest;
      }
    };
    if (is_m) {
      double all = 1.0, G = 1.0;             // products of all decays up to t
#pragma unroll 4
      for (int t = 0; t < CL; ++t) {
        const double gt = __shfl_sync(0xffffffffu, g, t);
        x = t == lane ? 1.0 : (t > lane ? x * gt : 0.0);
        all *= gt;
        if (t == lane) G = all;
        store3(Mp + t * CL + lane, lane <= t ? x * qsc[t] * sQK[t][lane] : 0.0);
      }
      fac[lane] = static_cast<float>(G * ks);
      fac[CL + lane] = static_cast<float>(G * qsc[lane]);
      fac[2 * CL + lane] = static_cast<float>(x);        // (tokens behind the end decay by 1)
      fac[3 * CL + lane] = static_cast<float>(beta * ks);
      if (lane == 0) fac[4 * CL] = static_cast<float>(all);
    } else {
      float(*A)[CL + 4] = sA[warp >> 1];
#pragma unroll 4
      for (int t = 0; t < CL; ++t) {
        const double gt = __shfl_sync(0xffffffffu, g, t), bt = __shfl_sync(0xffffffffu, beta, t);
        x = t == lane ? 1.0 : (t > lane ? x * gt : 0.0);
        A[t][lane] = lane < t ? static_cast<float>(bt * x * (ksc[t] * ks) * sKK[t][lane]) : 0.f;
      }
      __syncwarp();
      float col[CL];                         // column `lane` of (I + A)^-1
#pragma unroll
      for (int t = 0; t < CL; ++t) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < t; ++s) acc[s & 3] += A[t][s] * col[s];
        col[t] = t == lane ? 1.f : (t > lane ? -((acc[0] + acc[1]) + (acc[2] + acc[3])) : 0.f);
        store3(Tp + t * CL + lane, t > lane ? ksc[t] * col[t] * beta : 0.0);
      }
      __syncwarp();
    }
  }
}

template <int DP>
struct DeltaChunkStage {
  bf16 k[CL * (DP + 8)], q[CL * (DP + 8)];
  bf16 tm[6 * CL * CL_LD];                   // T, M: three parts each
  bf16 v[CL * (CL_COLS + 8)];
  float fac[4 * CL + 4];
};
template <int DP>
struct DeltaChunkSmem {
  DeltaChunkStage<DP> st[2];
  float slow[CL_WARPS][2][16][CL + 1];       // Y and U, O of columns with numbers that are not finite
};

// block = (sequence and head, CL_COLS columns)
template <int DP>
__global__ void __launch_bounds__(32 * CL_WARPS)
delta_chunk_scan_kernel(const bf16* __restrict__ qkv, long ldq, int koff, int voff, const float* __restrict__ scratch, float* __restrict__ S,
                        const int* __restrict__ seq_off, const int* __restrict__ slots, const int* __restrict__ past, float* __restrict__ out,
                        int H, int KH, int D, int V) {
  lb::chain_next();
  constexpr int LD = DP + 8, VLD = CL_COLS + 8, THREADS = 32 * CL_WARPS;
  extern __shared__ __align__(16) unsigned char delta_sm[];
  DeltaChunkSmem<DP>& sm = *reinterpret_cast<DeltaChunkSmem<DP>*>(delta_sm);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q2 = (lane & 3) * 2;
  const int b = blockIdx.x / H, h = blockIdx.x % H, kh = h / (H / KH), j0 = blockIdx.y * CL_COLS;
  const int n = seq_off[b + 1] - seq_off[b];
  if (n < CL_MIN) return;
  int before = 0;                            // chunks of the sequences before this one
  for (int i = lane; i < b; i += 32) {
    const int m = seq_off[i + 1] - seq_off[i];
    before += m >= CL_MIN ? (m + CL - 1) / CL : 0;
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) before += __shfl_xor_sync(0xffffffffu, before, m);
  const long tok0 = seq_off[b];
  const float* base = scratch + ((long)before * H + h) * CL_SCRATCH;
  const long step = (long)H * CL_SCRATCH;
  float* Sg = S + ((long)slots[b] * H + h) * (long)D * V;
  const int jc = j0 + warp * 16 + g;         // this thread's columns: jc, jc + 8
  float st[DP / 8][4];                       // Sᵀ: rows are columns of S; n-tile i, element e: row jc + 8 (e / 2), column 8 i + q2 + e % 2
#pragma unroll
  for (int i = 0; i < DP / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * i + q2 + (e & 1), col = jc + 8 * (e >> 1);
      st[i][e] = past[b] > 0 && d < D && col < V ? Sg[(long)d * V + col] : 0.f;
    }
  auto stage = [&](int c) {
    DeltaChunkStage<DP>& p = sm.st[c & 1];
    const int nt = min(CL, n - c * CL);
    const long tok = tok0 + c * CL;
    const float* w = base + c * step;
    for (int e = tid; e < CL * DP / 8; e += THREADS) {
      const int t = e / (DP / 8), i = e % (DP / 8) * 8;
      const int bytes = t < nt ? max(0, min(8, D - i)) * 2 : 0;
      const bf16* src = qkv + (bytes ? (tok + t) * ldq + (long)kh * D + i : 0);
      cp_async16(p.q + t * LD + i, src, bytes);
      cp_async16(p.k + t * LD + i, src + (bytes ? koff : 0), bytes);
    }
    for (int e = tid; e < 6 * CL * CL / 8; e += THREADS)
      cp_async16(p.tm + e / (CL / 8) * CL_LD + e % (CL / 8) * 8, reinterpret_cast<const bf16*>(w) + e * 8, 16);
    for (int e = tid; e < CL * CL_COLS / 8; e += THREADS) {
      const int t = e / (CL_COLS / 8), j = e % (CL_COLS / 8) * 8;
      const bool in = t < nt && j0 + j < V;
      cp_async16(p.v + t * VLD + j, qkv + (in ? (tok + t) * ldq + voff + (long)h * V + j0 + j : 0), in ? 16 : 0);
    }
    if (tid < (4 * CL + 4) / 4) cp_async16(p.fac + 4 * tid, w + 3 * CL * CL + 4 * tid, 16);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  const int chunks = (n + CL - 1) / CL;
  stage(0);
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();                         // the chunk is here, and nobody reads the other stage any more
    if (c + 1 < chunks) stage(c + 1);
    const DeltaChunkStage<DP>& p = sm.st[c & 1];
    const int nt = min(CL, n - c * CL);
    // ---- S0ᵀ [Kᵀ Qᵀ]: [16, 32 + 32]
    float x[8][4] = {}, xl[8][4] = {};       // sums of the first parts; of the smaller ones
#pragma unroll
    for (int kk = 0; kk < DP / 16; ++kk) {
      uint32_t am[3][4];
      a_parts(st[2 * kk], st[2 * kk + 1], am);
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) {
        uint32_t bm[4];
        ldsm4(bm, smem_at((n2 < 2 ? p.k : p.q) + ((n2 & 1) * 16 + (lane & 7) + (lane >> 4) * 8) * LD + kk * 16 + ((lane >> 3) & 1) * 8));
#pragma unroll
        for (int i = 0; i < 2; ++i) mma16816(xl[n2 * 2 + i], am[2], bm[2 * i], bm[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) add_mma16816(x[n2 * 2 + i], am[0], bm[2 * i], bm[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) mma16816(xl[n2 * 2 + i], am[1], bm[2 * i], bm[2 * i + 1]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i][e] += xl[i][e];
    // ---- Y = V - G K S0; O starts with G Q S0
    bool odd[2] = {false, false};            // columns g, g + 8 with a number that is not finite or close to that
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * i + q2 + (e & 1);
        if (__float_as_uint(p.fac[t]) == 0x80000000u) x[i][e] = 0.f;
        x[i][e] = fmaf(-p.fac[t], x[i][e], __bfloat162float(p.v[t * VLD + warp * 16 + g + 8 * (e >> 1)]));
        if (__float_as_uint(p.fac[CL + t]) == 0x80000000u) x[4 + i][e] = 0.f;
        odd[e >> 1] = odd[e >> 1] || !(fabsf(x[i][e]) < 1e37f);
      }
    float u[4][4] = {};
    {
      // D = [16, 32] (as A, three parts) times the three parts of a lower triangular matrix at `tri`
      auto times = [&](const float (*y)[4], const bf16* tri, float (&d)[4][4]) {
        float r[4][4] = {};
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          uint32_t am[3][4];
          a_parts(y[2 * kk], y[2 * kk + 1], am);
#pragma unroll
          for (int n2 = kk; n2 < 2; ++n2) {  // tokens 16 n2 .. + 15 from 16 kk .. + 15
            uint32_t bm[3][4];
#pragma unroll
            for (int e = 0; e < 3; ++e)
              ldsm4(bm[e], smem_at(tri + (e * CL + n2 * 16 + (lane & 7) + (lane >> 4) * 8) * CL_LD + kk * 16 + ((lane >> 3) & 1) * 8));
#pragma unroll
            for (int i = 0; i < 2; ++i) add_mma16816(d[n2 * 2 + i], am[0], bm[0][2 * i], bm[0][2 * i + 1]);
#pragma unroll
            for (int order = 3; order > 0; --order)          // the smaller products first
#pragma unroll
              for (int e = 2; e >= 0; --e)
                if (order - e >= 0 && order - e <= 2) {
#pragma unroll
                  for (int i = 0; i < 2; ++i) mma16816(r[n2 * 2 + i], am[e], bm[order - e][2 * i], bm[order - e][2 * i + 1]);
                }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) d[i][e] += r[i][e];
      };
      times(x, p.tm, u);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {        // the diagonal
          u[i][e] = fmaf(p.fac[3 * CL + 8 * i + q2 + (e & 1)], x[i][e], u[i][e]);
          odd[e >> 1] = odd[e >> 1] || !(fabsf(u[i][e]) < 1e37f);
        }
      float o[4][4] = {};
      times(u, p.tm + 3 * CL * CL_LD, o);
      const unsigned any = __ballot_sync(0xffffffffu, odd[0] || odd[1]);
      if (any == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) x[4 + i][e] = fmaf(p.fac[CL + 8 * i + q2 + (e & 1)], x[4 + i][e], o[i][e]);
      } else {
#pragma unroll
        for (int r = 0; r < 2; ++r) odd[r] = (__ballot_sync(0xffffffffu, odd[r]) >> (lane & ~3) & 15u) != 0;
        float(*ys)[CL + 1] = sm.slow[warp][0];
        float(*us)[CL + 1] = sm.slow[warp][1];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) ys[g + 8 * (e >> 1)][8 * i + q2 + (e & 1)] = x[i][e];
        __syncwarp();
        for (int pass = 0; pass < 2; ++pass) {       // U from Y, then the rest of O (in Y's place) from U
          const bf16* tri = p.tm + pass * 3 * CL * CL_LD;
          for (int at = lane; at < 16 * CL; at += 32) {
            const int col = at & 15, t = at / 16;
            float sum = 0.f;
            for (int s = 0; s <= t; ++s) {
              const float m = !pass && s == t ? p.fac[3 * CL + t]
                                              : (__bfloat162float(tri[(2 * CL + t) * CL_LD + s]) + __bfloat162float(tri[(CL + t) * CL_LD + s])) + __bfloat162float(tri[t * CL_LD + s]);
              sum += m * (pass ? us[col][s] : ys[col][s]);
            }
            if (pass) ys[col][t] = sum; else us[col][t] = sum;
          }
          __syncwarp();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int t = 8 * i + q2 + (e & 1), col = g + 8 * (e >> 1);
            if (odd[e >> 1]) u[i][e] = us[col][t];
            x[4 + i][e] = fmaf(p.fac[CL + t], x[4 + i][e], odd[e >> 1] ? ys[col][t] : o[i][e]);
          }
        __syncwarp();
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * i + q2 + (e & 1), col = jc + 8 * (e >> 1);
        if (t < nt && col < V) out[(tok0 + c * CL + t) * (long)(H * V) + (long)h * V + col] = x[4 + i][e];
        u[i][e] = t < nt ? u[i][e] * p.fac[2 * CL + t] : 0.f;
      }
    // ---- Sᵀ <- G_L Sᵀ + Uᵀ K
    const float gl = p.fac[4 * CL];
    uint32_t am[2][3][4];
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) a_parts(u[2 * kk], u[2 * kk + 1], am[kk]);
#pragma unroll
    for (int d2 = 0; d2 < DP / 16; ++d2) {
      uint32_t bm[2][4];
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) ldsm4_trans(bm[kk], smem_at(p.k + (kk * 16 + (lane & 15)) * LD + d2 * 16 + (lane >> 4) * 8));
      // the smaller parts and the earlier tokens, the state, then the later tokens
      float y[2][4], z[2][2][4];
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll
        for (int i = 0; i < 2; ++i) mma16816_new(z[kk][i], am[kk][0], bm[kk][2 * i], bm[kk][2 * i + 1]);
#pragma unroll
      for (int i = 0; i < 2; ++i) mma16816_new(y[i], am[0][2], bm[0][2 * i], bm[0][2 * i + 1]);
#pragma unroll
      for (int i = 0; i < 2; ++i) mma16816(y[i], am[1][2], bm[1][2 * i], bm[1][2 * i + 1]);
#pragma unroll
      for (int kk = 1; kk >= 0; --kk)
#pragma unroll
        for (int i = 0; i < 2; ++i) mma16816(y[i], am[kk][1], bm[kk][2 * i], bm[kk][2 * i + 1]);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) st[2 * d2 + i][e] = fmaf(gl, st[2 * d2 + i][e], y[i][e] + z[0][i][e]) + z[1][i][e];
    }
  }
#pragma unroll
  for (int i = 0; i < DP / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * i + q2 + (e & 1), col = jc + 8 * (e >> 1);
      if (d < D && col < V) Sg[(long)d * V + col] = st[i][e];
    }
}

// y[tok, h, :] = o / rms(o over V) * w * act(gate[tok, h, :]);  act 0: silu, 1: sigmoid.  One warp per (token, head).
template <typename T>
__global__ void gated_rmsnorm_kernel(const float* __restrict__ o, const T* __restrict__ gate, long ldg, const T* __restrict__ w,
                                     float eps, int act, T* __restrict__ y, long ldy, long rows, int H, int V) {
  const long wid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= rows * H) return;
  const long tok = wid / H; const int h = (int)(wid - tok * H);
  const float* orow = o + (tok * H + h) * (long)V;
  float ss = 0.f;
  for (int i = lane; i < V; i += 32) ss += orow[i] * orow[i];
  ss = warp_sum(ss);
  const float rr = 1.f / sqrtf(ss / (float)V + eps);
  for (int i = lane; i < V; i += 32) {
    const float g = ldf(gate + tok * ldg + h * V + i);
    const float ga = act == 0 ? g * sigmoidf_(g) : sigmoidf_(g);
    stf(y + tok * ldy + h * V + i, orow[i] * rr * ldf(w + i) * ga);
  }
}

// The same with 16-byte loads of o (8 bytes of gate, weight and y in bf16), the row kept in registers: V % 4 == 0, V <= 4 LANES R, rows on their
// vectors.  [2560, 16, 128]: 21.6 -> 12.5 us.  Half of the instructions of a row of 128 are sums, root and addresses, so 16 lanes take it (8 up to 64):
// [3027, 16, 128] 16.3 -> 15.3 us.
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) { const float4 x = *reinterpret_cast<const float4*>(p); v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; }
__device__ __forceinline__ void ld4(const bf16* p, float (&v)[4]) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(x.x << 16); v[1] = __uint_as_float(x.x & 0xffff0000u); v[2] = __uint_as_float(x.y << 16); v[3] = __uint_as_float(x.y & 0xffff0000u);
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void st4(bf16* p, const float (&v)[4]) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
template <typename T, int LANES, int R>
__global__ void __launch_bounds__(256)
gated_rmsnorm_vec_kernel(const float* __restrict__ o, const T* __restrict__ gate, long ldg, const T* __restrict__ w, float eps, int act, T* __restrict__ y,
                         long ldy, long rows, int H, int V) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x, wid = idx / LANES;
  const int lane = threadIdx.x % LANES;
  const long tok = wid <= 0xffffffffL ? (unsigned)wid / (unsigned)H : wid / H;
  const int h = (int)(wid - tok * H);
  lb::chain_wait(o, gate, w);
  lb::chain_next();
  const bool here = wid < rows * H;          // (the lanes of the others take part in the sums)
  const float* orow = o + wid * V;
  float x[R][4], g[R][4], ss = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = (r * LANES + lane) * 4;
    if (here && i < V) {
      ld4(orow + i, x[r]);
      ld4(gate + tok * ldg + h * V + i, g[r]);
#pragma unroll
      for (int e = 0; e < 4; ++e) ss += x[r][e] * x[r][e];
    }
  }
#pragma unroll
  for (int m = LANES / 2; m > 0; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
  const float rr = 1.f / sqrtf(ss / (float)V + eps);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = (r * LANES + lane) * 4;
    if (here && i < V) {
      float wv[4];
      ld4(w + i, wv);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float ga = act == 0 ? g[r][e] * sigmoidf_(g[r][e]) : sigmoidf_(g[r][e]);
        x[r][e] = x[r][e] * rr * wv[e] * ga;
      }
      st4(y + tok * ldy + h * V + i, x[r]);
    }
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Latent cache: ring[slot][p % ring_len] holds the latent of position p; ring_len >= window.  `gather` lays out, for every
// sequence, the still-visible cached latents followed by the step's new ones (ext rows); `write` stores the new ones.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void latent_gather_kernel(const T* __restrict__ ring, const T* __restrict__ cnew, const int* __restrict__ ext_seq,
                                     const int* __restrict__ ext_off, const int* __restrict__ seq_off, const int* __restrict__ slots,
                                     const int* __restrict__ past, T* __restrict__ ext, long rows, int C, int ring_len) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * C) return;
  const long e = idx / C; const int c = (int)(idx - e * C);
  const int b = ext_seq[e];
  const int ie = (int)(e - ext_off[b]);
  const int n = seq_off[b + 1] - seq_off[b];
  const int npast = ext_off[b + 1] - ext_off[b] - n;
  if (ie < npast) {
    const int pos = past[b] - npast + ie;
    ext[idx] = ring[((long)slots[b] * ring_len + pos % ring_len) * C + c];
  } else {
    ext[idx] = cnew[((long)seq_off[b] + ie - npast) * C + c];
  }
}

template <typename T>
__global__ void latent_write_kernel(T* __restrict__ ring, const T* __restrict__ cnew, const int* __restrict__ tok_seq,
                                    const int* __restrict__ seq_off, const int* __restrict__ slots, const int* __restrict__ past,
                                    long tokens, int C, int ring_len) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= tokens * C) return;
  const long tok = idx / C; const int c = (int)(idx - tok * C);
  const int b = tok_seq[tok];
  const int t = (int)(tok - seq_off[b]), n = seq_off[b + 1] - seq_off[b];
  if (t < n - ring_len) return;                 // an older token of this step would be overwritten anyway
  const int pos = past[b] + t;
  ring[((long)slots[b] * ring_len + pos % ring_len) * C + c] = cnew[idx];
}

// ------------------------------------------------------------------------------------------------------------------
// Sliding-window attention on expanded keys / values.  q: [tokens, H*D]; kv: [ext rows, H*D + H*V] (keys, then values);
// query t of sequence b sits at ext row ext_off[b] + npast + t and sees the `window` ext rows ending at its own, never
// crossing the start of its sequence's ext range.  One warp per (token, head): lanes take keys for the scores and value
// channels for the output; softmax in fp32, streamed 32 keys at a time.  The head's output is multiplied by
// sigmoid(gate[tok, h]) when a gate is given.
// ------------------------------------------------------------------------------------------------------------------
constexpr int ATT_MAXV = 8;    // value channels per lane: V <= 256

template <typename T>
__global__ void window_attention_kernel(const T* __restrict__ q, long ldq, const T* __restrict__ kv, long ldkv, const T* __restrict__ gate,
                                        long ldg, const int* __restrict__ tok_seq, const int* __restrict__ seq_off,
                                        const int* __restrict__ ext_off, T* __restrict__ y, long ldy, long tokens, int H, int D,
                                        int V, int window, float scale) {
  extern __shared__ float sm[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + wib;
  if (wid >= tokens * H) return;                 // no block-level sync below
  const long tok = wid / H; const int h = (int)(wid - tok * H);
  const int b = tok_seq[tok];
  const int n = seq_off[b + 1] - seq_off[b];
  const int npast = ext_off[b + 1] - ext_off[b] - n;
  const long eq = (long)ext_off[b] + npast + (tok - seq_off[b]);
  long e0 = eq - window + 1;
  if (e0 < ext_off[b]) e0 = ext_off[b];
  float* qs = sm + wib * D;
  for (int i = lane; i < D; i += 32) qs[i] = ldf(q + tok * ldq + h * D + i) * scale;
  __syncwarp();
  float m = -INFINITY, l = 0.f, acc[ATT_MAXV];
#pragma unroll
  for (int i = 0; i < ATT_MAXV; ++i) acc[i] = 0.f;
  for (long e = e0; e <= eq; e += 32) {
    const long mine = e + lane;
    float sc = -INFINITY;
    if (mine <= eq) {
      const T* kr = kv + mine * ldkv + h * D;
      float d = 0.f;
      for (int i = 0; i < D; ++i) d += qs[i] * ldf(kr + i);
      sc = d;
    }
    const float mn = fmaxf(m, warp_max(sc));
    const float corr = expf(m - mn);             // m = -inf on the first block: exp(-inf) = 0
    const float p = mine <= eq ? expf(sc - mn) : 0.f;
    l = l * corr + warp_sum(p);
#pragma unroll
    for (int i = 0; i < ATT_MAXV; ++i) acc[i] *= corr;
    const int cnt = (int)min((long)32, eq - e + 1);
    for (int k = 0; k < cnt; ++k) {
      const float pk = __shfl_sync(0xffffffffu, p, k);
      const T* vr = kv + (e + k) * ldkv + (long)H * D + h * V;
#pragma unroll
      for (int i = 0; i < ATT_MAXV; ++i) { const int c = lane + 32 * i; if (c < V) acc[i] += pk * ldf(vr + c); }
    }
    m = mn;
  }
  const float g = gate ? sigmoidf_(ldf(gate + tok * ldg + h)) : 1.f;
  const float inv = g / l;
#pragma unroll
  for (int i = 0; i < ATT_MAXV; ++i) { const int c = lane + 32 * i; if (c < V) stf(y + tok * ldy + h * V + c, acc[i] * inv); }
}

// ------------------------------------------------------------------------------------------------------------------
// The same attention on the tensor cores (bf16 operands, fp32 accumulation and softmax): a block of 4 warps owns 64
// consecutive queries of one (sequence, head) — 16 per warp, held as A fragments — and walks the key rows its queries can
// see in tiles of 64 staged through shared memory: S = Q Kᵀ with mma.m16n8k16, online softmax on the accumulator
// fragments, P re-packed as A fragments, O += P V with the V fragments fetched by ldmatrix.trans.  Query tiles are
// listed by the host (qt_seq / qt_start), so ragged batches cost no empty blocks.
// ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int D, int V>
__global__ void __launch_bounds__(128)
window_attention_mma_kernel(const __nv_bfloat16* __restrict__ q, long ldq, const __nv_bfloat16* __restrict__ kv, long ldkv,
                            const __nv_bfloat16* __restrict__ gate, long ldg, const int* __restrict__ qt_seq,
                            const int* __restrict__ qt_start, const int* __restrict__ seq_off, const int* __restrict__ ext_off,
                            __nv_bfloat16* __restrict__ y, long ldy, int H, int window, float scale) {
  constexpr int KT = 64, KS = D + 8, VS = V + 8;
  __shared__ __align__(16) __nv_bfloat16 Ks[KT * KS];
  __shared__ __align__(16) __nv_bfloat16 Vs[KT * VS];
  const int h = blockIdx.y, b = qt_seq[blockIdx.x], t0 = qt_start[blockIdx.x];
  const int n = seq_off[b + 1] - seq_off[b];
  const int elo = ext_off[b], ehi = ext_off[b + 1], npast = ehi - elo - n;
  const long tokbase = seq_off[b];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int r0 = t0 + warp * 16 + gid, r1 = r0 + 8;                    // this lane's two query rows
  const int e0 = elo + npast + r0, e1 = e0 + 8;                          // their key rows
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) {
    const int col = h * D + kk * 16 + tig * 2;
    qf[kk][0] = r0 < n ? *reinterpret_cast<const uint32_t*>(q + (tokbase + r0) * ldq + col) : 0u;
    qf[kk][1] = r1 < n ? *reinterpret_cast<const uint32_t*>(q + (tokbase + r1) * ldq + col) : 0u;
    qf[kk][2] = r0 < n ? *reinterpret_cast<const uint32_t*>(q + (tokbase + r0) * ldq + col + 8) : 0u;
    qf[kk][3] = r1 < n ? *reinterpret_cast<const uint32_t*>(q + (tokbase + r1) * ldq + col + 8) : 0u;
  }
  float o[V / 8][4];
#pragma unroll
  for (int j = 0; j < V / 8; ++j) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f; }
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;              // l: this lane's share of the row sums
  const int eq_first = elo + npast + t0, eq_last = elo + npast + min(t0 + 63, n - 1);
  const int ew0 = eq_first + warp * 16;                                   // first key row of this warp's queries
  int kbeg = eq_first - window + 1;
  if (kbeg < elo) kbeg = elo;
  for (int k0 = kbeg; k0 <= eq_last; k0 += KT) {
    __syncthreads();
    for (int c = threadIdx.x; c < KT * (D / 8); c += 128) {
      const int row = c / (D / 8), ch = c - row * (D / 8);
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (k0 + row < ehi) val = *reinterpret_cast<const uint4*>(kv + (long)(k0 + row) * ldkv + h * D + ch * 8);
      *reinterpret_cast<uint4*>(&Ks[row * KS + ch * 8]) = val;
    }
    for (int c = threadIdx.x; c < KT * (V / 8); c += 128) {
      const int row = c / (V / 8), ch = c - row * (V / 8);
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (k0 + row < ehi) val = *reinterpret_cast<const uint4*>(kv + (long)(k0 + row) * ldkv + (long)H * D + h * V + ch * 8);
      *reinterpret_cast<uint4*>(&Vs[row * VS + ch * 8]) = val;
    }
    __syncthreads();
    if (k0 > ew0 + 15 || k0 + KT - 1 <= ew0 - window) continue;          // nothing in this tile for the warp's 16 queries
    float sacc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) { sacc[j][0] = sacc[j][1] = sacc[j][2] = sacc[j][3] = 0.f; }
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const __nv_bfloat16* kr = &Ks[(j * 8 + gid) * KS + kk * 16 + tig * 2];
        mma_bf16(sacc[j], qf[kk], *reinterpret_cast<const uint32_t*>(kr), *reinterpret_cast<const uint32_t*>(kr + 8));
      }
    }
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int key = k0 + j * 8 + tig * 2 + (c & 1), eq = c < 2 ? e0 : e1;
        const bool valid = key <= eq && key > eq - window;
        const float sv = valid ? sacc[j][c] * scale : -INFINITY;
        sacc[j][c] = sv;
        if (c < 2) mx0 = fmaxf(mx0, sv); else mx1 = fmaxf(mx1, sv);
      }
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1)); mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1)); mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
    const float c0 = mn0 == -INFINITY ? 1.f : __expf(m0 - mn0), c1 = mn1 == -INFINITY ? 1.f : __expf(m1 - mn1);
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float sv = sacc[j][c];
        const float pv = sv == -INFINITY ? 0.f : __expf(sv - (c < 2 ? mn0 : mn1));
        sacc[j][c] = pv;
        if (c < 2) s0 += pv; else s1 += pv;
      }
    }
    l0 = l0 * c0 + s0; l1 = l1 * c1 + s1; m0 = mn0; m1 = mn1;
#pragma unroll
    for (int j = 0; j < V / 8; ++j) { o[j][0] *= c0; o[j][1] *= c0; o[j][2] *= c1; o[j][3] *= c1; }
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      uint32_t a[4];
      a[0] = pack_bf16(sacc[2 * k2][0], sacc[2 * k2][1]); a[1] = pack_bf16(sacc[2 * k2][2], sacc[2 * k2][3]);
      a[2] = pack_bf16(sacc[2 * k2 + 1][0], sacc[2 * k2 + 1][1]); a[3] = pack_bf16(sacc[2 * k2 + 1][2], sacc[2 * k2 + 1][3]);
      const uint32_t vrow = (uint32_t)__cvta_generic_to_shared(&Vs[(k2 * 16 + (lane & 15)) * VS]);
#pragma unroll
      for (int j = 0; j < V / 8; ++j) {
        uint32_t b0, b1;
        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(b0), "=r"(b1) : "r"(vrow + j * 16));
        mma_bf16(o[j], a, b0, b1);
      }
    }
  }
  l0 += __shfl_xor_sync(0xffffffffu, l0, 1); l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
  l1 += __shfl_xor_sync(0xffffffffu, l1, 1); l1 += __shfl_xor_sync(0xffffffffu, l1, 2);
  const float g0 = (gate && r0 < n) ? sigmoidf_(__bfloat162float(gate[(tokbase + r0) * ldg + h])) : 1.f;
  const float g1 = (gate && r1 < n) ? sigmoidf_(__bfloat162float(gate[(tokbase + r1) * ldg + h])) : 1.f;
  const float i0 = g0 / l0, i1 = g1 / l1;
#pragma unroll
  for (int j = 0; j < V / 8; ++j) {
    const int col = h * V + j * 8 + tig * 2;
    if (r0 < n) *reinterpret_cast<uint32_t*>(y + (tokbase + r0) * ldy + col) = pack_bf16(o[j][0] * i0, o[j][1] * i0);
    if (r1 < n) *reinterpret_cast<uint32_t*>(y + (tokbase + r1) * ldy + col) = pack_bf16(o[j][2] * i1, o[j][3] * i1);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Single-token steps in the absorbed form: the query already carries the key up-projection (qa [B, H, C], fp32), so the
// scores and the weighted sum run on the cached latents themselves; the new token's latent (cnew [B, C]) is position
// past[b], the others come from the ring.  out: [B, H, C] fp32 = softmax-weighted latent per head (the value
// up-projection follows as a batched matrix product).  One warp per (sequence, head).
// ------------------------------------------------------------------------------------------------------------------
constexpr int ABS_MAXC = 32;   // latent channels per lane: C <= 1024

template <typename T>
__global__ void latent_decode_kernel(const float* __restrict__ qa, const T* __restrict__ ring, const T* __restrict__ cnew,
                                     const int* __restrict__ slots, const int* __restrict__ past, float* __restrict__ out, int B, int H,
                                     int C, int ring_len, int window, float scale) {
  extern __shared__ float sm[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + wib;
  if (wid >= (long)B * H) return;
  const int b = (int)(wid / H), h = (int)(wid - (long)b * H);
  const int p = past[b];
  int p0 = p - window + 1; if (p0 < 0) p0 = 0;
  float* qs = sm + wib * C;
  for (int i = lane; i < C; i += 32) qs[i] = qa[((long)b * H + h) * C + i] * scale;
  __syncwarp();
  const T* rb = ring + (long)slots[b] * ring_len * C;
  float m = -INFINITY, l = 0.f, acc[ABS_MAXC];
#pragma unroll
  for (int i = 0; i < ABS_MAXC; ++i) acc[i] = 0.f;
  for (int e = p0; e <= p; e += 32) {
    const int mine = e + lane;
    float sc = -INFINITY;
    if (mine <= p) {
      const T* cr = mine == p ? cnew + (long)b * C : rb + (long)(mine % ring_len) * C;
      float d = 0.f;
      for (int i = 0; i < C; ++i) d += qs[i] * ldf(cr + i);
      sc = d;
    }
    const float mn = fmaxf(m, warp_max(sc));
    const float corr = expf(m - mn);
    const float pr = mine <= p ? expf(sc - mn) : 0.f;
    l = l * corr + warp_sum(pr);
#pragma unroll
    for (int i = 0; i < ABS_MAXC; ++i) acc[i] *= corr;
    const int cnt = min(32, p - e + 1);
    for (int k = 0; k < cnt; ++k) {
      const float pk = __shfl_sync(0xffffffffu, pr, k);
      const T* cr = (e + k) == p ? cnew + (long)b * C : rb + (long)((e + k) % ring_len) * C;
#pragma unroll
      for (int i = 0; i < ABS_MAXC; ++i) { const int c = lane + 32 * i; if (c < C) acc[i] += pk * ldf(cr + c); }
    }
    m = mn;
  }
  const float inv = 1.f / l;
#pragma unroll
  for (int i = 0; i < ABS_MAXC; ++i) { const int c = lane + 32 * i; if (c < C) out[((long)b * H + h) * C + c] = acc[i] * inv; }
}

// Split form of the same step for long windows: all heads of a sequence share its latents, so a block stages KC = 32
// of them once (plus the queries of up to 16 heads) in shared memory, computes the scores of every head against them,
// a partial softmax (max, sum) and the partial weighted sum; a second kernel merges the partials of a (sequence, head).
constexpr int KC = 32, HG = 16;

template <typename T>
__global__ void __launch_bounds__(256)
latent_decode_split_kernel(const float* __restrict__ qa, const T* __restrict__ ring, const T* __restrict__ cnew,
                           const int* __restrict__ slots, const int* __restrict__ past, float* __restrict__ part_o,
                           float* __restrict__ part_ml, int H, int C, int ring_len, int window, int nch, float scale) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int b = blockIdx.x, ch = blockIdx.y, h0 = blockIdx.z * HG;
  const int hg = min(HG, H - h0);
  const int p = past[b];
  int p0 = p - window + 1; if (p0 < 0) p0 = 0;
  const int e0 = p0 + ch * KC;
  if (e0 > p) return;                                           // the whole block leaves: no barrier is skipped
  const int cnt = min(KC, p - e0 + 1);
  const int LS = C + (sizeof(T) == 2 ? 2 : 1);                  // tile row stride: an odd number of 32-bit words
  float* sq = reinterpret_cast<float*>(smraw);                  // [HG][C]
  float* ss = sq + HG * C;                                      // [HG][KC]
  T* sl = reinterpret_cast<T*>(ss + HG * KC);                   // [KC][LS]
  const int tid = threadIdx.x;
  for (int e = tid; e < hg * C; e += 256) sq[e] = qa[((long)b * H + h0) * C + e] * scale;
  const T* rb = ring + (long)slots[b] * ring_len * C;
  for (int e = tid; e < cnt * C; e += 256) {
    const int kk = e / C, c = e - kk * C, pos = e0 + kk;
    sl[kk * LS + c] = pos == p ? cnew[(long)b * C + c] : rb[(long)(pos % ring_len) * C + c];
  }
  __syncthreads();
  const int lane = tid & 31, w = tid >> 5;
  for (int hh = w; hh < hg; hh += 8) {                          // one warp per head: lane = key
    float sc = -INFINITY;
    if (lane < cnt) {
      float d = 0.f;
      const float* qr = sq + hh * C; const T* lr = sl + lane * LS;
      for (int c = 0; c < C; ++c) d += qr[c] * ldf(lr + c);
      sc = d;
    }
    const float m = warp_max(sc);
    const float pr = lane < cnt ? expf(sc - m) : 0.f;
    const float l = warp_sum(pr);
    ss[hh * KC + lane] = pr;
    if (lane == 0) { float* ml = part_ml + (((long)b * H + h0 + hh) * nch + ch) * 2; ml[0] = m; ml[1] = l; }
  }
  __syncthreads();
  for (int c = tid; c < C; c += 256) {
    float acc[HG];
#pragma unroll
    for (int hh = 0; hh < HG; ++hh) acc[hh] = 0.f;
    for (int kk = 0; kk < cnt; ++kk) {
      const float lv = ldf(sl + kk * LS + c);
#pragma unroll
      for (int hh = 0; hh < HG; ++hh) acc[hh] += ss[hh * KC + kk] * lv;   // rows >= hg hold stale values that are not stored
    }
#pragma unroll
    for (int hh = 0; hh < HG; ++hh)
      if (hh < hg) part_o[(((long)b * H + h0 + hh) * nch + ch) * C + c] = acc[hh];
  }
}

__global__ void latent_decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                           const int* __restrict__ past, float* __restrict__ out, int H, int C, int window, int nch) {
  const int b = blockIdx.x / H;
  const int p = past[b];
  int p0 = p - window + 1; if (p0 < 0) p0 = 0;
  const int used = (p - p0) / KC + 1;
  const float* ml = part_ml + (long)blockIdx.x * nch * 2;
  float M = -INFINITY;
  for (int c = 0; c < used; ++c) M = fmaxf(M, ml[2 * c]);
  float L = 0.f;
  for (int c = 0; c < used; ++c) L += expf(ml[2 * c] - M) * ml[2 * c + 1];
  for (int i = threadIdx.x; i < C; i += blockDim.x) {
    float acc = 0.f;
    for (int c = 0; c < used; ++c) acc += expf(ml[2 * c] - M) * part_o[((long)blockIdx.x * nch + c) * C + i];
    out[(long)blockIdx.x * C + i] = acc / L;
  }
}

// y[b, h*V + v] = x[b, h, v] * sigmoid(gate[b, h]) (fp32 in, T out)
template <typename T>
__global__ void head_gate_kernel(const float* __restrict__ x, const T* __restrict__ gate, long ldg, T* __restrict__ y, long ldy,
                                 long rows, int H, int V) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * H * V) return;
  const long row = idx / ((long)H * V); const int hv = (int)(idx - row * (long)H * V); const int h = hv / V;
  const float g = gate ? sigmoidf_(ldf(gate + row * ldg + h)) : 1.f;
  stf(y + row * ldy + hv, x[idx] * g);
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }
inline int ok() { return (int)cudaGetLastError(); }

}  // namespace

#define DISPATCH(dtype, ...)                         \
  if ((dtype) == 0) { typedef float T; __VA_ARGS__; } \
  else { typedef bf16 T; __VA_ARGS__; }

extern "C" {

// x: rows of `xdtype` (0 fp32, 1 bf16); w and y: `dtype`; ids optional row gather
int lbs_rmsnorm(const void* x, long ldx, int xdtype, const int64_t* ids, const void* w, float offset, float eps, void* y, long ldy,
                int ydtype, int wdtype, long rows, int n, cudaStream_t s) {
  if (rows == 0) return 0;
  const int th = n >= 1024 ? 256 : (n >= 256 ? 128 : 64);
#define RN(TI, TW, TO) rmsnorm_kernel<TI, TW, TO><<<(unsigned)rows, th, 0, s>>>((const TI*)x, ldx, ids, (const TW*)w, offset, eps, (TO*)y, ldy, n)
  const int key = xdtype * 4 + wdtype * 2 + ydtype;
  switch (key) {
    case 0: RN(float, float, float); break;
    case 1: RN(float, float, bf16); break;
    case 2: RN(float, bf16, float); break;
    case 3: RN(float, bf16, bf16); break;
    case 4: RN(bf16, float, float); break;
    case 5: RN(bf16, float, bf16); break;
    case 6: RN(bf16, bf16, float); break;
    default: RN(bf16, bf16, bf16); break;
  }
#undef RN
  return ok();
}

int lbs_slice_act(const void* in, long ldi, int idtype, void* out, long ldo, int odtype, long rows, int n, int act, cudaStream_t s) {
  if (rows * n == 0) return 0;
  if (idtype == 1 && odtype == 1 && n % 8 == 0 && ldi % 8 == 0 && ldo % 8 == 0 && ((uintptr_t)in) % 16 == 0 && ((uintptr_t)out) % 16 == 0) {
    slice_act_vec8_kernel<<<cdiv(rows * (n / 8), 256), 256, 0, s>>>((const bf16*)in, ldi, (bf16*)out, ldo, rows, n / 8, act);
    return ok();
  }
  const int g = cdiv(rows * n, 256);
  if (idtype == 0 && odtype == 0) slice_act_kernel<float, float><<<g, 256, 0, s>>>((const float*)in, ldi, (float*)out, ldo, rows, n, act);
  else if (idtype == 0) slice_act_kernel<float, bf16><<<g, 256, 0, s>>>((const float*)in, ldi, (bf16*)out, ldo, rows, n, act);
  else if (odtype == 0) slice_act_kernel<bf16, float><<<g, 256, 0, s>>>((const bf16*)in, ldi, (float*)out, ldo, rows, n, act);
  else slice_act_kernel<bf16, bf16><<<g, 256, 0, s>>>((const bf16*)in, ldi, (bf16*)out, ldo, rows, n, act);
  return ok();
}

int lbs_short_conv(const void* in, long ldi, const void* w, void* tail, const int* tok_seq, const int* seq_off, const int* slots,
                   const int* past, void* out, long ldo, long tokens, int B, int C, int taps, int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  const bool vec = dtype == 1 && C % 8 == 0 && ldi % 8 == 0 && ldo % 8 == 0 && taps >= 2 && taps <= 4 && ((uintptr_t)in) % 16 == 0 &&
                   ((uintptr_t)out) % 16 == 0 && ((uintptr_t)tail) % 16 == 0 && ((uintptr_t)w) % 16 == 0;
  if (vec) {
    // strips once they fill the SMs: fewer tokens have more threads with one token each
    const bool strips = tokens * (C / 8) >= 148L * 8 * 128 * CONV_STRIP / 4;
    const int g = strips ? cdiv((tokens + CONV_STRIP - 1) / CONV_STRIP * (C / 8), 128) : cdiv(tokens * (C / 8), 256);
#define SC(TP)                                                                                                                   \
  if (strips) lb_host::launch_chained(short_conv_strip_kernel<TP>, dim3(g), dim3(128), 0, s, 0, (const bf16*)in, ldi, (const bf16*)w, (const bf16*)tail, tok_seq, seq_off, \
                                      slots, past, (bf16*)out, ldo, tokens, C);                                                  \
  else short_conv_vec8_kernel<TP><<<g, 256, 0, s>>>((const bf16*)in, ldi, (const bf16*)w, (const bf16*)tail, tok_seq, seq_off, slots, past, \
                                                    (bf16*)out, ldo, tokens, C)
    if (taps == 2) { SC(2); } else if (taps == 3) { SC(3); } else { SC(4); }
#undef SC
    lb_host::launch_chained(conv_tail_kernel<bf16>, dim3(cdiv((long)B * C, 256)), dim3(256), 0, s, 0, (const bf16*)in, ldi, (bf16*)tail, seq_off, slots, past, B, C, taps);
    return ok();
  }
  DISPATCH(dtype, {
    short_conv_kernel<T><<<cdiv(tokens * C, 256), 256, 0, s>>>((const T*)in, ldi, (const T*)w, (const T*)tail, tok_seq, seq_off, slots,
                                                                past, (T*)out, ldo, tokens, C, taps);
    if (taps > 1)
      lb_host::launch_chained(conv_tail_kernel<T>, dim3(cdiv((long)B * C, 256)), dim3(256), 0, s, 0, (const T*)in, ldi, (T*)tail, seq_off, slots, past, B, C, taps);
  });
  return ok();
}

// can bf16 sequences of these sizes be scanned in chunks?  (every row of q, k and v in whole aligned vectors)
static bool delta_chunks_apply(long ldq, int koff, int voff, int H, int D, int V, int chan, int dtype) {
  return dtype != 0 && !chan && D <= 128 && D % 4 == 0 && V % 8 == 0 && ldq % 8 == 0 && koff % 8 == 0 && voff % 8 == 0 && H <= 65535;
}
// fp32 scratch of lbs_delta_scan, in floats; longest: tokens of the longest sequence
long lbs_delta_work(long tokens, int B, long ldq, int koff, int voff, int H, int KH, int D, int V, int chan, int dtype, long longest) {
  const long prep = (tokens * (2L * KH * D + KH + H + (chan ? (long)H * D : (long)H)) + 3) / 4 * 4;
  return prep + (longest >= CL_MIN && delta_chunks_apply(ldq, koff, voff, H, D, V, chan, dtype) ? (tokens / CL + B) * H * CL_SCRATCH : 0);
}

// work: lbs_delta_work(...) floats; shortest, longest: tokens of the shortest and the longest sequence
int lbs_delta_scan(const void* qkv, long ldq, int koff, int voff, const void* a, long lda, const void* bl, long ldb, const void* A_log,
                   const void* dt_bias, float* S, const int* seq_off, const int* slots, const int* past, float* out, float* work,
                   long tokens, int B, int H, int KH, int D, int V, int chan, int dtype, long shortest, long longest, cudaStream_t s) {
  if (B == 0 || tokens == 0) return 0;
  if (D > 256 || H % KH != 0) return -1;
  // Long sequences in chunks, the others in pairs or token by token; which one depends on a sequence's own length only.
  int shorter_than = 0x7fffffff;
  if (longest >= CL_MIN && delta_chunks_apply(ldq, koff, voff, H, D, V, chan, dtype) && (reinterpret_cast<uintptr_t>(qkv) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(work) & 15) == 0 && (D % 8 == 0 || KH == 1)) {
    float* scratch = work + (tokens * (2L * KH * D + KH + 2L * H) + 3) / 4 * 4;
    const dim3 pg((unsigned)(tokens / CL + B), (unsigned)KH), sg((unsigned)(B * H), (unsigned)((V + CL_COLS - 1) / CL_COLS));
#define DCH(DP)                                                                                                                          \
  {                                                                                                                                      \
    const int smem = (int)sizeof(DeltaChunkSmem<DP>);                                                                                    \
    const cudaError_t e = cudaFuncSetAttribute(delta_chunk_scan_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);          \
    if (e != cudaSuccess) return (int)e;                                                                                                 \
    lb_host::launch_chained(delta_chunk_prep_kernel<DP>, pg, dim3(128), 0, s, 0, (const bf16*)qkv, ldq, koff, (const bf16*)a, lda, (const bf16*)bl, ldb, \
                            (const bf16*)A_log, (const bf16*)dt_bias, seq_off, scratch, B, H, KH, D);                                    \
    delta_chunk_scan_kernel<DP><<<sg, 32 * CL_WARPS, smem, s>>>((const bf16*)qkv, ldq, koff, voff, scratch, S, seq_off, slots, past, out, H, KH, D, V); \
  }
    if (D <= 64) DCH(64) else DCH(128)
#undef DCH
    if (shortest >= CL_MIN) return ok();
    shorter_than = CL_MIN;
  }
  float* qn = work;
  float* kn = qn + tokens * KH * D;
  float* kq = kn + tokens * KH * D;
  float* beta = kq + tokens * KH;
  float* g = beta + tokens * H;
  DISPATCH(dtype, delta_prep_kernel<T><<<cdiv(tokens * KH * 32, 256), 256, 0, s>>>((const T*)qkv, ldq, koff, (const T*)a, lda, (const T*)bl,
                                                                                  ldb, (const T*)A_log, (const T*)dt_bias, qn, kn, kq, g,
                                                                                  beta, tokens, H, KH, D, chan));
  // one decay per head: two tokens at a time where rows and columns come in whole 16-byte vectors (the general kernel takes the rest:
  // decays per channel, more than 128 rows, odd sizes)
  const int vec = dtype == 0 ? 4 : 8;
  if (!chan && D <= 128 && D % 4 == 0 && V % vec == 0 && ldq % vec == 0 && voff % vec == 0 && (reinterpret_cast<uintptr_t>(qkv) & 15) == 0 &&
      (reinterpret_cast<uintptr_t>(work) & 15) == 0 && (tokens * KH * D) % 4 == 0) {
    const int cpt = (long)B * H * ((V + 63) / 64) >= 100 ? 2 : 1;    // two columns per lane once the blocks fill two thirds of the SMs
    const dim3 pgrid((unsigned)(B * H), (unsigned)((V + 32 * cpt - 1) / (32 * cpt)));
#define DSP(TT, D4, CPT)                                                                                                                \
  delta_scan_pair_kernel<TT, D4, CPT><<<pgrid, PAIR_THREADS, pair_smem_floats(16 * D4, 32 * CPT) * sizeof(float), s>>>(                 \
      (const TT*)qkv, ldq, voff, qn, kn, kq, g, beta, S, seq_off, slots, past, out, H, KH, D, V, shorter_than)
#define DSP4(TT)                                          \
  {                                                       \
    if (D <= 64) { if (cpt == 2) DSP(TT, 4, 2); else DSP(TT, 4, 1); } \
    else { if (cpt == 2) DSP(TT, 8, 2); else DSP(TT, 8, 1); }         \
  }
    if (dtype == 0) DSP4(float) else DSP4(bf16)
#undef DSP4
#undef DSP
    return ok();
  }
  const int dpt = D <= 32 ? 8 : (D <= 128 ? 16 : 32);  // rows per lane: 4 lanes per column up to D = 64, 8 lanes up to 256
  int R = 1;
  while (R * dpt < D) R <<= 1;                   // a power of two <= 8
  int VT = R <= 4 ? 64 : 32;                     // columns per block (columns are independent: more blocks per head)
  if (V < VT) VT = V;
  int threads = ((VT * R + 31) / 32) * 32;
  const int Dp = R * (dpt + 4);
  const size_t smem = sizeof(float) * ((size_t)CT * Dp * 2 + (size_t)CT * (chan ? Dp : 4) + (size_t)CT * VT + 2 * CT);
  dim3 grid((unsigned)(B * H), (unsigned)((V + VT - 1) / VT));
#define DS(TT, P)                                                                                                              \
  {                                                                                                                            \
    if (smem > 48 * 1024) cudaFuncSetAttribute(delta_scan_kernel<TT, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    delta_scan_kernel<TT, P><<<grid, threads, smem, s>>>((const TT*)qkv, ldq, voff, qn, kn, kq, g, beta, S, seq_off, slots, past, out, \
                                                        H, KH, D, V, R, VT, chan);                                              \
  }
  if (dtype == 0) { if (dpt == 8) DS(float, 8) else if (dpt == 16) DS(float, 16) else DS(float, 32) }
  else { if (dpt == 8) DS(bf16, 8) else if (dpt == 16) DS(bf16, 16) else DS(bf16, 32) }
#undef DS
  return ok();
}

int lbs_gated_rmsnorm(const float* o, const void* gate, long ldg, const void* w, float eps, int act, void* y, long ldy, long rows,
                      int H, int V, int dtype, cudaStream_t s) {
  if (rows == 0) return 0;
  const uintptr_t vec = dtype == 0 ? 16 : 8;                    // bytes of four elements
  if (V % 4 == 0 && V <= 512 && ldg % 4 == 0 && ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(o) & 15) == 0 &&
      ((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) & (vec - 1)) == 0) {
#define GRV(LN, R) DISPATCH(dtype, lb_host::launch_chained(gated_rmsnorm_vec_kernel<T, LN, R>, dim3(cdiv(rows * H * LN, 256)), dim3(256), 0, s, 0, o, (const T*)gate, ldg, (const T*)w, eps, act, (T*)y, ldy, rows, H, V))
    if (V <= 64) { GRV(8, 2); } else if (V <= 128) { GRV(16, 2); } else if (V <= 256) { GRV(32, 2); } else { GRV(32, 4); }
#undef GRV
    return ok();
  }
  DISPATCH(dtype, gated_rmsnorm_kernel<T><<<cdiv(rows * H * 32, 256), 256, 0, s>>>(o, (const T*)gate, ldg, (const T*)w, eps, act,
                                                                                    (T*)y, ldy, rows, H, V));
  return ok();
}

int lbs_latent_gather(const void* ring, const void* cnew, const int* ext_seq, const int* ext_off, const int* seq_off, const int* slots,
                      const int* past, void* ext, long rows, int C, int ring_len, int dtype, cudaStream_t s) {
  if (rows == 0) return 0;
  DISPATCH(dtype, latent_gather_kernel<T><<<cdiv(rows * C, 256), 256, 0, s>>>((const T*)ring, (const T*)cnew, ext_seq, ext_off, seq_off,
                                                                               slots, past, (T*)ext, rows, C, ring_len));
  return ok();
}

int lbs_latent_write(void* ring, const void* cnew, const int* tok_seq, const int* seq_off, const int* slots, const int* past,
                     long tokens, int C, int ring_len, int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  DISPATCH(dtype, latent_write_kernel<T><<<cdiv(tokens * C, 256), 256, 0, s>>>((T*)ring, (const T*)cnew, tok_seq, seq_off, slots, past,
                                                                                tokens, C, ring_len));
  return ok();
}

int lbs_window_attention(const void* q, long ldq, const void* kv, long ldkv, const void* gate, long ldg, const int* tok_seq,
                         const int* seq_off, const int* ext_off, const int* qt_seq, const int* qt_start, int n_qtiles, void* y,
                         long ldy, long tokens, int H, int D, int V, int window, float scale, int dtype, cudaStream_t s) {
  if (tokens == 0) return 0;
  if (V > 32 * ATT_MAXV) return -1;
  const bool aligned = (ldkv % 8 == 0) && (ldq % 2 == 0) && (ldy % 2 == 0) && (((uintptr_t)kv) % 16 == 0) &&
                       (((uintptr_t)q) % 4 == 0) && (((uintptr_t)y) % 4 == 0);
  if (dtype == 1 && qt_seq != nullptr && n_qtiles > 0 && aligned) {
    dim3 grid((unsigned)n_qtiles, (unsigned)H);
#define WA(DD, VV)                                                                                                        \
  if (D == DD && V == VV) {                                                                                                \
    window_attention_mma_kernel<DD, VV><<<grid, 128, 0, s>>>((const bf16*)q, ldq, (const bf16*)kv, ldkv, (const bf16*)gate, ldg, \
                                                             qt_seq, qt_start, seq_off, ext_off, (bf16*)y, ldy, H, window, scale); \
    return ok();                                                                                                           \
  }
    WA(32, 32) WA(64, 64) WA(128, 128) WA(64, 128) WA(128, 64) WA(32, 64) WA(64, 32)
#undef WA
  }
  const int warps = 4;
  const size_t smem = sizeof(float) * warps * D;
  DISPATCH(dtype, window_attention_kernel<T><<<cdiv(tokens * H, warps), warps * 32, smem, s>>>(
                      (const T*)q, ldq, (const T*)kv, ldkv, (const T*)gate, ldg, tok_seq, seq_off, ext_off, (T*)y, ldy, tokens, H, D, V,
                      window, scale));
  return ok();
}

// part_o: [B, H, nch, C] fp32 and part_ml: [B, H, nch, 2] fp32 workspaces with nch = ceil(window / 32), or null: then (and for
// windows of at most 64 positions) one warp per (sequence, head) does the whole window
int lbs_latent_decode(const float* qa, const void* ring, const void* cnew, const int* slots, const int* past, float* out,
                      float* part_o, float* part_ml, int B, int H, int C, int ring_len, int window, float scale, int dtype,
                      cudaStream_t s) {
  if (B == 0) return 0;
  if (part_o != nullptr && part_ml != nullptr && window > 64) {
    const int nch = (window + KC - 1) / KC;
    const int hg = H < HG ? H : HG;
    const size_t esz = dtype == 0 ? 4 : 2;
    const size_t smem = sizeof(float) * ((size_t)HG * C + HG * KC) + esz * KC * (C + (dtype == 0 ? 1 : 2));
    (void)hg;
    if (smem <= 200 * 1024) {
      dim3 grid((unsigned)B, (unsigned)nch, (unsigned)((H + HG - 1) / HG));
      DISPATCH(dtype, {
        if (smem > 48 * 1024) cudaFuncSetAttribute(latent_decode_split_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        latent_decode_split_kernel<T><<<grid, 256, smem, s>>>(qa, (const T*)ring, (const T*)cnew, slots, past, part_o, part_ml, H, C,
                                                              ring_len, window, nch, scale);
      });
      latent_decode_merge_kernel<<<B * H, 128, 0, s>>>(part_o, part_ml, past, out, H, C, window, nch);
      return ok();
    }
  }
  if (C > 32 * ABS_MAXC) return -1;
  const int warps = 4;
  const size_t smem = sizeof(float) * warps * C;
  DISPATCH(dtype, latent_decode_kernel<T><<<cdiv((long)B * H, warps), warps * 32, smem, s>>>(qa, (const T*)ring, (const T*)cnew, slots,
                                                                                              past, out, B, H, C, ring_len, window, scale));
  return ok();
}

int lbs_head_gate(const float* x, const void* gate, long ldg, void* y, long ldy, long rows, int H, int V, int dtype, cudaStream_t s) {
  if (rows == 0) return 0;
  DISPATCH(dtype, head_gate_kernel<T><<<cdiv(rows * H * V, 256), 256, 0, s>>>(x, (const T*)gate, ldg, (T*)y, ldy, rows, H, V));
  return ok();
}

}  // extern "C"

// Activation quantizers and the non-matmul operators of a transformer block
// (crates/aot-kernels/src/quant.rs:231-283, crates/aot-kernels/src/ops.rs,
// crates/aot-kernels/src/sampler.rs:99-109) as CUDA kernels.
//
// The reference's f32 reductions are strictly sequential loops. Results here
// are bit-identical: every reduction whose order is observable (sum of
// squares, q.k dots, softmax denominator, the value mix) is evaluated in the
// reference's order with unfused round-to-nearest operations; order-free
// reductions (max, argmax, integer sums) run in parallel.
#pragma once
#include <cuda_fp16.h>

#include "blockmath.cuh"
#include "device_utils.cuh"
#include "expf_exact.cuh"
#include "groupsum.cuh"

namespace aot {

// ---- sequential-order sum of a shared-memory array --------------------------------
// (((0 + p[0]) + p[1]) + ...) exactly as a scalar loop would round it. Called by
// the whole block; the result is returned to every thread. `slot` is one float of
// shared memory.
__device__ __forceinline__ float block_seq_sum(const float* p, int n, float* slot) {
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    int i = 0;
    for (; i + 8 <= n; i += 8) {
      float a0 = p[i], a1 = p[i + 1], a2 = p[i + 2], a3 = p[i + 3], a4 = p[i + 4], a5 = p[i + 5], a6 = p[i + 6],
            a7 = p[i + 7];
      s = fadd(s, a0);
      s = fadd(s, a1);
      s = fadd(s, a2);
      s = fadd(s, a3);
      s = fadd(s, a4);
      s = fadd(s, a5);
      s = fadd(s, a6);
      s = fadd(s, a7);
    }
    for (; i < n; i++) s = fadd(s, p[i]);
    *slot = s;
  }
  __syncthreads();
  return *slot;
}

// ---- Q8_K quantization of one 256-value block by one warp ----------------------------
// quant.rs:248-283. `src` may be shared or global. The block is written either in
// the reference's BlockQ8_K layout (image == 0) or as the 304-byte image the GEMV
// kernels read (image == 1).
// Core: lane holds elements 8*lane .. 8*lane+7 of the block in v[].
struct Q8kLane {
  uint32_t w0, w1;  // the lane's eight quants
  int s;            // their sum
  float d;          // the block's scale
};
__device__ __forceinline__ Q8kLane warp_q8k_lane(const float (&v)[8]) {
  const int lane = threadIdx.x & 31;
  // signed extreme: the first element with strictly larger |v|. |v| orders like its bit
  // pattern; a NaN never compares larger in the reference and counts as zero here. Two
  // warp-wide integer reductions find the largest pattern and the first index holding it.
  uint32_t best = 0;
  float mx = 0.0f;
  int idx = 8 * lane;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    uint32_t a = __float_as_uint(v[i]) & 0x7FFFFFFFu;
    a = a > 0x7F800000u ? 0u : a;
    if (a > best) {
      best = a;
      mx = v[i];
      idx = 8 * lane + i;
    }
  }
  const uint32_t wmax = __reduce_max_sync(0xffffffffu, best);
  const uint32_t widx = __reduce_min_sync(0xffffffffu, best == wmax ? (uint32_t)idx : 256u);
  mx = __shfl_sync(0xffffffffu, mx, (int)(widx >> 3));
  const float amax = __uint_as_float(wmax);
  Q8kLane r{0u, 0u, 0, 0.0f};
  if (amax != 0.0f) {
    float iscale = fdiv(-127.0f, mx);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      int q = (int)roundf(fmul(iscale, v[i]));
      q = q > 127 ? 127 : q;
      r.s += q;
      uint32_t b = (uint32_t)(q & 0xFF);
      if (i < 4) r.w0 |= b << (8 * i); else r.w1 |= b << (8 * (i - 4));
    }
    r.d = fdiv(1.0f, iscale);
  }
  return r;
}
__device__ __forceinline__ void warp_quantize_q8k_vals(const float (&v)[8], uint8_t* dst, int image) {
  const int lane = threadIdx.x & 31;
  const Q8kLane r = warp_q8k_lane(v);
  int8_t* qs = reinterpret_cast<int8_t*>(dst + (image ? 0 : 4));
  int16_t* bs = reinterpret_cast<int16_t*>(dst + (image ? 256 : 260));
  float* dptr = reinterpret_cast<float*>(dst + (image ? 288 : 0));
  reinterpret_cast<uint32_t*>(qs)[2 * lane] = r.w0;
  reinterpret_cast<uint32_t*>(qs)[2 * lane + 1] = r.w1;
  int s2 = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);
  if ((lane & 1) == 0) bs[lane >> 1] = (int16_t)s2;
  if (lane == 0) *dptr = r.d;
}

// Activations of several rows in the orders in which the tensor-core products read them: two arrays of
// blocks, [super-block][token group of 8], XF_BLOCK bytes each for kmma.cuh and XT_BLOCK bytes each for
// ktensor.cuh.
constexpr int XF_BLOCK = 2336, XF_BSUMS = 2048, XF_D = 2304;
constexpr int XT_BLOCK = 2368, XT_BSUMS = 2048, XT_D = 2304, XT_SUMS = 2336;
// Token tok of nt groups, super-block b; either array may be absent. Lane l of the warp holds the quants
// 8l .. 8l+7; lanes 0..15 the sums of the 16-element groups.
__device__ __forceinline__ void xf_store(uint8_t* xf, uint8_t* xt, int tok, int b, int nt, int lane, uint32_t w0, uint32_t w1, int bsum, float d) {
  const int g = tok & 7, s = lane >> 1, h = lane & 1;
  const size_t at = (size_t)b * nt + (tok >> 3);
  const __half bs = __int2half_rn(bsum);
  if (xf) {
    uint8_t* const o = xf + at * XF_BLOCK;
    uint32_t* q = reinterpret_cast<uint32_t*>(o + ((s >> 2) * 32 + g * 4 + 2 * h) * 16 + (s & 3) * 4);
    q[0] = w0;
    q[4] = w1;
    if (lane < 16) reinterpret_cast<__half*>(o + XF_BSUMS + (g * 4 + ((lane & 7) >> 1)) * 8)[(lane >> 3) * 2 + (lane & 1)] = bs;
    if (lane == 0) *reinterpret_cast<float*>(o + XF_D + 4 * g) = d;
  }
  if (xt) {
    uint8_t* const o = xt + at * XT_BLOCK;
    *reinterpret_cast<uint2*>(o + s * 128 + g * 16 + h * 8) = make_uint2(w0, w1);
    if (lane < 16) reinterpret_cast<__half*>(o + XT_BSUMS + (lane >> 3) * 128 + g * 16)[lane & 7] = bs;
    int sum = lane < 16 ? bsum : 0;
#pragma unroll
    for (int i = 8; i > 0; i >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, i);
    if (lane < 2) *reinterpret_cast<uint32_t*>(o + (lane ? XT_SUMS : XT_D) + 4 * g) = lane ? (uint32_t)(-4096 * sum) : __float_as_uint(d);
  }
}
// Block b of row `tok` (of nt groups of 8 rows), quantized straight into that order. `wide`: src is
// 16-byte aligned (a buffer read at an offset of the caller's need not be).
__device__ __forceinline__ void warp_quantize_xf(const float* src, uint8_t* xf, uint8_t* xt, int tok, int b, int nt, bool wide) {
  const int lane = threadIdx.x & 31;
  float v[8];
  if (wide) {
    const float4 a = reinterpret_cast<const float4*>(src)[2 * lane], c = reinterpret_cast<const float4*>(src)[2 * lane + 1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = src[8 * lane + i];
  }
  const Q8kLane r = warp_q8k_lane(v);
  const int s2 = r.s + __shfl_xor_sync(0xffffffffu, r.s, 1);
  const int bs = __shfl_sync(0xffffffffu, s2, (2 * lane) & 31);
  xf_store(xf, xt, tok, b, nt, lane, r.w0, r.w1, bs, r.d);
}

template <bool CG = false>
__device__ __forceinline__ void warp_quantize_q8k(const float* src, uint8_t* dst, int image) {
  const int lane = threadIdx.x & 31;
  float v[8];
  if (CG) {
    // data written by other CTAs of the same launch: bypass L1
    float4 a = __ldcg(reinterpret_cast<const float4*>(src) + 2 * lane), b = __ldcg(reinterpret_cast<const float4*>(src) + 2 * lane + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = src[8 * lane + i];
  }
  warp_quantize_q8k_vals(v, dst, image);
}

// quant.rs:231-245 for one 32-value block handled by one warp (lane = element).
__device__ __forceinline__ void warp_quantize_q80(const float* src, uint8_t* dst, int image) {
  const int lane = threadIdx.x & 31;
  float v = src[lane];
  float amax = fabsf(v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  float d = fdiv(amax, 127.0f);
  float id = d != 0.0f ? fdiv(1.0f, d) : 0.0f;
  int q = (int)roundf(fmul(v, id));
  q = q < -127 ? -127 : (q > 127 ? 127 : q);
  reinterpret_cast<int8_t*>(dst + (image ? 0 : 4))[lane] = (int8_t)q;
  if (lane == 0) *reinterpret_cast<float*>(dst + (image ? 32 : 0)) = d;
}

constexpr int XIMG_K = 304;  // bytes per Q8_K block image
constexpr int XIMG_0 = 48;   // bytes per Q8_0 block image

// Quantize `n_total` floats (a multiple of the block size; rows back to back).
__global__ void quantize_q8k_kernel(const float* __restrict__ x, uint8_t* __restrict__ out, int n_blocks, int image) {
  pdl_launch_dependents();
  pdl_wait();
  int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int nw = (gridDim.x * blockDim.x) >> 5;
  for (int b = wid; b < n_blocks; b += nw) warp_quantize_q8k(x + (size_t)b * 256, out + (size_t)b * (image ? XIMG_K : 292), image);
}
// m rows of nb blocks into the fragment order.
__global__ void quantize_xf_kernel(const float* __restrict__ x, uint8_t* __restrict__ xf, uint8_t* __restrict__ xt, int m, int nb) {
  pdl_launch_dependents();
  pdl_wait();
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5, nt = (m + 7) >> 3;
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 15) == 0;  // blocks lie 1024 bytes apart
  for (int i = wid; i < m * nb; i += nw) warp_quantize_xf(x + (size_t)i * 256, xf, xt, i / nb, i % nb, nt, wide);
}
__global__ void quantize_q80_kernel(const float* __restrict__ x, uint8_t* __restrict__ out, int n_blocks, int image) {
  pdl_launch_dependents();
  pdl_wait();
  int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int nw = (gridDim.x * blockDim.x) >> 5;
  for (int b = wid; b < n_blocks; b += nw) warp_quantize_q80(x + (size_t)b * 32, out + (size_t)b * (image ? XIMG_0 : 36), image);
}

// Reference-layout blocks -> images (for callers that hand in BlockQ8_K / BlockQ8_0 arrays).
__global__ void q8k_to_image_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int n_blocks) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_blocks * 73; i += gridDim.x * blockDim.x) {
    int b = i / 73, w = i - b * 73;
    int off = w == 0 ? 288 : (w <= 64 ? (w - 1) * 4 : 256 + (w - 65) * 4);
    *reinterpret_cast<uint32_t*>(out + (size_t)b * XIMG_K + off) = reinterpret_cast<const uint32_t*>(in)[i];
  }
}
__global__ void q80_to_image_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, int n_blocks) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_blocks * 9; i += gridDim.x * blockDim.x) {
    int b = i / 9, w = i - b * 9;
    int off = w == 0 ? 32 : (w - 1) * 4;
    *reinterpret_cast<uint32_t*>(out + (size_t)b * XIMG_0 + off) = reinterpret_cast<const uint32_t*>(in)[i];
  }
}

// ---- rmsnorm (ops.rs:7-18), one CTA per row, optional fused quantization ------------------
// out may alias x. When q8k_out / q80_out are given, the normalised row is also
// quantized (as the generated code does right after every rmsnorm, emit.rs:131-139).
struct RmsnormParams {
  const float* x;
  const float* w;
  float* out;
  int n;
  int x_stride, out_stride;
  float eps;
  int accumulate;    // out[i] = out[i] + y[i] (Gemma post-norm residual join)
  uint8_t* q8k_out;  // images, n/256 per row
  int xf_nt;         // > 0: q8k_out and xt_out (if not null) in the orders of xf_store instead, this many groups of 8 rows
  uint8_t* xt_out;
  uint8_t* q80_out;  // images, n/32 per row
  int w_constant;    // w is a model's: no kernel before this one writes it
};

__global__ void __launch_bounds__(512) rmsnorm_kernel(const RmsnormParams P) {
  extern __shared__ __align__(16) float sm_f[];
  float* row = sm_f;          // n
  float* sq = sm_f + ((P.n + 3) & ~3);  // n, 16-byte aligned, zero-filled to a multiple of eight
  __shared__ SeqSumScratch ssc;
  pdl_launch_dependents();
  // The weights are asked for first: behind the sum they cost a trip to L2 of their own.
  constexpr int NW = 8;
  float w[NW];
  auto weights = [&]() {
#pragma unroll
    for (int k = 0; k < NW; k++) {
      const int i = threadIdx.x + k * 512;
      w[k] = i < P.n ? P.w[i] : 0.0f;
    }
  };
  if (P.w_constant) weights();
  pdl_wait();
  if (!P.w_constant) weights();
  const float* x = P.x + (size_t)blockIdx.x * P.x_stride;
  float* out = P.out + (size_t)blockIdx.x * P.out_stride;
  for (int i = threadIdx.x; i < P.n; i += blockDim.x) {
    float v = x[i];
    row[i] = v;
    sq[i] = fmul(v, v);
  }
  if (P.n + (int)threadIdx.x < ((P.n + 7) & ~7)) sq[P.n + threadIdx.x] = 0.0f;
  float ss = group_seq_sum(sq, P.n, &ssc, CtaGroup{(int)threadIdx.x, (int)blockDim.x, 0});
  float r = fdiv(1.0f, fsqrt(fadd(fdiv(ss, (float)P.n), P.eps)));
  auto scale = [&](int i, float wi) {
    float y = fmul(fmul(row[i], r), wi);
    row[i] = y;
    if (P.out) out[i] = P.accumulate ? fadd(out[i], y) : y;
  };
#pragma unroll
  for (int k = 0; k < NW; k++)
    if ((int)threadIdx.x + k * 512 < P.n) scale(threadIdx.x + k * 512, w[k]);
  for (int i = threadIdx.x + NW * 512; i < P.n; i += 512) scale(i, P.w[i]);
  __syncthreads();
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (P.q8k_out) {
    int nb = P.n / 256;
    for (int b = warp; b < nb; b += nwarps) {
      if (P.xf_nt) warp_quantize_xf(row + b * 256, P.q8k_out, P.xt_out, blockIdx.x, b, P.xf_nt, true);
      else warp_quantize_q8k(row + b * 256, P.q8k_out + ((size_t)blockIdx.x * nb + b) * XIMG_K, 1);
    }
  }
  if (P.q80_out) {
    int nb = P.n / 32;
    for (int b = warp; b < nb; b += nwarps)
      warp_quantize_q80(row + b * 32, P.q80_out + ((size_t)blockIdx.x * nb + b) * XIMG_0, 1);
  }
}

// ---- per-head rmsnorm + RoPE + KV store ("qk post") -----------------------------------------
// After the q/k/v products of one or more tokens: optional per-head RMSNorm of q
// and k (ops.rs:74-87), RoPE in the adjacent-pair or NEOX layout (ops.rs:40-70)
// with the (cos, sin) row of each token's position, then k and v are copied into
// the cache (ops.rs:152-157, 505-510). One CTA per (head slot, token): head slots
// 0..n_head-1 are query heads, n_head..n_head+n_kv-1 key heads (which also move
// the matching value head).
struct QkPostParams {
  float* q;           // m x q_dim, in place
  const float* k;     // m x kv_dim
  const float* v;     // m x kv_dim
  float* k_cache;     // already offset to the layer: ctx x kv_dim
  float* v_cache;
  const float* q_norm;  // head_dim weights or null
  const float* k_norm;
  const float* rope_table;  // ctx x rot_dim, interleaved (cos, sin)
  const int* pos_ptr;       // device word holding pos0 (or null -> pos0 below)
  int pos0;
  int n_head, n_kv_head, head_dim, rot_dim;
  int neox;
  float eps;
};

__global__ void __launch_bounds__(128) qk_post_kernel(const QkPostParams P) {
  __shared__ float h[256];
  __shared__ float sq[256];
  __shared__ float slot;
  pdl_launch_dependents();
  // Nothing here but loads and a few operations, so what is needed is asked for together: the model's tables
  // before the previous kernel ends, the value row beside the head.
  const int hs = blockIdx.x, tok = blockIdx.y, t = threadIdx.x;
  const int hd = P.head_dim, half = P.rot_dim / 2;  // at most 256: two elements and one pair per thread
  const bool is_q = hs < P.n_head;
  const int kvh = hs - P.n_head;
  const int q_dim = P.n_head * hd, kv_dim = P.n_kv_head * hd;
  const float* src = is_q ? P.q + (size_t)tok * q_dim + hs * hd : P.k + (size_t)tok * kv_dim + kvh * hd;
  const float* vs = is_q ? nullptr : P.v + (size_t)tok * kv_dim + kvh * hd;
  const float* nw = is_q ? P.q_norm : P.k_norm;
  float w[2] = {0.0f, 0.0f}, a[2], v[2] = {0.0f, 0.0f}, c = 0.0f, s = 0.0f;
  if (nw) {
    if (t < hd) w[0] = nw[t];
    if (t + 128 < hd) w[1] = nw[t + 128];
  }
  auto angles = [&](int pos) {
    if (t < half) {
      c = P.rope_table[(size_t)pos * P.rot_dim + 2 * t];
      s = P.rope_table[(size_t)pos * P.rot_dim + 2 * t + 1];
    }
  };
  if (!P.pos_ptr) angles(P.pos0 + tok);
  pdl_wait();
  const int pos = (P.pos_ptr ? *P.pos_ptr : P.pos0) + tok;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int i = t + 128 * k;
    if (i < hd) {
      a[k] = src[i];
      if (vs) v[k] = vs[i];
    }
  }
  if (P.pos_ptr) angles(pos);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int i = t + 128 * k;
    if (i < hd) {
      h[i] = a[k];
      sq[i] = fmul(a[k], a[k]);
    }
  }
  if (nw) {
    const float ss = block_seq_sum(sq, hd, &slot);
    const float r = fdiv(1.0f, fsqrt(fadd(fdiv(ss, (float)hd), P.eps)));
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (t + 128 * k < hd) h[t + 128 * k] = fmul(fmul(a[k], r), w[k]);
  }
  __syncthreads();
  float* dst = is_q ? P.q + (size_t)tok * q_dim + hs * hd : P.k_cache + (size_t)pos * kv_dim + kvh * hd;
  if (t < half) {
    const int i0 = P.neox ? t : 2 * t, i1 = P.neox ? t + half : 2 * t + 1;
    const float x0 = h[i0], x1 = h[i1];
    dst[i0] = fsub(fmul(x0, c), fmul(x1, s));
    dst[i1] = fadd(fmul(x0, s), fmul(x1, c));
  }
  float* vd = is_q ? nullptr : P.v_cache + (size_t)pos * kv_dim + kvh * hd;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int i = t + 128 * k;
    if (i >= P.rot_dim && i < hd) dst[i] = h[i];
    if (vd && i < hd) vd[i] = v[k];
  }
}

// Stand-alone pieces of the same, for the operator-level API.
__global__ void rope_kernel(float* x, int m, int n_heads, int head_dim, int rot_dim, const float* cs, int cs_stride,
                            int neox) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  const int half = rot_dim / 2;
  const size_t total = (size_t)m * n_heads * half;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(t % half);
    size_t hh = t / half;
    int row = (int)(hh / n_heads);
    float* v = x + hh * head_dim;
    const float* c_s = cs + (size_t)row * cs_stride;
    int i0 = neox ? i : 2 * i, i1 = neox ? i + half : 2 * i + 1;
    float c = c_s[2 * i], s = c_s[2 * i + 1];
    float x0 = v[i0], x1 = v[i1];
    v[i0] = fsub(fmul(x0, c), fmul(x1, s));
    v[i1] = fadd(fmul(x0, s), fmul(x1, c));
  }
}

__global__ void __launch_bounds__(128) rmsnorm_heads_kernel(float* x, const float* w, int head_dim, float eps) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  __shared__ float h[256];
  __shared__ float sq[256];
  __shared__ float slot;
  float* v = x + (size_t)blockIdx.x * head_dim;
  for (int i = threadIdx.x; i < head_dim; i += blockDim.x) {
    float a = v[i];
    h[i] = a;
    sq[i] = fmul(a, a);
  }
  float ss = block_seq_sum(sq, head_dim, &slot);
  float r = fdiv(1.0f, fsqrt(fadd(fdiv(ss, (float)head_dim), eps)));
  for (int i = threadIdx.x; i < head_dim; i += blockDim.x) v[i] = fmul(fmul(h[i], r), w[i]);
}

// ---- element-wise ----------------------------------------------------------------------------------
__global__ void silu_mul_kernel(float* h, const float* up, size_t n) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v = h[i];
    h[i] = fmul(fdiv(v, fadd(1.0f, expf_exact(-v))), up[i]);
  }
}
// GELU, tanh approximation (ops.rs:124-127): 0.5 v (1 + tanh(k (v + 0.044715 v^3))) with every
// product and sum rounded to f32 in the reference's order. The reference takes tanh from
// the platform's libm; here it is the correctly rounded f32 value (double tanh, then one
// rounding), which is what a correctly rounded libm returns.
__device__ __forceinline__ float gelu_exact(float v) {
  const float k = 1.1283791670955126f / 1.4142135623730951f;  // FRAC_2_SQRT_PI / SQRT_2 in f32
  const float cube = fmul(fmul(fmul(0.044715f, v), v), v);
  const float t = (float)tanh((double)fmul(k, fadd(v, cube)));
  return fmul(fmul(0.5f, v), fadd(1.0f, t));
}
// h = gelu(h) * up (ops.rs:130-134)
__global__ void gelu_mul_kernel(float* h, const float* up, size_t n) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    h[i] = fmul(gelu_exact(h[i]), up[i]);
}
__global__ void add_inplace_kernel(float* x, const float* y, size_t n) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    x[i] = fadd(x[i], y[i]);
}
__global__ void add_bias_rows_kernel(float* x, const float* b, size_t n, size_t m) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n * m; i += (size_t)gridDim.x * blockDim.x)
    x[i] = fadd(x[i], b[i % n]);
}
__global__ void scale_inplace_kernel(float* x, float s, size_t n) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    x[i] = fmul(x[i], s);
}
__global__ void store_kv_kernel(float* k_cache, float* v_cache, const float* k, const float* v, size_t n,
                                const int* pos_ptr, int pos0, int kv_dim) {
  pdl_launch_dependents();
  pdl_wait();  // a launch with programmatic stream serialization must not run ahead of its predecessor
  size_t at = (size_t)(pos_ptr ? *pos_ptr : pos0) * kv_dim;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    k_cache[at + i] = k[i];
    v_cache[at + i] = v[i];
  }
}

// ---- token embedding rows (quant.rs:300-443 through emit.rs:469, 497) ---------------------------------
__global__ void embed_rows_kernel(float* out, const uint8_t* table, const int* tokens, int kind, int dim,
                                  size_t row_bytes, float scale, int do_scale) {
  pdl_launch_dependents();
  pdl_wait();
  const int tok = tokens[blockIdx.y];
  const uint8_t* row = table + (size_t)tok * row_bytes;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < dim; e += gridDim.x * blockDim.x) {
    float v = dequant_elem(kind, row, (size_t)e);
    out[(size_t)blockIdx.y * dim + e] = do_scale ? fmul(v, scale) : v;
  }
}

// ---- greedy argmax (sampler.rs:99-109): the first maximum wins, NaN never does ----------------------------
// `step`, when given, is the device-side decode cursor {token, pos, n_generated}:
// the winner becomes the next step's token, is appended to `history`, and the
// position advances, so a generation loop needs no host round trip per token.
__global__ void __launch_bounds__(1024) argmax_kernel(const float* x, int n, int* out_token, int* step, int* history,
                                                      int history_cap) {
  __shared__ float bv[32];
  __shared__ int bi[32];
  pdl_launch_dependents();
  pdl_wait();
  float best = -INFINITY;
  int idx = 0x7fffffff;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    float v = x[i];
    if (v > best) {
      best = v;
      idx = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float v2 = __shfl_xor_sync(0xffffffffu, best, o);
    int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
    if (v2 > best || (v2 == best && i2 < idx)) {
      best = v2;
      idx = i2;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    bv[threadIdx.x >> 5] = best;
    bi[threadIdx.x >> 5] = idx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      if (bv[w] > best || (bv[w] == best && bi[w] < idx)) {
        best = bv[w];
        idx = bi[w];
      }
    }
    if (idx == 0x7fffffff) idx = 0;  // nothing exceeded -inf
    if (out_token) *out_token = idx;
    if (step) {
      int g = step[2];
      if (history && g < history_cap) history[g] = idx;
      step[0] = idx;
      step[1] = step[1] + 1;
      step[2] = g + 1;
    }
  }
}

}  // namespace aot

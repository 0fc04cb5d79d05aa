// Products of Q4_0 / Q5_0 / Q8_0 matrices with several Q8_0 activation rows on the tensor cores
// (matvec.rs:170-262), bit-identical to the reference.
//
// A result is eight f32 chains ("AVX2 lanes"), one fused multiply-add acc = fma(d_w * d_x, p, acc)
// per 32-weight block, p the integer dot of the lane's four weights: no sum over k may be longer than four
// products. The integer dots come from m16n8k8 f16 instructions with the activations as a
// block-diagonal operand: the eight columns are four tokens x two lanes, and a column holds its
// lane's four activations and zeros for the other lane. Weights and activations are integers of at
// most eight bits, so operands, products and sums are exact, and the results are f32 already.
//
// What bounds it: issue. The matrix instruction gives 128 dots (a dp4a and a conversion for 32 each
// otherwise), the packed multiply-adds of two tokens two results each; the rest is kept short:
//  * weights become f16 fragments once per CTA, four blocks ahead of their use, and every warp of
//    the CTA (16 tokens each) reads them with two 16-byte loads per block and row tile;
//  * activations lie in global memory in fragment order (x0f_kernel) and travel through a private
//    ring per warp; lanes whose operand is the zero half read one 16-byte line of zeros;
//  * a warp holds its 2 x 16 rows x 16 tokens x 8 lanes of sums in registers from the first block
//    to the last.
// Q8_0 14336x4096, 64 rows: 242 us on q80_stream_kernel, 192 here (about 9.7 instructions per matrix
// instruction; a bare loop of loads, products and sums runs with 4.7 at 14 cycles each, 88 us).
// Smaller tiles (one row tile, 8 tokens) fill small launches better but lose what the reuse gains. A
// launch takes 0.7 us per 32 columns and round of two CTAs of four warps per SM, also where the round is
// not full; where that is more than the streaming kernel takes, launch_q80_mma leaves the product to it.
#pragma once
#include <cuda_fp16.h>

#include "mmautils.cuh"
#include "q80stream.cuh"

namespace aot {

constexpr int X0F_BLOCK = 544;      // bytes of one block of eight tokens: 2 x 16 x 16 operand bytes, 8 scales
constexpr int QM_CHUNK = 8;         // blocks of a raw weight chunk: its rows are multiples of 16 bytes for every kind
constexpr int QM_STEP = 4;          // blocks converted at a time
constexpr int QM_XRING = 4;         // activation blocks in a warp's ring
constexpr int QM_FRAG = 1024 + 128; // bytes of a block's fragments: 16 rows x 32 f16 and their scales, each twice
constexpr int QM_RT = 2;             // row tiles of 16 per warp
constexpr int QM_NG = 2;             // token groups of 8 per warp
constexpr int QM_MAX_WARPS = 8;      // one CTA per SM's registers at most, two of four warps

// Reference-layout BlockQ8_0 (36 bytes) or block images -> fragments, a warp per (block, eight tokens).
// Lane (q, h, tok, u) writes elements 2u, 2u+1 of lanes 4h .. 4h+3 of token 4q + tok.
__global__ void __launch_bounds__(256) x0f_kernel(const uint8_t* __restrict__ x, int x_image, uint8_t* __restrict__ out, int m, int nb) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, ntg = (m + 7) >> 3;
  if (wid >= ntg * nb) return;
  const int b = wid / ntg, tg = wid - b * ntg, stride = x_image ? X0_STRIDE : 36;
  uint8_t* const o = out + (size_t)wid * X0F_BLOCK;
  {
    const int tok = 8 * tg + 4 * (lane >> 4) + ((lane >> 1) & 3), h = (lane >> 3) & 1, sh = 16 * (lane & 1);
    uint32_t v[4] = {0, 0, 0, 0};
    if (tok < m) {
      const uint32_t* qs = reinterpret_cast<const uint32_t*>(x + ((size_t)tok * nb + b) * stride + (x_image ? 0 : 4)) + 4 * h;
#pragma unroll
      for (int s = 0; s < 4; s++) {
        const uint32_t w = __ldg(qs + s) >> sh;
        const __half2 p = __halves2half2(__int2half_rn((int)(int8_t)w), __int2half_rn((int)(int8_t)(w >> 8)));
        v[s] = *reinterpret_cast<const uint32_t*>(&p);
      }
    }
    *reinterpret_cast<uint4*>(o + lane * 16) = make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (lane < 8) {  // scales: [u][group of four][token 2u, 2u+1]
    const int u = lane >> 2, q = (lane >> 1) & 1, tok = 8 * tg + 4 * q + 2 * u + (lane & 1);
    float d = 0.0f;
    if (tok < m) d = *reinterpret_cast<const float*>(x + ((size_t)tok * nb + b) * stride + (x_image ? X0_D : 0));
    *reinterpret_cast<float*>(o + 512 + 4 * lane) = d;
  }
}

struct Q80MmaParams {
  GemvSeg seg[3];
  int nseg, cols, m, epilogue;
  int ntg, wt, n_tcta;  // groups of eight tokens, warps of a CTA, CTAs per row unit
  int n_units, units_before[4];
  const uint8_t* xf;        // fragments of all ntg groups
};

template <int KIND>
struct QmShape {
  static constexpr int BS = Q80Kind<KIND>::BS;
  static constexpr int CB = QM_CHUNK * BS;           // bytes of a raw chunk row
  static constexpr int RAW = QM_RT * 16 * CB;           // one chunk
  static constexpr int FRAG = QM_RT * QM_STEP * QM_FRAG;
  static_assert(CB % 16 == 0, "");
  __host__ __device__ static constexpr int unit_bytes(int wt) { return 2 * RAW + 2 * FRAG + wt * QM_XRING * QM_NG * X0F_BLOCK; }
};

__device__ __forceinline__ uint32_t qm_half2(uint32_t bytes, uint32_t sel, __half2 bias) {
  const uint32_t p = __byte_perm(bytes, 0x64646464u, sel);  // two f16: 1024 + byte
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&p), bias);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Weights of lanes 4h + 2p, 4h + 2p + 1 of a block at wb: four biased bytes each.
template <int KIND>
__device__ __forceinline__ void qm_words(uint32_t wb, int h, int p, uint32_t (&v)[2]) {
  uint32_t q = wb + (KIND == Q5_0 ? 6 : 2) + 8 * p + (KIND == Q8_0 ? 16 * h : 0);
  const uint32_t sh = (q & 2u) * 8u;
  q &= ~3u;
  const uint32_t w0 = gm_lds32(q), w1 = gm_lds32(q + 4), w2 = gm_lds32(q + (sh >> 1));
  v[0] = funnel_r(w0, w1, sh);
  v[1] = funnel_r(w1, w2, sh);
#pragma unroll
  for (int s = 0; s < 2; s++) v[s] = KIND == Q8_0 ? v[s] ^ 0x80808080u : (v[s] >> (4 * h)) & 0x0F0F0F0Fu;
  if (KIND == Q5_0) {
    const uint32_t qh = lds32_a2s(wb + 2) >> (16 * h + 8 * p);
#pragma unroll
    for (int s = 0; s < 2; s++) {  // bits 4s .. 4s+3 to bit 4 of the four bytes
      const uint32_t b = qh >> (4 * s);
      v[s] |= ((b & 1u) << 4) | ((b & 2u) << 11) | ((b & 4u) << 18) | ((b & 8u) << 25);
    }
  }
}

__device__ __forceinline__ void mma_f16_k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0), "f"(0.0f));
}
__device__ __forceinline__ void lds_f2x2(uint32_t a, F2& x, F2& y) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(a));
}

// A unit is 32 rows of one matrix (PAIR: 16 rows of both) and is worked on by P.wt warps.
template <int KIND, bool PAIR>
__global__ void __launch_bounds__(QM_MAX_WARPS * 32, 1) q80_mma_kernel(const __grid_constant__ Q80MmaParams P) {
  using S = QmShape<KIND>;
  constexpr int RT = QM_RT, NG = QM_NG;
  constexpr int CB = S::CB, BS = S::BS, ROWS = 16 * RT, PPR = CB / 16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) uint32_t zeros[4 * 8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wt = warp;
  const int tile = blockIdx.x / P.n_tcta, tcta = blockIdx.x - tile * P.n_tcta;
  const int unit = tile, tg = (tcta * P.wt + wt) * NG;
  if (threadIdx.x < 32) zeros[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t raw = smem_addr(smem), frag = raw + 2 * S::RAW,
                 xring = frag + 2 * S::FRAG + (uint32_t)wt * (QM_XRING * NG * X0F_BLOCK);
  int sg = 0;
  if (!PAIR)
    while (sg < P.nseg - 1 && unit >= P.units_before[sg + 1]) sg++;
  const int row0 = (unit - P.units_before[sg]) * (PAIR ? 16 : ROWS), n_rows = P.seg[sg].rows;
  const int nb = P.cols >> 5, n_steps = nb / QM_STEP, n_chunks = nb / QM_CHUNK;
  const uint32_t row_bytes = (uint32_t)nb * BS;
  constexpr int RPI = 32 / PPR;  // rows a warp copies at a time
  const int rl = lane / PPR, pl = lane - rl * PPR;
  auto issue_raw = [&](int c) {
    if (rl < RPI) {
      for (int r = wt * RPI + rl; r < ROWS; r += P.wt * RPI) {
        const int row = min(row0 + (PAIR ? r & 15 : r), n_rows - 1);
        cp_async16(raw + (uint32_t)((c & 1) * S::RAW + r * CB + pl * 16),
                   (PAIR && r >= 16 ? P.seg[1].w : P.seg[sg].w) + (size_t)row * row_bytes + (uint32_t)(c * CB + pl * 16));
      }
    }
  };
  const uint8_t* xsrc = P.xf + (size_t)tg * X0F_BLOCK + lane * 16;
  const size_t xstep = (size_t)P.ntg * X0F_BLOCK;
  const bool live = tg < P.ntg;
  const int xbytes = min(NG, P.ntg - tg) * X0F_BLOCK;
  auto issue_x = [&](int b) {
    if (live && b < nb) {
      const uint32_t dst = xring + (uint32_t)(b & (QM_XRING - 1)) * (NG * X0F_BLOCK) + lane * 16;
#pragma unroll
      for (int i = 0; i < NG * X0F_BLOCK; i += 512)
        if (i + lane * 16 < xbytes) cp_async16(dst + i, xsrc + i);
      xsrc += xstep;
    }
    cp_async_commit();
  };
  // Fragments of step s. Lane (g, tig = 2h + u) of the instruction for lanes 4h + i takes elements
  // 2u, 2u+1 of rows g and g + 8 from byte 512 (i / 2) + 16 lane + 8 (i % 2); it converts here as
  // (g, h, p) both rows' lanes 4h + 2p and 4h + 2p + 1.
  const int cg = lane & 7, ch = (lane >> 3) & 1, cp = lane >> 4;
  const uint32_t csrc = raw + (uint32_t)cg * CB, cdst = frag + (uint32_t)(cp * 512 + (cg * 4 + 2 * ch) * 16);
  auto convert = [&](int s) {
    const __half2 bias = __half2half2(__ushort_as_half(KIND == Q8_0 ? 0x6480 : KIND == Q4_0 ? 0x6408 : 0x6410));
    for (int i = wt; i < RT * QM_STEP; i += P.wt) {
      const uint32_t wb = csrc + (uint32_t)(((s >> 1) & 1) * S::RAW + (i / QM_STEP) * 16 * CB + ((s & 1) * QM_STEP + i % QM_STEP) * BS);
      const uint32_t dst = cdst + (uint32_t)((s & 1) * S::FRAG + i * QM_FRAG);
      uint32_t v[2], w[2];
      qm_words<KIND>(wb, ch, cp, v);
      qm_words<KIND>(wb + 8 * CB, ch, cp, w);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t sel = u ? 0x4342 : 0x4140;
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst + 16 * u), "r"(qm_half2(v[0], sel, bias)), "r"(qm_half2(w[0], sel, bias)),
                     "r"(qm_half2(v[1], sel, bias)), "r"(qm_half2(w[1], sel, bias)) : "memory");
      }
      if (lane < 8) {
        uint32_t h0, h1;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(h0) : "r"(wb));
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(h1) : "r"(wb + 8 * CB));
        asm volatile("st.shared.v4.f32 [%0], {%1, %1, %2, %2};" ::"r"(frag + (uint32_t)((s & 1) * S::FRAG + i * QM_FRAG) + 1024 + lane * 16), "f"(half_bits_hw(h0)),
                     "f"(half_bits_hw(h1)) : "memory");
      }
    }
  };

  issue_raw(0);
  cp_async_commit();
  if (n_chunks > 1) issue_raw(1);
  cp_async_commit();
  pdl_wait();  // weights do not depend on the previous kernel, activations do
#pragma unroll
  for (int b = 0; b < QM_XRING - 1; b++) issue_x(b);
  cp_async_wait<QM_XRING>();
  __syncthreads();
  convert(0);

  const int g = lane >> 2, tig = lane & 3, h = tig >> 1;
  const bool nz = h == (g >> 2);  // this lane's half of the block-diagonal operand
  const uint32_t xoff = (uint32_t)((h * 4 + (g & 3)) * 2 + (tig & 1)) * 16, zaddr = smem_addr(zeros) + (g & 1 ? 0u : 64u);
  F2 acc[RT][2 * NG][2][4];  // [row tile][group of four tokens][row g, g + 8][lane 4h + i], two tokens each
#pragma unroll
  for (int i = 0; i < RT * NG * 16; i++) (&acc[0][0][0][0])[i] = 0ull;
#pragma unroll 1
  for (int s = 0; s < n_steps; s++) {
    __syncthreads();
    if ((s & 1) && (s + 3) / 2 < n_chunks) issue_raw((s + 3) / 2);  // goes with the next activation group
    if (s + 1 < n_steps) convert(s + 1);
    const uint32_t fs = frag + (uint32_t)((s & 1) * S::FRAG);
#pragma unroll 1
    for (int j = 0; j < QM_STEP; j++) {
      cp_async_wait<QM_XRING - 2>();
      __syncwarp();
      issue_x(QM_STEP * s + j + QM_XRING - 1);
      const uint32_t xb = xring + (uint32_t)(j & (QM_XRING - 1)) * (NG * X0F_BLOCK);
      U4 b4[2 * NG];
      F2 dx[2 * NG];
#pragma unroll
      for (int q = 0; q < 2 * NG; q++) b4[q] = gm_lds128(nz ? xb + (q >> 1) * X0F_BLOCK + (q & 1) * 256 + xoff : zaddr);
#pragma unroll
      for (int n = 0; n < NG; n++) lds_f2x2(xb + n * X0F_BLOCK + 512 + (tig & 1) * 16, dx[2 * n], dx[2 * n + 1]);
#pragma unroll
      for (int rt = 0; rt < RT; rt++) {
        const uint32_t fb = fs + (uint32_t)((rt * QM_STEP + j) * QM_FRAG);
        const U4 a[2] = {gm_lds128(fb + lane * 16), gm_lds128(fb + 512 + lane * 16)};
        F2 dw0, dw1;
        lds_f2x2(fb + 1024 + g * 16, dw0, dw1);
#pragma unroll
        for (int q = 0; q < 2 * NG; q++) {
          const F2 d0 = f2_mul(dw0, dx[q]), d1 = f2_mul(dw1, dx[q]);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            float c[4];
            mma_f16_k8(c, u4_get(a[i >> 1], 2 * (i & 1)), u4_get(a[i >> 1], 2 * (i & 1) + 1), u4_get(b4[q], i));
            acc[rt][q][0][i] = f2_fma(d0, f2_pack(c[0], c[1]), acc[rt][q][0][i]);
            acc[rt][q][1][i] = f2_fma(d1, f2_pack(c[2], c[3]), acc[rt][q][1][i]);
          }
        }
      }
    }
  }
  cp_async_wait<0>();
  pdl_launch_dependents();  // not before: CTAs of the next launch would share SMs with this one's last wave
  if (!live) return;
  // ((a0+a4)+(a2+a6)) + ((a1+a5)+(a3+a7)): the partner lane holds the other four; lane h stores row g + 8h
#pragma unroll
  for (int q = 0; q < 2 * NG; q++) {
    float v[RT][2];
#pragma unroll
    for (int rt = 0; rt < RT; rt++) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        F2 t[4];
#pragma unroll
        for (int i = 0; i < 4; i++) t[i] = f2_add(acc[rt][q][r][i], __shfl_xor_sync(0xffffffffu, acc[rt][q][r][i], 2));
        const F2 y = f2_add(f2_add(t[0], t[2]), f2_add(t[1], t[3]));
        if (h == r) f2_unpack(y, v[rt][0], v[rt][1]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int tok = 8 * tg + 4 * q + 2 * (tig & 1) + j;
      if (tok >= P.m) continue;
      if (PAIR) {
        const int row = row0 + g + 8 * h;
        if (row < n_rows) {
          const size_t o = (size_t)tok * n_rows + row;
          P.seg[0].out[o] = P.epilogue == EPI_SILU_MUL ? silu_mul_exact(v[0][j], v[RT - 1][j]) : v[0][j];
          P.seg[1].out[o] = v[RT - 1][j];
        }
      } else {
#pragma unroll
        for (int rt = 0; rt < RT; rt++) {
          const int row = row0 + 16 * rt + g + 8 * h;
          if (row < n_rows) {
            float* const o = P.seg[sg].out + (size_t)tok * n_rows + row;
            *o = P.epilogue == EPI_ACCUM ? fadd(*o, v[rt][j]) : v[rt][j];
          }
        }
      }
    }
  }
}

}  // namespace aot

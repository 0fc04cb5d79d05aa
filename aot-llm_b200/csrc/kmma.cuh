// Q4_K / Q5_K / Q6_K matrices against 2..64 activation rows on warp-level int8 tensor-core
// tiles (matmul_rows of crates/aot-kernels/src/matvec.rs:479-522): the batches and matrices that are
// too small for ktensor.cuh.
//
// What bounds it. A product costs, per 16 weight rows x 64 tokens x 256 weights, 64 (Q6_K: 128)
// MMAs of 8 issue cycles and four integer multiply-adds per MMA and lane for the sub-block
// scales; streaming the weights is an order of magnitude cheaper. So everything else has to
// be paid once per weight, not once per token group:
//  * a warp owns one super-block of 16 (RT = 1) or 32 (RT = 2) rows and all tokens: the nibbles
//    are unpacked into A fragments once and stay in registers while the tokens pass by, eight
//    at a time;
//  * the warps of a CTA split a tile's super-blocks, WK at a time; every warp leaves its blocks'
//    f32 terms in shared memory and, after a barrier, each thread adds the terms of its outputs
//    in block order: the order of the single-row products, so batched == single bit for bit
//    (crates/aot-kernels/tests/dots.rs:205-266);
//  * activations come from global memory (they stay in L2) in fragment order (layout below);
//    they and the weight blocks travel through small rings of the warp's own, filled with
//    cp.async, so that warps wait for each other only where terms change hands;
//  * the mins term sum_j m_j * (bsums[2j] + bsums[2j+1]) is one f16 MMA per block (mins <= 63 and
//    16-element sums <= 2048 are exact in f16, their products and sums in f32) instead of eight
//    dp2a per output.
// Measured (back-to-back launches, us; the kernels it replaced in brackets): 4096 x 14336 x 64
// Q4_K 43 (230), Q6_K 58 (322); 4096 x 4096 x 64 Q4_K 14 (47); 2048 x 2048 x 64 Q4_K 7.4 (17).
// About 1040 instructions per 16 rows x 64 tokens x 256 weights at 0.45 per cycle and scheduler:
// MMA and shared-memory latencies of two warps per scheduler are what is left. 16 warps of 128
// registers and one row tile each were slower (50 us: 1725 instructions), as were bulk copies of
// the token groups by one lane (48 us).
//
// Activation fragments ("XF"), [super-block][token group of 8]: 2336 bytes =
//   4 x 32 lanes x 16 bytes  int8: lane (g = token, q), chunk c: bytes 4q..4q+3 of the 16-element
//                            groups 4c .. 4c+3 (the B operands of m16n8k32 / m16n8k16)
//   32 lanes x 8 bytes       f16 sums of 16-element groups 2q, 2q+1, 2q+8, 2q+9
//   8 x f32                  block scales of the 8 tokens
#pragma once
#include <cuda_fp16.h>

#include "mmautils.cuh"
#include "ops.cuh"
#include "rowdot.cuh"

namespace aot {

constexpr int KM_WARPS = 8;
constexpr int KM_MAX_M = 64;
constexpr int KM_PARK = 2;       // token groups whose terms are parked at a time
constexpr int KM_B_SLOTS = 3;    // token groups in a ring

// Reference-layout BlockQ8_K (292 bytes) or block images (304 bytes) -> the orders of xf_store; a warp
// per (token slot, super-block), slots past the last token zeroed.
__global__ void __launch_bounds__(256) xf_kernel(const uint8_t* __restrict__ x, int x_image, uint8_t* __restrict__ xf, uint8_t* __restrict__ xt, int m, int nb) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nt = (m + 7) >> 3;
  if (wid >= nt * 8 * nb) return;
  const int tok = wid / nb, b = wid - tok * nb;
  uint32_t w0 = 0, w1 = 0;
  int bs = 0;
  float d = 0.0f;
  if (tok < m) {
    const uint8_t* p = x + ((size_t)tok * nb + b) * (x_image ? XK_STRIDE : 292);
    const uint32_t* qs = reinterpret_cast<const uint32_t*>(p + (x_image ? 0 : 4));
    w0 = __ldg(qs + 2 * lane);
    w1 = __ldg(qs + 2 * lane + 1);
    if (lane < 16) bs = reinterpret_cast<const int16_t*>(p + (x_image ? XK_BSUMS : 260))[lane];
    d = *reinterpret_cast<const float*>(p + (x_image ? XK_D : 0));
  }
  xf_store(xf, xt, tok, b, nt, lane, w0, w1, bs, d);
}

struct KmmaParams {
  GemvSeg seg[3];
  int nseg, cols, m, nt, epilogue;  // nt: token groups of this launch (at most 8)
  int xf_nt;                        // token groups of the fragment buffer
  const uint8_t* xf;                // its first group of this launch
  int tiles_before[4];              // first tile of each matrix (pair: one list for both)
  int n_tiles;
  int n_stages;                     // weight blocks in a warp's ring
};

// m16n8k16 f16 x f16 -> f32 from a zero accumulator.
__device__ __forceinline__ void mma_f16_k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void mma_s8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
               : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
               : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ uint32_t half2_of_int(int v) {  // (v, v), |v| <= 2048
  const uint32_t h = __half_as_ushort(__int2half_rn(v));
  return h | (h << 16);
}

// One warp's super-block of 16 weight rows as MMA operands: lane (g, q) holds rows g and g + 8.
template <int KIND>
struct KFrag {
  static constexpr int NSC = KIND == Q6_K ? 4 : 8;  // scales per row: one per sub-block, Q6_K packed by four
  uint32_t a[32];     // K4: [sub-block j][a0..a3]; Q6_K: [group s][a0, a1], q - 32 as signed bytes
  int sc[2][NSC];
  uint32_t mins[4];   // K4: A operand of the mins MMA
  float d[2], dmin[2];

  // pa, pb: shared addresses of the block in rows g and g + 8
  __device__ __forceinline__ void load(uint32_t pa, uint32_t pb, int q) {
    if (KIND == Q6_K) {
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const uint32_t p = r ? pb : pa;  // 2-byte aligned
        const uint32_t sh = (p & 2u) * 8u, base = p & ~3u;
        auto word = [&](int off) { return funnel_r(gm_lds32(base + off), gm_lds32(base + off + 4), sh); };
#pragma unroll
        for (int n = 0; n < 2; n++) {
#pragma unroll
          for (int hh = 0; hh < 2; hh++) {
            const uint32_t l0 = word(64 * n + 16 * hh + 4 * q), l32 = word(64 * n + 16 * hh + 32 + 4 * q);
            const uint32_t h = word(128 + 32 * n + 16 * hh + 4 * q);
#pragma unroll
            for (int qu = 0; qu < 4; qu++) {
              const uint32_t l = (qu & 1) ? l32 : l0;
              const uint32_t lo = ((qu & 2) ? l >> 4 : l) & 0x0F0F0F0Fu;
              const uint32_t hi = (qu == 0 ? h << 4 : qu == 1 ? h << 2 : qu == 2 ? h : h >> 2) & 0x30303030u;
              const uint32_t v = lo | hi | 0x80808080u;
              a[2 * (8 * n + 2 * qu + hh) + r] = (v - 0x20202020u) ^ 0x80808080u;  // 0..63 -> -32..31, no borrow between bytes
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) sc[r][i] = (int)word(192 + 4 * i);
        uint32_t h;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(h) : "r"(p + 208));
        d[r] = half_bits_hw(h);
      }
      return;
    }
    constexpr bool Q5 = KIND == Q5_K;
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const uint32_t p = r ? pb : pa;  // 16-byte aligned
      const U4 hdr = gm_lds128(p);
      d[r] = half_bits_hw(hdr.x & 0xFFFFu);
      dmin[r] = half_bits_hw(hdr.x >> 16);
      const K4Scales s = k4_unpack(hdr.y, hdr.z, hdr.w);
#pragma unroll
      for (int j = 0; j < 8; j++) sc[r][j] = byte_of(j < 4 ? s.sc_lo : s.sc_hi, j & 3);
      mins[r] = half2_of_int((int)((s.m_lo >> (8 * q)) & 0xFFu));      // groups 2q, 2q + 1: sub-block q
      mins[2 + r] = half2_of_int((int)((s.m_hi >> (8 * q)) & 0xFFu));  // groups 2q + 8, 2q + 9: sub-block q + 4
      uint32_t h0 = 0, h1 = 0;
      if (Q5) {
        h0 = gm_lds32(p + 16 + 4 * q);
        h1 = gm_lds32(p + 32 + 4 * q);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const uint32_t qs = p + (Q5 ? 48 : 16) + 32 * c + 4 * q;
        const uint32_t w0 = gm_lds32(qs), w1 = gm_lds32(qs + 16);
#pragma unroll
        for (int hi = 0; hi < 2; hi++) {
          const int j = 2 * c + hi;
          uint32_t v0 = (hi ? w0 >> 4 : w0) & 0x0F0F0F0Fu, v1 = (hi ? w1 >> 4 : w1) & 0x0F0F0F0Fu;
          if (Q5) {
            v0 |= ((h0 >> j) & 0x01010101u) << 4;
            v1 |= ((h1 >> j) & 0x01010101u) << 4;
          }
          a[4 * j + r] = v0;
          a[4 * j + 2 + r] = v1;
        }
      }
    }
  }

  // f32 terms of the block against 8 tokens: t[0], t[1] row g tokens 2q, 2q + 1; t[2], t[3] row g + 8.
  __device__ __forceinline__ void terms(const uint4 (&b)[4], const uint2& bs, const float2& dx, float (&t)[4]) const {
    int s[4] = {0, 0, 0, 0};
    float sm[4];
    if (KIND != Q6_K) mma_f16_k16(sm, mins[0], mins[1], mins[2], mins[3], bs.x, bs.y);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t w[4] = {b[c].x, b[c].y, b[c].z, b[c].w};
      if (KIND == Q6_K) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int k = 4 * c + i;
          int cc[4];
          mma_s8s8_k16(cc, a[2 * k], a[2 * k + 1], w[i]);
          const int ca = sext_byte((uint32_t)sc[0][c], i), cb = sext_byte((uint32_t)sc[1][c], i);
          s[0] += ca * cc[0];
          s[1] += ca * cc[1];
          s[2] += cb * cc[2];
          s[3] += cb * cc[3];
        }
      } else {
#pragma unroll
        for (int hi = 0; hi < 2; hi++) {
          const int j = 2 * c + hi;
          int cc[4];
          mma_u8s8_k32(cc, a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3], w[2 * hi], w[2 * hi + 1]);
          const int ca = sc[0][j], cb = sc[1][j];
          s[0] += ca * cc[0];
          s[1] += ca * cc[1];
          s[2] += cb * cc[2];
          s[3] += cb * cc[3];
        }
      }
    }
    // two tokens of a row at a time
    const F2 x = f2_pack(dx.x, dx.y);
#pragma unroll
    for (int r = 0; r < 2; r++) {
      F2 v = f2_mul(f2_mul(f2_pack(d[r], d[r]), x), f2_pack(i2f(s[2 * r]), i2f(s[2 * r + 1])));
      f2_unpack(v, t[2 * r], t[2 * r + 1]);
      if (KIND != Q6_K) {
        // (scalar subtractions: ptxas contracts a packed product and sum into one rounding)
        v = f2_mul(f2_mul(f2_pack(dmin[r], dmin[r]), x), f2_pack(sm[2 * r], sm[2 * r + 1]));
        float m0, m1;
        f2_unpack(v, m0, m1);
        t[2 * r] = fsub(t[2 * r], m0);
        t[2 * r + 1] = fsub(t[2 * r + 1], m1);
      }
    }
  }
};

// One token group's fragments of a super-block, from the warp's ring.
struct XFrag {
  uint4 b[4];
  uint2 bs;
  float2 dx;
  __device__ __forceinline__ void load(uint32_t p, int lane) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const U4 v = gm_lds128(p + 512 * c + 16 * lane);
      b[c] = make_uint4(v.x, v.y, v.z, v.w);
    }
    gm_lds64(p + XF_BSUMS + 8 * lane, bs.x, bs.y);
    uint32_t d0, d1;
    gm_lds64(p + XF_D + 8 * (lane & 3), d0, d1);
    dx = make_float2(__uint_as_float(d0), __uint_as_float(d1));
  }
};

// A CTA: 8 warps, WK of them per row group splitting its super-blocks. A warp holds RT row tiles
// (PAIR, RT = 2: the gate and the up tile of the same rows), which share its activation loads.
template <int KIND, int RT, bool PAIR, int WK>
struct KmmaShape {
  static constexpr int WM = KM_WARPS / WK;                     // row groups
  static constexpr int UNITS = PAIR ? WM : WM * RT;            // row tiles whose outputs are finished together
  static constexpr int UPT = (UNITS + 1) / 2;                  // of them per thread
  static constexpr int ROWS = 16 * UNITS;                      // rows of the row space per CTA tile
  static constexpr int TERMS = KM_WARPS * RT * KM_PARK * 128;  // floats of one terms buffer
  static constexpr int BS = KIND == Q4_K ? 144 : KIND == Q5_K ? 176 : 210;
  // A row's block in the weight ring: 16-byte pieces (Q6_K: of the aligned superset) and a pitch
  // that puts the eight rows of a fragment on different banks.
  static constexpr int PIECES = KIND == Q6_K ? 14 : BS / 16;
  static constexpr int PITCH = KIND == Q6_K ? 240 : BS;
  static constexpr int A_SLOT = 16 * RT * PITCH;
  static constexpr int FIXED = 2 * TERMS * 4 + KM_WARPS * KM_B_SLOTS * XF_BLOCK;  // shared memory besides the weight rings
};

template <bool PAIR>
__device__ __forceinline__ int kmma_seg(const KmmaParams& P, int tile) {
  int sg = 0;
  while (!PAIR && sg < P.nseg - 1 && tile >= P.tiles_before[sg + 1]) sg++;
  return sg;
}

// A CTA walks its tiles stage by stage (WK super-blocks of a tile); a warp's task is its
// super-block of one stage. Weight blocks and token groups arrive through rings of the
// warp's own, filled with cp.async, so warps meet only at the barrier after every KM_PARK token
// groups. One instantiation per weight kind: with the three kinds in one kernel the register
// allocator spills the fragments, which costs 5x.
template <int KIND, int RT, bool PAIR, int WK>
__global__ void __launch_bounds__(KM_WARPS * 32, 1) kmma_kernel(const __grid_constant__ KmmaParams P) {
  using S = KmmaShape<KIND, RT, PAIR, WK>;
  constexpr int NQ = KM_MAX_M / (8 * KM_PARK), UPT = S::UPT;
  extern __shared__ __align__(128) uint8_t smem[];
  // [terms x 2][token group rings][weight rings]
  float* const terms = reinterpret_cast<float*>(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wk = warp % WK, wm = warp / WK, g = lane >> 2, q = lane & 3;
  const uint32_t b_ring = smem_addr(smem) + 2 * S::TERMS * 4 + warp * (KM_B_SLOTS * XF_BLOCK);
  const uint32_t a_ring = smem_addr(smem) + S::FIXED + warp * (P.n_stages * S::A_SLOT);
  const int nb = P.cols >> 8, n_st = (nb + WK - 1) / WK, nt = P.nt, na = P.n_stages;
  const uint32_t xf_sb = (uint32_t)P.xf_nt * XF_BLOCK;
  const size_t row_bytes = (size_t)nb * S::BS;
  pdl_launch_dependents();

  // ---- weight ring: four lanes per row, eight rows at a time ----
  int a_tile = blockIdx.x, a_s = 0, a_slot = 0;  // the next task to request
  auto issue_a = [&]() {
    if (a_tile < P.n_tiles && a_s * WK + wk < nb) {
      const int sg0 = kmma_seg<PAIR>(P, a_tile), r0 = (a_tile - P.tiles_before[sg0]) * S::ROWS + wm * 16 * (PAIR ? 1 : RT);
#pragma unroll
      for (int rt = 0; rt < RT; rt++) {
        const GemvSeg& G = P.seg[PAIR ? rt : sg0];
        const uint8_t* const base = G.w + (size_t)(a_s * WK + wk) * S::BS;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          // rows past the matrix repeat its last row; their results are dropped
          const uint8_t* src = base + (size_t)min(r0 + (PAIR ? 0 : rt * 16) + h * 8 + g, G.rows - 1) * row_bytes;
          if (KIND == Q6_K) src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15);
          src += q * 16;
          const uint32_t dst = a_ring + a_slot * S::A_SLOT + (rt * 16 + h * 8 + g) * S::PITCH + q * 16;
#pragma unroll
          for (int j = 0; j < (S::PIECES + 3) / 4; j++)
            if (4 * j + 3 < S::PIECES || 4 * j + q < S::PIECES) cp_async16(dst + 64 * j, src + 64 * j);
        }
      }
    }
    if (++a_slot == na) a_slot = 0;
    if (++a_s == n_st) {
      a_s = 0;
      a_tile += gridDim.x;
    }
  };
  // ---- token group ring; one commit group per token group, with the weights requested before it ----
  const uint8_t* b_src = P.xf + (size_t)wk * xf_sb + lane * 16;  // the next group to request
  int b_n = 0, b_sb = wk;
  uint32_t b_dst = b_ring + lane * 16;
  auto issue_b = [&]() {
    if (b_sb < nb) {
#pragma unroll
      for (int i = 0; i < 5; i++)
        if (i < 4 || lane < XF_BLOCK / 16 - 128) cp_async16(b_dst + 512 * i, b_src + 512 * i);
    }
    cp_async_commit();
    b_src += XF_BLOCK;
    b_dst = b_dst == b_ring + lane * 16 + (KM_B_SLOTS - 1) * XF_BLOCK ? b_ring + lane * 16 : b_dst + XF_BLOCK;
    if (++b_n == nt) {
      b_n = 0;
      b_sb += WK;
      if (b_sb >= n_st * WK) b_sb = wk;
      b_src = P.xf + (size_t)b_sb * xf_sb + lane * 16;
    }
  };
  // weights do not depend on the previous kernel, activations do
  for (int i = 0; i < na - 1; i++) issue_a();
  pdl_wait();
#pragma unroll
  for (int i = 0; i < KM_B_SLOTS - 1; i++) issue_b();
  const bool deep = (na - 1) * nt >= KM_B_SLOTS - 1;  // a task's weights lie behind the groups a wait leaves pending

  int c_slot = 0;
  uint32_t x_at = b_ring;
  uint32_t buf = 0;
  // this thread's outputs: token group (tid >> 6) & 1 of every KM_PARK, two tokens of one row of units tid >> 7, + 2, ...
  const int nti = (tid >> 6) & 1, u0 = tid >> 7, pos = tid & 63;
#pragma unroll 1
  for (int tile = blockIdx.x; tile < P.n_tiles; tile += gridDim.x) {
    const int sg = kmma_seg<PAIR>(P, tile), r0 = (tile - P.tiles_before[sg]) * S::ROWS;
    float2 acc[NQ][UPT][PAIR ? 2 : 1];
#pragma unroll
    for (int i = 0; i < NQ; i++)
#pragma unroll
      for (int j = 0; j < UPT; j++)
#pragma unroll
        for (int k = 0; k < (PAIR ? 2 : 1); k++) acc[i][j][k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int s = 0; s < n_st; s++) {
      const int sb = s * WK + wk, cnt = min(WK, nb - s * WK);
      const bool active = sb < nb;
      KFrag<KIND> f[RT];
      // one task's weights and one token group ahead of the ring, into slots read before this
      __syncwarp();
      issue_a();
      issue_b();
      if (deep) cp_async_wait<KM_B_SLOTS - 1>();
      else cp_async_wait<0>();
      __syncwarp();
      if (active) {
#pragma unroll
        for (int rt = 0; rt < RT; rt++) {
          uint32_t row[2];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            row[h] = a_ring + c_slot * S::A_SLOT + (rt * 16 + h * 8 + g) * S::PITCH;
            if (KIND == Q6_K) {
              const GemvSeg& G = P.seg[PAIR ? rt : sg];
              const int r = min(r0 + wm * 16 * (PAIR ? 1 : RT) + (PAIR ? 0 : rt * 16) + h * 8 + g, G.rows - 1);
              row[h] += ((uint32_t)(uintptr_t)G.w + (uint32_t)(r * nb + sb) * 210u) & 15u;
            }
          }
          f[rt].load(row[0], row[1], q);
        }
      }
      if (++c_slot == na) c_slot = 0;
#pragma unroll
      for (int qd = 0; qd < NQ; qd++) {
        const int nn = min(KM_PARK, nt - qd * KM_PARK);
        if (nn <= 0) break;
        float* const tb = terms + buf * S::TERMS;
        buf ^= 1u;
        float* td = tb + warp * RT * KM_PARK * 128 + lane * 4;
#pragma unroll 1
        for (int i = 0; i < nn; i++) {
          if (qd != 0 || i != 0) {
            __syncwarp();  // every lane has read the slot that is requested now
            issue_b();
            cp_async_wait<KM_B_SLOTS - 1>();
            __syncwarp();
          }
          if (active) {
            XFrag x;
            x.load(x_at, lane);
#pragma unroll
            for (int rt = 0; rt < RT; rt++) {
              float t[4];
              f[rt].terms(x.b, x.bs, x.dx, t);
              *reinterpret_cast<float4*>(td + rt * KM_PARK * 128) = make_float4(t[0], t[1], t[2], t[3]);
            }
          }
          x_at = x_at == b_ring + (KM_B_SLOTS - 1) * XF_BLOCK ? b_ring : x_at + XF_BLOCK;
          td += 128;
        }
        __syncthreads();
        // the stage's terms of this thread's outputs, in block order
        if (nti < nn) {
#pragma unroll
          for (int j = 0; j < UPT; j++) {
            const int u = u0 + 2 * j;
            if (S::UNITS % 2 == 0 || u < S::UNITS) {
#pragma unroll
              for (int k = 0; k < (PAIR ? 2 : 1); k++) {
                const int w0 = PAIR ? u * WK : u / RT * WK, rt = PAIR ? k : u % RT;
                const float* tp = tb + ((w0 * RT + rt) * KM_PARK + nti) * 128 + 2 * pos;
                float2 v[WK];
#pragma unroll
                for (int w = 0; w < WK; w++)
                  if (w < cnt) v[w] = *reinterpret_cast<const float2*>(tp + w * RT * KM_PARK * 128);
#pragma unroll
                for (int w = 0; w < WK; w++)
                  if (w < cnt) {
                    acc[qd][j][k].x = fadd(acc[qd][j][k].x, v[w].x);
                    acc[qd][j][k].y = fadd(acc[qd][j][k].y, v[w].y);
                  }
              }
            }
          }
        }
      }
    }
    const int l2 = pos >> 1, rr = (l2 >> 2) + 8 * (pos & 1);
    const GemvSeg& G = P.seg[sg];
#pragma unroll
    for (int j = 0; j < UPT; j++) {
      const int u = u0 + 2 * j, row = r0 + u * 16 + rr;
      if (u >= S::UNITS || row >= G.rows) continue;
#pragma unroll
      for (int qd = 0; qd < NQ; qd++) {
        const int tok = (qd * KM_PARK + nti) * 8 + 2 * (l2 & 3);
#pragma unroll
        for (int e = 0; e < 2; e++) {
          if (tok + e >= P.m) continue;
          const size_t o = (size_t)(tok + e) * G.rows + row;
          const float v = e ? acc[qd][j][0].y : acc[qd][j][0].x;
          if (PAIR) {
            const float2 a = acc[qd][j][PAIR ? 1 : 0];
            const float up = e ? a.y : a.x;
            P.seg[0].out[o] = P.epilogue == EPI_SILU_MUL ? silu_mul_exact(v, up) : v;
            P.seg[1].out[o] = up;
          } else {
            G.out[o] = P.epilogue == EPI_ACCUM ? fadd(G.out[o], v) : v;
          }
        }
      }
    }
  }
  cp_async_wait<0>();
}

}  // namespace aot

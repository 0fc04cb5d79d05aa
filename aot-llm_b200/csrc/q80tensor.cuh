// Q4_0 / Q5_0 / Q8_0 matrices against several Q8_0 activation rows on the tensor cores: tcgen05.mma
// kind::f16 (matvec.rs:170-262).
//
// A result is eight f32 chains ("AVX2 lanes"), one fused multiply-add acc = fma(d_w * d_x, p, acc) per
// 32-weight block, p the integer dot of the chain's four weights: no sum over k may be longer than four
// products. So the activations are a block-diagonal operand: a step of 16 weights has four chains, and
// the columns of B are (token, chain), with the chain's four activations and zeros for the others.
// Weights and activations are integers of at most eight bits: operands, products and sums are exact, and
// the results in tensor memory are f32 already. Three quarters of the products are with zeros, which
// the tensor cores have to spare.
//
// What bounds it: instructions of the warps that run the chains. A block of 128 rows x 32 tokens needs
// 390 cycles of their packed multiply-adds and scales and takes 930 (24 tokens 780, 16 tokens 680), its
// MMAs 128. Measured with the conversion of the activations (us; the faster of the kernels before in
// brackets): Q8_0 14336 x 4096, 64 rows 131 (196; 129 before the lanes of a warp voted on their waits), 33 rows 110 (181), 17 rows 58 (114); Q4_0 6144 x 4096,
// 40 rows 51 (95). Tried: a wait and a release per step instead of per block 187; scalar multiply-adds, no
// faster in their pipe, 1265 cycles against 1410 at 32 tokens but 940 against 830 at 16; the weights in
// tensor memory, which leaves room for fewer results.
// Warp roles of a CTA, which walks tiles of 128 weight rows x T tokens, T = 4 * TPW:
//   warp 0        requests: eight blocks of the rows and of the tokens per stage, two tensor copies
//   warp 1        tensor memory, MMAs: a block's results are 8 * T columns
//   warps 2, 3    activations: bytes -> f16 on the diagonal (the zeros are written once), scales
//   warps 4..7    weights: thread = row; block -> f16 core matrices, scale
//   warps 8..23   chains: thread = row and TPW tokens, its 8 * TPW sums in registers from the first block to
//                 the last; tensor memory -> multiply-adds; at the end the fixed tree and the outputs
#pragma once
#include <cuda_fp16.h>

#include "ktensor.cuh"

namespace aot {

constexpr int QT_THREADS = 768;
constexpr int QT_CHUNK = 8;    // blocks of a stage: their rows are multiples of 16 bytes for every kind
constexpr int QT_SLOTS = 6;    // blocks between the warps that prepare them and the chains
constexpr int QT_MAX_RAW = 3;
constexpr int QT_A = KT_ROWS * 64;  // bytes of a block's weights, two steps
// registers move in warpgroups: four of chains, two of the others; 80 per thread at launch
constexpr int QT_REGS_CHAINS = 96, QT_REGS_REST = 48;
static_assert(512 * QT_REGS_CHAINS + 256 * QT_REGS_REST <= QT_THREADS * 80, "more registers than the CTA is launched with");
constexpr int QT_BARS = 2 * QT_MAX_RAW + 3 * QT_SLOTS + 1;

struct QtParams {
  alignas(64) CUtensorMap map[3];  // each matrix as u32 [rows][row_bytes / 4], box [128, pair: 64][a stage's words]
  alignas(64) CUtensorMap xmap;    // activation images as u32 [m][nb * 12], box [T][96]
  GemvSeg seg[3];
  int nseg, cols, m, pair, epilogue;
  int tiles_before[4];             // first row tile of each matrix (pair: one list, 64 rows of both per tile)
  int n_tiles, n_groups;           // row tiles, groups of T tokens
  int n_raw;
  int give_up;                     // stages requested after which the CTA's waits end (0: never)
  int* err;
};

template <int V>
struct QtInt {
  static constexpr int value = V;
};
template <int KIND>
struct QtKind {
  static constexpr int BS = KIND == Q4_0 ? 18 : KIND == Q5_0 ? 22 : 34;
  static constexpr int PITCH = BS * QT_CHUNK;  // odd in 16-byte units: a row per thread meets no bank conflicts
  static constexpr int RAW = KT_ROWS * PITCH;
};
template <int TPW>
struct QtShape {
  static constexpr int T = 4 * TPW, N = 4 * T;   // tokens of a CTA, columns of a step
  static constexpr int X = T * QT_CHUNK * X0_STRIDE;  // bytes of a stage's activations
  static constexpr int STEP = N * 32, B = 2 * STEP;   // bytes of a step's and of a block's operand
  static constexpr int XCH = 512 * (TPW / 2) * 4;     // pairs: exchange between gate and up rows
  static constexpr int SETS = 512 / (2 * N);          // blocks whose results tensor memory holds
};
template <int KIND, int TPW>
constexpr size_t qt_smem(int n_raw, bool pair) {
  return (size_t)n_raw * (QtKind<KIND>::RAW + QtShape<TPW>::X) + QT_SLOTS * (QtShape<TPW>::B + QT_A + KT_ROWS * 4 + 256) + (QT_BARS + 3) / 2 * 16 + 16 +
         (pair ? QtShape<TPW>::XCH : 0);
}

// Four signed bytes as f16: w has them offset by 128, `minus` is 1024 + 128 as a negative pair.
__device__ __forceinline__ uint2 qt_halves(uint32_t w, uint32_t minus) {
  uint32_t a = prmt(w, 0x64u, 0x4140), b = prmt(w, 0x64u, 0x4342);
  asm("add.rn.f16x2 %0, %0, %1;" : "+r"(a) : "r"(minus));
  asm("add.rn.f16x2 %0, %0, %1;" : "+r"(b) : "r"(minus));
  return make_uint2(a, b);
}

// Block J of the row's stage at shared address p: 32 weights as f16 at a, in core matrices of 8 rows x 16
// bytes (two per row group and step). Returns the scale.
template <int KIND, int J>
__device__ __forceinline__ float qt_unpack(uint32_t p, uint32_t a) {
  constexpr int BS = QtKind<KIND>::BS, at = BS * J, base = at & ~15, L = ((at + BS - 1) >> 4) - (base >> 4) + 1;
  uint32_t w[4 * L + 1];
#pragma unroll
  for (int i = 0; i < L; i++) {
    const U4 v = gm_lds128(p + base + 16 * i);
    w[4 * i] = v.x;
    w[4 * i + 1] = v.y;
    w[4 * i + 2] = v.z;
    w[4 * i + 3] = v.w;
  }
  w[4 * L] = 0;
  auto word = [&](int off) {  // off: static
    const int i = (at + off - base) >> 2;
    return (at + off) & 2 ? funnel_r(w[i], w[i + 1], 16) : w[i];
  };
  const float d = half_bits_hw(word(0) & 0xFFFFu);
  uint32_t q[8];  // quants 4i .. 4i + 3, offset to positive bytes
  uint32_t minus;
  if (KIND == Q8_0) {
#pragma unroll
    for (int i = 0; i < 8; i++) q[i] = word(2 + 4 * i) ^ 0x80808080u;
    minus = 0xE480E480u;  // -1152
  } else {
    uint32_t h = 0;
    if (KIND == Q5_0) h = word(2);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t v = word((KIND == Q5_0 ? 6 : 2) + 4 * i);
      q[i] = v & 0x0F0F0F0Fu;
      q[4 + i] = (v >> 4) & 0x0F0F0F0Fu;
    }
    if (KIND == Q5_0) {
#pragma unroll
      for (int i = 0; i < 8; i++) {  // bits 4i .. 4i + 3 of h to bit 4 of the four bytes
        const uint32_t b = (h >> (4 * i)) & 0xFu;
        q[i] |= ((b * 0x00204081u) & 0x01010101u) << 4;
      }
    }
    minus = KIND == Q5_0 ? 0xE410E410u : 0xE408E408u;  // -1040, -1032
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint2 t = qt_halves(q[2 * i], minus), v = qt_halves(q[2 * i + 1], minus);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + (i >> 1) * (QT_A / 2) + (i & 1) * 128), "r"(t.x), "r"(t.y), "r"(v.x), "r"(v.y) : "memory");
  }
  return d;
}

__device__ __forceinline__ void qt_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%4, %4, %4, %4}, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(0u)
      : "memory");
}

template <int KIND, int TPW>
__global__ void __launch_bounds__(QT_THREADS, 1) qt_kernel(const __grid_constant__ QtParams P) {
  using K = QtKind<KIND>;
  using S = QtShape<TPW>;
  extern __shared__ __align__(128) uint8_t smem[];
  // [stages: rows, tokens][operands of the slots][row scales][token scales][barriers][tensor memory base][abort][exchange]
  uint8_t* const raw_ring = smem;
  uint8_t* const b_ring = raw_ring + P.n_raw * (K::RAW + S::X);
  uint8_t* const a_ring = b_ring + QT_SLOTS * S::B;
  float* const dws = reinterpret_cast<float*>(a_ring + QT_SLOTS * QT_A);
  float2* const dxs = reinterpret_cast<float2*>(dws + QT_SLOTS * KT_ROWS);  // [slot][32], each twice
  uint64_t* const raw_full = reinterpret_cast<uint64_t*>(dxs + QT_SLOTS * 32);
  uint64_t* const raw_empty = raw_full + QT_MAX_RAW;
  uint64_t* const in_full = raw_empty + QT_MAX_RAW;
  uint64_t* const in_empty = in_full + QT_SLOTS;
  uint64_t* const d_full = in_empty + QT_SLOTS;  // the block's results are there, and its scales
  uint64_t* const drain = d_full + QT_SLOTS;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  Ring R;  // for its bounded waits
  R.abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  R.err = P.err;
  float* const exchange = reinterpret_cast<float*>(raw_full + (QT_BARS + 3) / 2 * 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = P.cols >> 5, n_chunk = nb / QT_CHUNK, n_items = P.n_tiles * P.n_groups, trows = P.pair ? KT_ROWS / 2 : KT_ROWS;
  if (warp == 0 && lane < 4 && (lane < P.nseg || lane == 3)) prefetch_map(lane == 3 ? &P.xmap : &P.map[lane]);
  if (tid < QT_BARS) {  // a thread per barrier
    const int i = tid;
    mbar_init(raw_full + i, i < QT_MAX_RAW ? 1 : i < 2 * QT_MAX_RAW ? 6 : i < 2 * QT_MAX_RAW + QT_SLOTS ? 5 : i < 2 * QT_MAX_RAW + 2 * QT_SLOTS ? 17
                            : i < 2 * QT_MAX_RAW + 3 * QT_SLOTS ? 6 : 1);
    if (i == 0) *R.abort = 0;
    mbar_fence_init();
  }
  for (int i = tid; i < QT_SLOTS * S::B / 16; i += QT_THREADS) reinterpret_cast<uint4*>(b_ring)[i] = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  if (warp == 1) tc_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  // an item's matrix, first row and first token
  auto locate = [&](int item, int& sg, int& r0, int& t0) {
    const int tile = item / P.n_groups;
    t0 = (item - tile * P.n_groups) * S::T;
    sg = 0;
    if (!P.pair)
      while (sg < P.nseg - 1 && tile >= P.tiles_before[sg + 1]) sg++;
    r0 = (tile - P.tiles_before[sg]) * trows;
  };

  if (warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(QT_REGS_REST));
    if (warp == 0) {
      // ---- requests ----
      KtPos pr;
      bool ok = true;
      int left = P.give_up;
      pdl_wait();  // (the weights alone do not depend on the previous kernel; they share their barrier with the activations)
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        int sg, r0, t0;
        locate(item, sg, r0, t0);
#pragma unroll 1
        for (int c = 0; c < n_chunk; c++) {
          ok = kt_wait(R, &raw_empty[pr.slot], pr.par ^ 1u);
          if (!ok) break;
          const uint32_t dst = smem_addr(raw_ring + pr.slot * (K::RAW + S::X));
          if (elect_one()) {
            mbar_expect_tx(&raw_full[pr.slot], K::RAW + S::X);
            tma_load_2d(dst, &P.map[sg], c * (K::PITCH / 4), r0, &raw_full[pr.slot]);
            if (P.pair) tma_load_2d(dst + K::RAW / 2, &P.map[1], c * (K::PITCH / 4), r0, &raw_full[pr.slot]);
            tma_load_2d(dst + K::RAW, &P.xmap, c * (QT_CHUNK * X0_STRIDE / 4), t0, &raw_full[pr.slot]);
            if (left && --left == 0) kt_give_up(R);
          }
          __syncwarp();
          pr.advance(P.n_raw);
        }
      }
    } else if (warp == 1) {
      // ---- MMAs ----
      constexpr uint32_t idesc = (1u << 4) | ((S::N >> 3) << 17) | ((KT_ROWS >> 4) << 24);
      KtPos pi, pf;  // the block; the one that held its results' place before
      int set = 0, first = S::SETS;
      bool ok = true;
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
#pragma unroll 1
        for (int b = 0; b < nb; b++) {
          if (first > 0) {
            first--;
          } else {
            ok = kt_wait(R, &in_empty[pf.slot], pf.par);
            pf.advance(QT_SLOTS);
          }
          ok = ok && kt_wait(R, &in_full[pi.slot], pi.par);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t da = tc_desc(smem_addr(a_ring + pi.slot * QT_A)), db = tc_desc(smem_addr(b_ring + pi.slot * S::B));
#pragma unroll
            for (int s = 0; s < 2; s++) qt_mma(tmem + set * 2 * S::N + s * S::N, da + s * (QT_A / 2 >> 4), db + s * (S::STEP >> 4), idesc);
            tc_commit(&d_full[pi.slot]);
            tc_commit(&in_empty[pi.slot]);
          }
          __syncwarp();
          if (++set == S::SETS) set = 0;
          pi.advance(QT_SLOTS);
        }
      }
      // every MMA has finished before the tensor memory and the operands go
      if (elect_one()) tc_commit(drain);
      __syncwarp();
      mbar_wait(drain, 0, P.err);
    } else if (warp < 4) {
      // ---- activations: every other block ----
      KtPos pr, pi;
      bool ok = true;
      const int c = lane & 7, tl = lane >> 3;
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
#pragma unroll 1
        for (int ch = 0; ch < n_chunk && ok; ch++) {
          ok = kt_wait(R, &raw_full[pr.slot], pr.par);
          if (!ok) break;
          const uint32_t xs = smem_addr(raw_ring + pr.slot * (K::RAW + S::X) + K::RAW);
#pragma unroll 1
          for (int j = 0; j < QT_CHUNK; j++) {
            if ((j & 1) == (warp & 1)) {
              ok = kt_wait(R, &in_empty[pi.slot], pi.par ^ 1u);
              if (!ok) break;
              // (token, chain): row n of the step, its 8 bytes on the diagonal
              const uint32_t dst = smem_addr(b_ring + pi.slot * S::B) + (c >> 2) * S::STEP + ((c >> 1) & 1) * 128 + (c & 1) * 8;
              uint32_t w[S::T / 4], d = 0;
#pragma unroll
              for (int i = 0; i < S::T / 4; i++) w[i] = gm_lds32(xs + ((4 * i + tl) * QT_CHUNK + j) * X0_STRIDE + 4 * c);
              if (lane < S::T) d = gm_lds32(xs + (lane * QT_CHUNK + j) * X0_STRIDE + X0_D);
#pragma unroll
              for (int i = 0; i < S::T / 4; i++) {
                const int n = 4 * (4 * i + tl) + (c & 3);
                const uint2 h = qt_halves(w[i] ^ 0x80808080u, 0xE480E480u);
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + (n >> 3) * 256 + (n & 7) * 16), "r"(h.x), "r"(h.y) : "memory");
              }
              if (lane < S::T) dxs[pi.slot * 32 + lane] = make_float2(__uint_as_float(d), __uint_as_float(d));
              fence_async_smem();
              __syncwarp();
              if (elect_one()) {
                mbar_arrive(&in_full[pi.slot]);
                mbar_arrive(&d_full[pi.slot]);
              }
              __syncwarp();
            }
            pi.advance(QT_SLOTS);
          }
          if (elect_one()) mbar_arrive(&raw_empty[pr.slot]);
          __syncwarp();
          pr.advance(P.n_raw);
        }
      }
    } else {
      // ---- weights ----
      const int row = tid - 128;
      const uint32_t a_row = smem_addr(a_ring) + (row >> 3) * 256 + (row & 7) * 16;
      KtPos pr, pi;
      bool ok = true;
      // two blocks at a time, under one proxy fence
      auto blocks = [&](auto jc, uint32_t p) {
        constexpr int J = decltype(jc)::value;
        const int s0 = pi.slot;
        ok = ok && kt_wait(R, &in_empty[s0], pi.par ^ 1u);
        pi.advance(QT_SLOTS);
        const int s1 = pi.slot;
        ok = ok && kt_wait(R, &in_empty[s1], pi.par ^ 1u);
        pi.advance(QT_SLOTS);
        if (!ok) return;
        dws[s0 * KT_ROWS + row] = qt_unpack<KIND, J>(p, a_row + s0 * QT_A);
        dws[s1 * KT_ROWS + row] = qt_unpack<KIND, J + 1>(p, a_row + s1 * QT_A);
        fence_async_smem();
        __syncwarp();
        if (elect_one()) {
          mbar_arrive(&in_full[s0]);
          mbar_arrive(&d_full[s0]);
          mbar_arrive(&in_full[s1]);
          mbar_arrive(&d_full[s1]);
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
#pragma unroll 1
        for (int ch = 0; ch < n_chunk && ok; ch++) {
          ok = kt_wait(R, &raw_full[pr.slot], pr.par);
          if (!ok) break;
          const uint32_t p = smem_addr(raw_ring + pr.slot * (K::RAW + S::X) + row * K::PITCH);
          blocks(QtInt<0>(), p);
          blocks(QtInt<2>(), p);
          blocks(QtInt<4>(), p);
          blocks(QtInt<6>(), p);
          __syncwarp();
          if (elect_one()) mbar_arrive(&raw_empty[pr.slot]);
          __syncwarp();
          pr.advance(P.n_raw);
        }
      }
    }
  } else {
    // ---- chains ----
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(QT_REGS_CHAINS));
    const int row = tid & 127, wg = (warp - 8) >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    KtPos pi;
    int set = 0;
    bool ok = true;
    pdl_wait();
#pragma unroll 1
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
      F2 acc[TPW][4];  // chains 2k, 2k + 1 of a token
#pragma unroll
      for (int t = 0; t < TPW; t++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[t][k] = f2_pack(0.0f, 0.0f);
#pragma unroll 1
      for (int b = 0; b < nb; b++) {
        ok = kt_wait_inline(R, &d_full[pi.slot], pi.par);
        if (!ok) break;
        tc_fence_after();
        const float dw = dws[pi.slot * KT_ROWS + row];
        const F2 dd = f2_pack(dw, dw);
        const uint32_t dx = smem_addr(dxs + pi.slot * 32 + wg * TPW), at = tmem + lanes + set * 2 * S::N + wg * (4 * TPW);
#pragma unroll
        for (int t = 0; t < TPW; t += 2) {
          uint32_t p[2][8];
          kt_ld8(at + 4 * t, p[0]);
          kt_ld8(at + S::N + 4 * t, p[1]);
          const U4 x = gm_lds128(dx + 8 * t);
          const F2 sc[2] = {f2_mul(dd, f2_pack(__uint_as_float(x.x), __uint_as_float(x.y))), f2_mul(dd, f2_pack(__uint_as_float(x.z), __uint_as_float(x.w)))};
          tc_wait_ld();
#pragma unroll
          for (int st = 0; st < 2; st++)
#pragma unroll
            for (int e = 0; e < 2; e++)
#pragma unroll
              for (int k = 0; k < 2; k++)
                acc[t + e][2 * st + k] = f2_fma(sc[e], f2_pack(__uint_as_float(p[st][4 * e + 2 * k]), __uint_as_float(p[st][4 * e + 2 * k + 1])), acc[t + e][2 * st + k]);
        }
        tc_fence_before();
        __syncwarp();
        if (elect_one()) mbar_arrive(&in_empty[pi.slot]);
        __syncwarp();
        if (++set == S::SETS) set = 0;
        pi.advance(QT_SLOTS);
      }
      if (!ok) {  // (not carried to the meeting below: sums that outlive a wait's failure made a product a third slower)
        if (P.pair) kt_meet(1 + wg, false);
        break;
      }
      // ((a0+a4)+(a2+a6)) + ((a1+a5)+(a3+a7)), then what is done with it
      float out[TPW];
#pragma unroll
      for (int t = 0; t < TPW; t++) {
        float a[8];
#pragma unroll
        for (int k = 0; k < 4; k++) f2_unpack(acc[t][k], a[2 * k], a[2 * k + 1]);
        out[t] = fadd(fadd(fadd(a[0], a[4]), fadd(a[2], a[6])), fadd(fadd(a[1], a[5]), fadd(a[3], a[7])));
      }
      int sg, r0, t0;
      locate(item, sg, r0, t0);
      t0 += wg * TPW;
      if (P.pair) {
        // rows 0..63 are of the gate, 64.. of the up matrix: after an exchange of half of the tokens both
        // finish half of the results
        constexpr int H = TPW / 2;
        const bool up = row >= 64;
        float* const mine = exchange + (wg * 128 + row) * H;
#pragma unroll
        for (int i = 0; i < H; i++) mine[i] = up ? out[2 * i] : out[2 * i + 1];
        ok = kt_meet(1 + wg, true);
        if (!ok) break;
        const float* const other = exchange + (wg * 128 + (row ^ 64)) * H;
        const int gr = r0 + (row & 63);
#pragma unroll
        for (int i = 0; i < H; i++) {
          const float o = other[i], gate = up ? o : out[2 * i], upv = up ? out[2 * i + 1] : o;
          const int tok = t0 + 2 * i + up;
          const size_t at = (size_t)tok * P.seg[0].rows + gr;
          if (tok < P.m && gr < P.seg[0].rows) {
            P.seg[0].out[at] = P.epilogue == EPI_SILU_MUL ? silu_mul_exact(gate, upv) : gate;
            P.seg[1].out[at] = upv;
          }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");  // the next item writes the exchange again
      } else {
        const GemvSeg& G = P.seg[sg];
        const int gr = r0 + row;
#pragma unroll
        for (int t = 0; t < TPW; t++) {
          float* const o = G.out + (size_t)(t0 + t) * G.rows + gr;
          if (t0 + t < P.m && gr < G.rows) *o = P.epilogue == EPI_ACCUM ? fadd(*o, out[t]) : out[t];
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*R.abort)  // whichever warp gave up, the copies in flight land before the CTA's shared memory goes
      for (int i = 0; i < P.n_raw; i++) mbar_drain(&raw_full[i]);
    tc_dealloc(tmem, 512);
  }
}

}  // namespace aot

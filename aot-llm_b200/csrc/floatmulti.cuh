// Products of F16 / BF16 / F32 matrices with several f32 activation rows (simd_avx2.rs:433-493: eight
// AVX2 lane accumulators per row, acc_k = fma(w[8j+k], x[8j+k], acc_k) for j in order, then the
// horizontal sum of simd_avx2.rs:29-34), bit-identical to the reference.
//
// What bounds it: one f32 fused multiply-add per weight and activation row, in chains that must not
// be split. Columns 2p, 2p+1 of a step are two chains whose operands lie side by side, so every
// operation is a packed one (two results in 2 cycles where two scalar ones take 3.3 and twice the
// issue slots). A lane owns chain pair p of 4 rows and T activation rows: 4 + T loads from shared
// memory and the conversion of 4 weight pairs per 4 T packed operations, against one load per
// operation when a lane owned one chain. A warp covers 32 rows, its eight row groups lie 16 bytes
// apart modulo the banks, and an activation pair is read by eight lanes at once.
// bf16 4096x4096, 37 rows: 119 us with a chain per lane (float_stream_kernel), 59 us now; f16 32768x4096, 2
// rows: 107 and 51. Its weak spot is a batch that just fills 16 rows on a matrix whose tiles fall
// unevenly on the SMs: launch_float_multi sends that to float_stream_kernel, by estimates of both.
#pragma once
#include "mmautils.cuh"
#include "rowdot.cuh"

namespace aot {

constexpr int FM_COLS = 64;         // columns of a chunk
constexpr int FM_STAGES = 4;
constexpr int FM_MAX_WARPS = 8;

struct FloatMultiParams {
  GemvSeg seg[3];
  int nseg, cols, m, epilogue;
  int wt, n_tcta;  // warps of a CTA (T activation rows each), CTAs per row tile
  int tiles_before[4];
  const float* x;
};

template <int KIND, int R, int T>
struct FmShape {
  static constexpr int ROWS = 8 * R;  // weight rows of a CTA
  static constexpr int ES = KIND == F32 ? 4 : 2;
  static constexpr int WROW = FM_COLS * ES + 8 * ES;  // 16 (32) bytes modulo 128: the 8 x 4 words (pairs of words) of a load fall on different banks
  static constexpr int WBYTES = ROWS * WROW;
  static constexpr int XROW = FM_COLS * 4;
  __host__ __device__ static constexpr int stage_bytes(int wt) { return WBYTES + wt * T * XROW; }
};

template <int KIND, int R, int T>
__global__ void __launch_bounds__(FM_MAX_WARPS * 32, R == 2 ? 3 : 2) float_multi_kernel(const __grid_constant__ FloatMultiParams P) {
  using S = FmShape<KIND, R, T>;
  constexpr int ES = S::ES, WROW = S::WROW, XROW = S::XROW;
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, p = lane & 3, rg = lane >> 2;
  const int tile = blockIdx.x / P.n_tcta, tc0 = (blockIdx.x - tile * P.n_tcta) * P.wt * T, tok0 = tc0 + warp * T;
  int sg = 0;
  while (sg < P.nseg - 1 && tile >= P.tiles_before[sg + 1]) sg++;
  const int row0 = (tile - P.tiles_before[sg]) * S::ROWS, n_rows = P.seg[sg].rows, n_chunks = (P.cols + FM_COLS - 1) / FM_COLS;
  const size_t row_bytes = (size_t)P.cols * ES;
  const uint32_t sm = smem_addr(smem), stage_bytes = (uint32_t)S::stage_bytes(P.wt);
  pdl_wait();
  // 16-byte pieces: piece pw of weight row rw, and of the rows below it; piece px of activation row rx
  constexpr int WP = FM_COLS * ES / 16, XP = XROW / 16;
  const int nth = P.wt * 32, pw = threadIdx.x % WP, rw = threadIdx.x / WP, px = threadIdx.x % XP, rx = threadIdx.x / XP;
  const uint8_t* const wsrc = P.seg[sg].w + pw * 16;
  const float* const xsrc = P.x + px * 4;
  auto issue = [&](int c) {
    if (c < n_chunks) {
      const uint32_t st = sm + (uint32_t)(c & (FM_STAGES - 1)) * stage_bytes;
      const int left = P.cols - c * FM_COLS;
      if (pw * (16 / ES) < left)
        for (int r = rw; r < S::ROWS; r += nth / WP)
          cp_async16(st + (uint32_t)(r * WROW + pw * 16), wsrc + (size_t)min(row0 + r, n_rows - 1) * row_bytes + (size_t)c * (FM_COLS * ES));
      if (px * 4 < left)
        for (int r = rx; r < P.wt * T; r += nth / XP)
          if (tc0 + r < P.m) cp_async16(st + (uint32_t)(S::WBYTES + r * XROW + px * 16), xsrc + (size_t)(tc0 + r) * P.cols + (size_t)c * FM_COLS);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int c = 0; c < FM_STAGES - 1; c++) issue(c);
  F2 acc[R][T];
#pragma unroll
  for (int r = 0; r < R; r++)
#pragma unroll
    for (int t = 0; t < T; t++) acc[r][t] = 0ull;
  const uint32_t woff = (uint32_t)(rg * WROW + p * 2 * ES), xoff = (uint32_t)(S::WBYTES + warp * T * XROW + p * 8);
#pragma unroll 1
  for (int c = 0; c < n_chunks; c++) {
    cp_async_wait<FM_STAGES - 2>();
    __syncthreads();
    issue(c + FM_STAGES - 1);
    const uint32_t st = sm + (uint32_t)(c & (FM_STAGES - 1)) * stage_bytes, wa = st + woff, xa = st + xoff;
    const int n_steps = min(FM_COLS, P.cols - c * FM_COLS) >> 3;
    // a step's operands are requested before the operations of the step before it
    uint32_t w[2][R][ES / 2];
    F2 x[2][T];
    auto load = [&](int j) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint32_t a = wa + (uint32_t)(r * 8 * WROW + j * 8 * ES);
        if (KIND == F32) gm_lds64(a, w[j & 1][r][0], w[j & 1][r][ES / 2 - 1]);
        else w[j & 1][r][0] = gm_lds32(a);
      }
#pragma unroll
      for (int t = 0; t < T; t++) asm volatile("ld.shared.u64 %0, [%1];" : "=l"(x[j & 1][t]) : "r"(xa + (uint32_t)(t * XROW + j * 32)));
    };
    auto mul = [&](int j) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint32_t v = w[j & 1][r][0];
        F2 wf;  // both conversions are exact (every f16 / bf16 value is an f32 value)
        if (KIND == F32) {
          wf = f2_pack(__uint_as_float(v), __uint_as_float(w[j & 1][r][ES / 2 - 1]));
        } else if (KIND == F16) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
          wf = f2_pack(f.x, f.y);
        } else {
          wf = f2_pack(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
        }
#pragma unroll
        for (int t = 0; t < T; t++) acc[r][t] = f2_fma(wf, x[j & 1][t], acc[r][t]);
      }
    };
    if (n_steps == FM_COLS / 8) {
      load(0);
#pragma unroll
      for (int j = 0; j < FM_COLS / 8; j++) {
        if (j + 1 < FM_COLS / 8) load(j + 1);
        mul(j);
      }
    } else {
#pragma unroll
      for (int j = 0; j < FM_COLS / 8 - 1; j++) {
        if (j < n_steps) {
          load(j);
          mul(j);
        }
      }
    }
  }
  pdl_launch_dependents();  // not before: CTAs of the next launch would share SMs with this one's last wave
  cp_async_wait<0>();
  // ((a0+a4)+(a2+a6)) + ((a1+a5)+(a3+a7)): pair p holds a_2p, a_2p+1
#pragma unroll
  for (int t = 0; t < T; t++) {
#pragma unroll
    for (int r = 0; r < R; r++) {
      F2 a = acc[r][t];
      a = f2_add(a, __shfl_xor_sync(0xffffffffu, a, 2));
      a = f2_add(a, __shfl_xor_sync(0xffffffffu, a, 1));
      float v0, v1;
      f2_unpack(a, v0, v1);
      const int row = row0 + r * 8 + rg, tok = tok0 + t;
      if (p == (r & 3) && row < n_rows && tok < P.m) {
        float* const o = P.seg[sg].out + (size_t)tok * n_rows + row;
        const float v = fadd(v0, v1);
        *o = P.epilogue == EPI_ACCUM ? fadd(__ldcg(o), v) : v;
      }
    }
  }
}

}  // namespace aot

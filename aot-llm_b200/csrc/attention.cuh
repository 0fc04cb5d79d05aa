// Attention over cached rows (crates/aot-kernels/src/ops.rs:185-218, 517-556), bit-identical to the
// reference: each q.k dot is one sequential chain, the softmax denominator is added in position
// order, the value mix runs over positions in order; products and sums are rounded separately.
//
// What bounds it: two rounded operations per (query, position, dimension) in each of the two
// contractions, with no reduction that could be reordered. So the work is arranged for the
// fp32 pipe, eight queries per CTA (consecutive (row, head) pairs of one KV head):
//  * packed operations take two queries at a time (f32x2: two results per 2 pipe cycles where two
//    scalar operations take 3.3); a product is an fma with -0 as addend, which is exact and which
//    the assembler cannot contract with the following sum;
//  * scores: a lane owns a position and all eight queries, so a cached K element is read from
//    shared memory once for eight dots; K rows travel through a private ring per warp, 8
//    dimensions of 32 positions at a time and three pieces ahead;
//  * scores and weights lie [position][query], so that the value mix (a lane owns a dimension and
//    four queries) reads a position's four weights with one broadcast load;
//  * the denominators of the eight queries are eight lanes' add chains in one warp.
// Two CTAs share an SM, so one's chains and barriers run under the other's arithmetic.
// 32 heads of 64 on 4 KV heads: 64 rows at position 448 took 53 us with one (row, head) pair per
// CTA and take 40; 7 rows at position 300, where no phase fills the chip, 32.7 and 22.9,
// and four pairs per CTA (ATTN_NQ / 2, taken where eight leave SMs idle) save 3.7 of those: a prompt
// of 7 at 300 takes 1577 us instead of 1661.
#pragma once
#include "blockmath.cuh"
#include "device_utils.cuh"
#include "expf_exact.cuh"
#include "mmautils.cuh"
#include "ops.cuh"

namespace aot {

struct AttnParams {
  float* out;            // m x q_dim
  const float* q;        // m x q_dim
  const float* k_cache;  // layer base: ctx x kv_dim
  const float* v_cache;
  float* scratch;        // [CTA][ctx][8] scores, when they do not fit shared memory
  const int* pos_ptr;
  int pos0;
  int n_head, n_kv_head, head_dim, ctx, window;
  int m;                 // query rows
  int v_chunk;           // cached V rows per staging buffer
  // quantized outputs as well, for the product that reads them next (null: none): rows of 256 values in the
  // orders of xf_store (xf_nt groups of 8 rows; attn_quantizes says when a CTA holds whole blocks), or Q8_0
  // images
  uint8_t *xf, *xt, *q80;
  int xf_nt;
  float scale, neg_zero; // neg_zero: -0.0f, from the host so that the compiler does not know it
};

constexpr int ATTN_NQ = 8;                       // queries per CTA, or half of them where that leaves SMs idle
constexpr int ATTN_WARPS = 8, ATTN_THREADS = ATTN_WARPS * 32;
static_assert(ATTN_WARPS >= ATTN_NQ, "a warp loads a query");
constexpr int ATTN_KD = 8;                       // dimensions of a staged K piece
constexpr int ATTN_KRING = 4;                    // pieces in a warp's ring
constexpr int ATTN_KPITCH = ATTN_KD + 4;         // floats per position: eight lanes' 16-byte reads fall on different banks
constexpr int ATTN_KBUF = 32 * ATTN_KPITCH;      // floats of one piece
constexpr int ATTN_STAGE = ATTN_WARPS * ATTN_KRING * ATTN_KBUF;  // floats of the staging area (K pieces of all warps, then V chunks)
// floats besides the scores
__host__ __device__ inline int attn_fixed(int nq, int head_dim) { return ATTN_STAGE + nq * head_dim + ATTN_WARPS * nq + nq; }

// A CTA's queries are whole blocks of 256 outputs: the heads of a block lie in one KV head's group.
inline bool attn_quantizes(int nq, int head_dim, int gqa) {
  return 256 % head_dim == 0 && nq % (256 / head_dim) == 0 && gqa % (256 / head_dim) == 0;
}

// SM: the scores are in shared memory (a pointer that could be either costs generic loads).
template <bool SM, int NQ>
__global__ void __launch_bounds__(ATTN_THREADS, 2) attention_kernel(const AttnParams P) {
  static_assert(NQ == 4 || NQ == 8, "");
  constexpr int NH = NQ / 4;  // groups of four queries
  extern __shared__ __align__(16) float sm_f[];
  __shared__ uint64_t exp_tab[32];
  // [staging][queries: dim x 4 pairs][maxima per warp][1 / denominator][scores: position x 8]
  float* const stage = sm_f;
  float* const qp = stage + ATTN_STAGE;
  float* const red = qp + NQ * P.head_dim;
  float* const inv = red + ATTN_WARPS * NQ;
  pdl_launch_dependents();
  exp_table_load(exp_tab);
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hd = P.head_dim, kv_dim = P.n_kv_head * hd, q_dim = P.n_head * hd, gqa = P.n_head / P.n_kv_head;
  const int kvh = blockIdx.x, n_query = P.m * gqa, q0 = blockIdx.y * NQ, nq = min(NQ, n_query - q0);
  float* const sc = SM ? sm_f + attn_fixed(NQ, P.head_dim) : P.scratch + (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * P.ctx * NQ;
  const int base = P.pos_ptr ? *P.pos_ptr : P.pos0;
  const int row_a = q0 / gqa, row_b = (q0 + nq - 1) / gqa;
  // positions [T0, N) are the union of the queries' ranges, [T1, N1) lie in every one of them
  auto first_of = [&](int row) { return P.window > 0 && base + row + 1 > P.window ? base + row + 1 - P.window : 0; };
  const int T0 = first_of(row_a), T1 = first_of(row_b), N = base + row_b + 1, N1 = base + row_a + 1, len = N - T0;
  auto in_range = [&](int q, int t) {  // query q of the CTA attends to position t
    const int row = (q0 + q) / gqa;
    return q < nq && t < base + row + 1 && t >= first_of(row);
  };
  // ---- scores: dot(q, k_t) * scale (ops.rs:160-166) ----
  const F2 nz = f2_pack(P.neg_zero, P.neg_zero), scale2 = f2_pack(P.scale, P.scale);
  float* const kb = stage + warp * ATTN_KRING * ATTN_KBUF;
  const int n_piece = (hd + ATTN_KD - 1) / ATTN_KD, n_block = (len + 31) / 32;
  // the next piece to request: one commit group each
  int s_blk = warp, s_piece = 0, s_buf = 0;
  auto stage_k = [&]() {
    const int d = s_piece * ATTN_KD + (lane & 1) * 4, r = lane >> 1;
    if (s_blk < n_block && d < hd) {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int t = min(T0 + s_blk * 32 + r + 16 * i, N - 1);
        cp_async16(smem_addr(kb + s_buf * ATTN_KBUF + (r + 16 * i) * ATTN_KPITCH + (lane & 1) * 4), P.k_cache + (size_t)t * kv_dim + kvh * hd + d);
      }
    }
    cp_async_commit();
    s_buf = (s_buf + 1) & (ATTN_KRING - 1);
    if (++s_piece == n_piece) {
      s_piece = 0;
      s_blk += ATTN_WARPS;
    }
  };
#pragma unroll
  for (int i = 0; i < ATTN_KRING - 1; i++) stage_k();
  // the queries, two by two per dimension (missing ones repeat the last)
  if (warp < NQ) {
    const int qi = q0 + min(warp, nq - 1), row = qi / gqa;  // a warp per query
    const float* src = P.q + (size_t)row * q_dim + (kvh * gqa + qi - row * gqa) * hd;
    for (int d = lane; d < hd; d += 32) qp[d * NQ + warp] = src[d];
  }
  __syncthreads();
  float mx[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) mx[q] = -INFINITY;
  int buf = 0;
  for (int blk = warp; blk < n_block; blk += ATTN_WARPS) {
    F2 s[NQ / 2];
#pragma unroll
    for (int p = 0; p < NQ / 2; p++) s[p] = 0ull;
    for (int piece = 0; piece < n_piece; piece++) {
      stage_k();
      cp_async_wait<ATTN_KRING - 1>();
      __syncwarp();
      const float* kt = kb + buf * ATTN_KBUF + lane * ATTN_KPITCH;
      const float4* q4 = reinterpret_cast<const float4*>(qp + piece * ATTN_KD * NQ);
      const int n4 = min(ATTN_KD, hd - piece * ATTN_KD) >> 2;
#pragma unroll 2
      for (int j = 0; j < n4; j++) {
        const float4 k4 = *reinterpret_cast<const float4*>(kt + 4 * j);
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const F2 k2 = f2_pack(kk[e], kk[e]);
#pragma unroll
          for (int g = 0; g < NH; g++) {
            const float4 a = q4[NH * (4 * j + e) + g];
            s[2 * g] = f2_add(s[2 * g], f2_fma(f2_pack(a.x, a.y), k2, nz));
            s[2 * g + 1] = f2_add(s[2 * g + 1], f2_fma(f2_pack(a.z, a.w), k2, nz));
          }
        }
      }
      __syncwarp();  // every lane has read the buffer that is filled next
      buf = (buf + 1) & (ATTN_KRING - 1);
    }
    const int t = blk * 32 + lane;
    if (t < len) {
      float v[NQ];
#pragma unroll
      for (int p = 0; p < NQ / 2; p++) f2_unpack(f2_mul(s[p], scale2), v[2 * p], v[2 * p + 1]);
      const bool all = T0 + t >= T1 && T0 + t < N1;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if (!all && !in_range(q, T0 + t)) v[q] = -INFINITY;
        mx[q] = fmaxf(mx[q], v[q]);
      }
#pragma unroll
      for (int g = 0; g < NH; g++) *reinterpret_cast<float4*>(sc + (size_t)t * NQ + 4 * g) = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int q = 0; q < NQ; q++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], o));
    if (lane == 0) red[warp * NQ + q] = mx[q];
  }
  __syncthreads();
  // V rows of positions [c0, c0 + v_chunk) of the union, into one of two buffers
  const int vch = P.v_chunk, hd4 = hd >> 2;
  const int rpw = hd4 < 32 ? 32 / hd4 : 1, vr = hd4 < 32 ? lane / hd4 : 0, vc = hd4 < 32 ? lane - vr * hd4 : lane;  // rows a warp copies at a time
  auto stage_v = [&](int c0, int b) {
    const int cn = min(vch, len - c0);
    if (vr < rpw) {
      const float* src = P.v_cache + (size_t)(T0 + c0) * kv_dim + kvh * hd;
      for (int t = warp * rpw + vr; t < cn; t += ATTN_WARPS * rpw)
        for (int c = vc; c < hd4; c += 32) cp_async16(smem_addr(stage + (b * vch + t) * hd + 4 * c), src + (size_t)t * kv_dim + 4 * c);
    }
    cp_async_commit();
  };
  stage_v(0, 0);

  // ---- softmax (ops.rs:98-112): exp, the denominators in position order, the scaled weights ----
  const int half = NH == 2 ? tid & 1 : 0;  // this thread's four queries
  {
    float m4[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      m4[q] = red[4 * half + q];
#pragma unroll
      for (int w = 1; w < ATTN_WARPS; w++) m4[q] = fmaxf(m4[q], red[w * NQ + 4 * half + q]);
    }
    for (int i = tid; i < NH * len; i += ATTN_THREADS) {
      float4 v = reinterpret_cast<float4*>(sc)[i];
      v.x = expf_exact(fsub(v.x, m4[0]), exp_tab);
      v.y = expf_exact(fsub(v.y, m4[1]), exp_tab);
      v.z = expf_exact(fsub(v.z, m4[2]), exp_tab);
      v.w = expf_exact(fsub(v.w, m4[3]), exp_tab);
      reinterpret_cast<float4*>(sc)[i] = v;
    }
  }
  __syncthreads();
  if (tid < NQ) {
    // positions outside the query's range are +0; eight terms load under the chain of the eight before
    float s = 0.0f, v[8], w[8];
    const float* p = sc + tid;
    auto load = [&](float (&x)[8], int t) {
      if (t + 8 <= len) {
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = p[(size_t)(t + j) * NQ];
      } else {
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = t + j < len ? p[(size_t)(t + j) * NQ] : 0.0f;
      }
    };
    load(v, 0);
#pragma unroll 1
    for (int t = 0; t < len; t += 16) {
      load(w, t + 8);
#pragma unroll
      for (int j = 0; j < 8; j++) s = fadd(s, v[j]);
      load(v, t + 16);
#pragma unroll
      for (int j = 0; j < 8; j++) s = fadd(s, w[j]);
    }
    inv[tid] = fdiv(1.0f, s);
  }
  __syncthreads();
  {
    const float4 f = reinterpret_cast<const float4*>(inv)[half];
    for (int i = tid; i < NH * len; i += ATTN_THREADS) {
      float4 v = reinterpret_cast<float4*>(sc)[i];
      v.x = fmul(v.x, f.x);
      v.y = fmul(v.y, f.y);
      v.z = fmul(v.z, f.z);
      v.w = fmul(v.w, f.w);
      reinterpret_cast<float4*>(sc)[i] = v;
    }
  }

  // ---- out[d] = sum_t a_t * v_t[d], t in order (ops.rs:208-214) ----
  // task = (32 dimensions, half of the queries); a warp takes tasks warp and warp + 8 (tasks of two
  // queries out of eight keep more warps busy, and cost a full chip 1 % of a prompt)
  constexpr int NT = 2, NG = 2, QT = NQ / NG, PAIRS = QT / 2;
  const int n_task = NG * ((hd + 31) >> 5);
  F2 o[NT][PAIRS];
#pragma unroll
  for (int k = 0; k < NT; k++)
#pragma unroll
    for (int i = 0; i < PAIRS; i++) o[k][i] = 0ull;
  for (int c0 = 0, ci = 0; c0 < len; c0 += vch, ci++) {
    const int cn = min(vch, len - c0);
    if (c0 + vch < len) {
      stage_v(c0 + vch, (ci + 1) & 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NT; k++) {
      const int task = warp + k * ATTN_WARPS, d = (task >> 1) * 32 + lane, g = task & 1;
      if (task < n_task) {
        const float* v = stage + (ci & 1) * vch * hd + min(d, hd - 1);
        const float* a = sc + (size_t)c0 * NQ + g * QT;
        const float4* a4 = reinterpret_cast<const float4*>(sc + (size_t)c0 * NQ) + g;
        const float2* a2 = reinterpret_cast<const float2*>(sc + (size_t)c0 * NQ) + g;
        // positions of every query's range (outside it a query adds nothing: a value there may
        // not even be finite)
        const int ta = max(0, min(cn, T1 - T0 - c0)), tb = max(ta, min(cn, N1 - T0 - c0));
        auto edge = [&](int from, int to) {
          for (int t = from; t < to; t++) {
            const float x = v[t * hd];
#pragma unroll
            for (int i = 0; i < PAIRS; i++) {
              float r[2];
              f2_unpack(o[k][i], r[0], r[1]);
#pragma unroll
              for (int q = 0; q < 2; q++)
                if (in_range(g * QT + 2 * i + q, T0 + c0 + t)) r[q] = fadd(r[q], fmul(a[t * NQ + 2 * i + q], x));
              o[k][i] = f2_pack(r[0], r[1]);
            }
          }
        };
        edge(0, ta);
        F2 p[PAIRS];
#pragma unroll
        for (int i = 0; i < PAIRS; i++) p[i] = o[k][i];
#pragma unroll 8
        for (int t = ta; t < tb; t++) {
          if (QT == 4) {
            const float4 w = a4[(NQ / 4) * t];
            const F2 x = f2_pack(v[t * hd], v[t * hd]);
            p[0] = f2_add(p[0], f2_fma(f2_pack(w.x, w.y), x, nz));
            p[PAIRS - 1] = f2_add(p[PAIRS - 1], f2_fma(f2_pack(w.z, w.w), x, nz));
          } else {
            const float2 w = a2[(NQ / 2) * t];
            p[0] = f2_add(p[0], f2_fma(f2_pack(w.x, w.y), f2_pack(v[t * hd], v[t * hd]), nz));
          }
        }
#pragma unroll
        for (int i = 0; i < PAIRS; i++) o[k][i] = p[i];
        edge(tb, cn);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < NT; k++) {
    const int task = warp + k * ATTN_WARPS, d = (task >> 1) * 32 + lane, g = task & 1;
    if (task < n_task && d < hd) {
#pragma unroll
      for (int i = 0; i < PAIRS; i++) {
        float r[2];
        f2_unpack(o[k][i], r[0], r[1]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int qi = q0 + g * QT + 2 * i + q, row = qi / gqa;
          if (qi < n_query) P.out[(size_t)row * q_dim + (kvh * gqa + qi - row * gqa) * hd + d] = r[q];
          stage[(g * QT + 2 * i + q) * hd + d] = r[q];
        }
      }
    }
  }
  // The quantized form here instead of in a launch of its own: 1.2 to 2.5 us a layer of a prompt (64 rows at 0,
  // TinyLlama shape: 90.5 to 88.6 us a layer; 7 at 300: 70.3 to 69.1; Qwen3-8B shape 166 to 163.5).
  if (P.xf || P.q80) {
    __syncthreads();
    const int per = P.xf ? 256 : 32, n_blk = nq * hd / per;
    for (int i = warp; i < n_blk; i += ATTN_WARPS) {
      const int qi = q0 + i * per / hd, row = qi / gqa, col = (kvh * gqa + qi - row * gqa) * hd + i * per % hd;
      if (P.xf) warp_quantize_xf(stage + i * 256, P.xf, P.xt, row, col >> 8, P.xf_nt, true);
      else warp_quantize_q80(stage + i * 32, P.q80 + ((size_t)row * (q_dim >> 5) + (col >> 5)) * XIMG_0, 1);
    }
  }
}

}  // namespace aot

// Q4_K / Q5_K / Q6_K matrices against 2..64 activation rows on the tensor cores: tcgen05.mma
// kind::i8, weights as the operand in tensor memory (matmul_rows of
// crates/aot-kernels/src/matvec.rs:479-522).
//
// A weight times the scale of its sub-block is an integer of at most 14 bits. It is held as two
// unsigned bytes (digits), so that one int32 accumulator per digit takes a whole super-block:
//   Q4_K, Q5_K: sc = 8 * s1 + s0; digits q * s0 and q * s1 (at most 31 * 7), sumi = 8 * acc1 + acc0
//   Q6_K:       v = sc * (q - 32) + 4096, 32..8192 (sc -128..127, q 0..63); its low and high byte (at most 32),
//               sumi = 256 * acc1 + acc0 - 4096 * (sum of the block's activations)
// The mins' sum_j m_j * (bsums[2j] + bsums[2j+1]) is one kind::f16 MMA per block (mins <= 63 and
// 16-element sums <= 2048 are exact in f16, their products and sums in f32). Accumulators are read
// once per super-block; the f32 terms are added in block order, the order of the single-row
// products, so batched == single bit for bit (crates/aot-kernels/tests/dots.rs:205-266).
//
// A tile is 128 weight rows x all tokens. Few matrices have 148 such tiles, so a cluster of C CTAs
// shares one: CTA r takes the super-blocks r, r + C, ... and sends the terms of every quad of four
// tokens to the CTA that owns the quad (quad % C), through distributed shared memory. Warp roles:
//   warp 0         requests a super-block's activations (one bulk copy)
//   warp 1         tensor memory, MMAs
//   warps 2, 3     request its rows: tensor copies, or 16 bytes at a time where those cannot take them
//   warps 4..11    unpack: thread = half of a weight row; raw block -> digits -> tensor memory
//   warps 12..19   terms: thread = weight row and every other 16 tokens; accumulators -> f32 terms -> the owners
//   warps 20..23   sums: thread = weight row; adds the stage's C terms of its quads, in order; outputs
//
// What bounds it: a stage (a super-block per CTA) of 64 tokens takes 1.65 us of Q4_K, 1.69 of Q5_K, 1.96 of Q6_K, and all
// the rest of a product 5 (fits to 1755 timings, within 9 %). Its MMAs are 0.28 us; the rest is unpacking, terms and sums (Q6_K 8500 warp
// instructions per stage and CTA at 2.3 per cycle) that wait for one another's barriers and for distributed shared
// memory (32 KB of terms per stage). The start of a product, from its first instruction to the first terms, is 4.5 us.
// Measured with the conversion of the activations (us; kmma.cuh, which unpacks into registers and has
// its MMAs wait on the same warps, in brackets): 4096 x 14336 x 64 Q4_K 31 (46), Q6_K 33 (61); 24576 x
// 4096 x 64 Q4_K 44 (74), Q6_K 48 (100); 2048 x 5632 x 64 Q6_K 17 (20). Tried: weights as f16 operands
// with one digit for Q4_K, which saves the conversion of the sums and doubles the activations' bytes,
// 27 against 27; one warpgroup each for unpacking and terms, 35 to 45; a release at cluster scope per
// stage instead of stores that count themselves at the owner's barrier, 1000 to 2000 cycles each.
//
// Activations ("XT"), [super-block][token group of 8], XT_BLOCK = 2368 bytes: the B operands as core
// matrices (K-major, no swizzle), [16 elements][token][16 bytes]; f16 sums of the sixteen 16-element
// groups, [8 groups][token][16 bytes]; 8 x f32 block scales; 8 x s32 -4096 * sums of 256.
#pragma once
#include <cuda_fp16.h>

#include "gemm_tc.cuh"
#include "mega.cuh"
#include "mmautils.cuh"
#include "ops.cuh"
#include "q80stream.cuh"
#include "rowdot.cuh"

namespace aot {

constexpr int KT_ROWS = 128;
constexpr int KT_MAX_M = 64;
constexpr int KT_THREADS = 768;
constexpr int KT_MAX_SLOTS = 4;
constexpr int KT_QUADS = KT_MAX_M / 4;
constexpr int KT_TERMS = KT_QUADS * KT_ROWS * 16;  // bytes of one stage's terms at their owner
constexpr int KT_SIDE_SLOTS = 4;
// tensor memory: two sets of accumulators of 32 tokens (low, high, mins), two of operands
constexpr int KT_D_COLS = 96, KT_A_COLS = 136, KT_A_BASE = 2 * KT_D_COLS;
static_assert(KT_A_BASE + 2 * KT_A_COLS <= 512, "tensor memory");

template <int KIND>
struct KtKind {
  static constexpr int BS = KIND == Q4_K ? 144 : KIND == Q5_K ? 176 : 210;
  // a row's block in shared memory: odd in 16-byte units, so that threads reading a row each meet
  // no bank conflicts (Q6_K: 16-byte aligned superset of the 2-byte aligned block)
  static constexpr int PITCH = KIND == Q6_K ? 240 : BS;
  static constexpr int PIECES = KIND == Q6_K ? 14 : BS / 16;
  static constexpr int RAW = KT_ROWS * PITCH;
};
template <int C>
constexpr int KT_XCH = KT_QUADS / C * 2 + 4;  // floats a thread exchanges with its partner of a pair, padded off the same banks
constexpr int KT_BARS = 4 * KT_MAX_SLOTS + 12 + KT_SIDE_SLOTS + 1;

struct KtParams {
  alignas(64) CUtensorMap map[3];  // tma: each matrix as u32 [rows][row_bytes / 4], box [128, pair: 64][PITCH / 4]
  GemvSeg seg[3];
  int nseg, cols, m, nt, pair, epilogue;  // nt: token groups of 8 of this launch (at most 8)
  int xf_nt;                              // token groups of the activation buffer
  const uint8_t* xf;                      // its first group of this launch
  int tiles_before[4];                    // first tile of each matrix (pair: one list, 64 rows of both per tile)
  int n_tiles;
  int tma, n_raw, n_b;                    // slots of the raw and the activation ring
  int give_up;                            // requests of activations after which the CTA's waits end (0: never)
  int* err;
};

// One lane of a converged warp. Asynchronous instructions take their operands from uniform
// registers: under this predicate they issue in a few cycles, under `lane == 0` in about 45.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ uint32_t half2_of_byte(uint32_t w, int i) {  // byte i of w twice, as f16: 1024 + b, minus 1024
  uint32_t h = prmt(w, 0x64u, i | 4 << 4 | i << 8 | 4 << 12);
  asm("add.rn.f16x2 %0, %0, %1;" : "+r"(h) : "r"(0xE400E400u));
  return h;
}
// ---- cluster ------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// "I have read it": the loads of this warp come before the arrive that lets their slot be overwritten, so it is a
// release (by default, for the CTA), which costs nothing here: 24576 x 4096 x 64 Q4_K 44.3 us and 44.3 with a
// relaxed arrive, Q6_K 48.5 and 48.5. A release at cluster scope, which the peers' acquire would ask for, also waits
// for what the warp has stored, which nobody reads, and is 50.7 and 55.6; what has to come first here is loads alone,
// and a load that has returned its value has been performed for every thread.
__device__ __forceinline__ void cluster_arrive(uint32_t mapped_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(mapped_bar) : "memory");
}
__device__ __forceinline__ void cluster_sync_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) { asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory"); }
// 16 bytes into a CTA of the cluster; its barrier counts them when they are there.
__device__ __forceinline__ void cluster_st128(uint32_t mapped, uint32_t mapped_bar, const float (&v)[4]) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(mapped), "f"(v[0]),
               "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(mapped_bar)
               : "memory");
}
// Waits of whole warps, as bounded as ring_wait. The lanes decide together: where some saw the phase end and others
// that a wait had run out, the warp would go on in two parts, over instructions that all of it has to execute.
// The loop is out of line: inline, around a phase that has already ended, it cost 100 to 180 cycles where the first
// test costs 40.
// CLUSTER: what the phase stands for was written, or read, by other CTAs of the cluster.
template <bool CLUSTER>
__device__ __forceinline__ bool kt_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  } else {
    ok = mbar_try_wait_at(bar, parity);
  }
  return __all_sync(0xffffffffu, ok);
}
template <bool CLUSTER>
__device__ __forceinline__ bool kt_wait_loop(uint32_t bar, uint32_t parity, volatile int* abort, int* err) {
  for (uint32_t it = 0; it < (1u << 22); ++it) {
    if (kt_try_wait<CLUSTER>(bar, parity)) return true;
    if (__any_sync(0xffffffffu, *abort)) return false;
  }
  *abort = 1;
  if (err) atomicOr(err, DEVERR_MBAR_TIMEOUT);
  return false;
}
template <bool CLUSTER>
__device__ __noinline__ bool kt_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort, int* err) { return kt_wait_loop<CLUSTER>(bar, parity, abort, err); }
template <bool CLUSTER = false>
__device__ __forceinline__ bool kt_wait(const Ring& R, uint64_t* bar, uint32_t parity) {
  if (kt_try_wait<CLUSTER>(smem_addr(bar), parity)) return true;
  return kt_wait_slow<CLUSTER>(smem_addr(bar), parity, R.abort, R.err);
}
// The same with the loop in line, after the first test: for warps whose registers leave no room for a call.
__device__ __forceinline__ bool kt_wait_inline(const Ring& R, uint64_t* bar, uint32_t parity) {
  if (kt_try_wait<false>(smem_addr(bar), parity)) return true;
  return kt_wait_loop<false>(smem_addr(bar), parity, R.abort, R.err);
}
// What a wait that runs out does, brought about by the option "give_up": after that many requests of a CTA.
__device__ __forceinline__ void kt_give_up(const Ring& R) {
  *R.abort = 1;
  if (R.err) atomicOr(R.err, DEVERR_MBAR_TIMEOUT);
}

// The exchange of a pair: 128 threads meet at barrier `bar`, and leave together: a warp whose wait gave up would
// leave the others waiting at the next meeting.
__device__ __forceinline__ bool kt_meet(int bar, bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "barrier.cta.red.and.pred.aligned q, %1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all)
      : "r"(bar), "r"((uint32_t)ok)
      : "memory");
  return all != 0;
}

// ---- tensor memory ------------------------------------------------------------------------
__device__ __forceinline__ void kt_st16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
      "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void kt_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void kt_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void kt_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
// A from tensor memory (a lane per row), B from shared memory, D in tensor memory.
__device__ __forceinline__ void kt_mma_i8(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void kt_mma_f16(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%4, %4, %4, %4}, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(0u)
      : "memory");
}
// Core matrices of 8 tokens x 16 bytes: the next 16 bytes of K 128 bytes on, the next 8 tokens a block on.
__device__ __forceinline__ uint64_t kt_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(XT_BLOCK >> 4) << 32) | (1ull << 46);
}

// Words [0, W) of a 2-byte aligned array that starts `off` bytes (even, 0..14) after the 16-byte
// aligned shared address `base`: aligned 16-byte loads (a row per thread: no bank conflicts, which
// word loads would have), then the shift.
template <int W>
__device__ __forceinline__ void kt_words(uint32_t base, uint32_t off, uint32_t (&out)[W]) {
  constexpr int L = (W + 4 + 3) / 4;
  uint32_t v[4 * L];
#pragma unroll
  for (int i = 0; i < L; i++) {
    const U4 t = gm_lds128(base + 16 * i);
    v[4 * i] = t.x;
    v[4 * i + 1] = t.y;
    v[4 * i + 2] = t.z;
    v[4 * i + 3] = t.w;
  }
  const bool k2 = off & 8u, k1 = off & 4u;
#pragma unroll
  for (int i = 0; i < W + 2; i++) v[i] = k2 ? v[i + 2] : v[i];
#pragma unroll
  for (int i = 0; i < W + 1; i++) v[i] = k1 ? v[i + 1] : v[i];
#pragma unroll
  for (int i = 0; i < W; i++) out[i] = funnel_r(v[i], v[i + 1], (off & 2u) * 8u);
}

// Half u of the row's block at shared address p (Q6_K: `off` bytes after it) -> digits in tensor
// memory at column address a (u = 1: and the mins). Returns {d, dmin}.
template <int KIND>
__device__ __forceinline__ float2 kt_unpack(uint32_t p, uint32_t off, uint32_t a, int u) {
  if constexpr (KIND == Q6_K) {
    uint32_t sc[5], l[16], h[8];
    kt_words<5>(p + 192, off, sc);
    kt_words<16>(p + 64 * u, off, l);
    kt_words<8>(p + 128 + 32 * u, off, h);
    const uint32_t sc0 = u ? sc[2] : sc[0], sc1 = u ? sc[3] : sc[1];
#pragma unroll
    for (int up = 0; up < 4; up++) {  // 32 elements: low or high nibbles, bits 2 * up, 2 * up + 1 of h
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t lb = l[8 * (up & 1) + i], hb = h[i];
        const uint32_t v = ((up & 2 ? lb >> 4 : lb) & 0x0F0F0F0Fu) | ((up == 0 ? hb << 4 : up == 1 ? hb << 2 : up == 2 ? hb : hb >> 2) & 0x30303030u);
        const int s = 2 * up + (i >> 2), scale = sext_byte(s < 4 ? sc0 : sc1, s & 3);
        // two 16-bit products at a time; they stay positive, so nothing carries between them
        const uint32_t add = (uint32_t)((4096 - 32 * scale) * 65537);
        const uint32_t e = prmt(v, 0, 0x4240) * (uint32_t)scale + add, o = prmt(v, 0, 0x4341) * (uint32_t)scale + add;
        lo[i] = prmt(e, o, 0x6240);
        hi[i] = prmt(e, o, 0x7351);
      }
      kt_st8(a + 32 * u + 8 * up, lo);
      kt_st8(a + 64 + 32 * u + 8 * up, hi);
    }
    return make_float2(half_bits_hw(sc[4] & 0xFFFFu), 0.0f);
  } else {
    const U4 hdr = gm_lds128(p);
    const K4Scales s = k4_unpack(hdr.y, hdr.z, hdr.w);
    const uint32_t scw = u ? s.sc_hi : s.sc_lo;
    if (u) {
      uint32_t mins[8];
#pragma unroll
      for (int j = 0; j < 8; j++) mins[j] = half2_of_byte(j < 4 ? s.m_lo : s.m_hi, j & 3);
      kt_st8(a + 128, mins);
    }
    const float2 d = make_float2(half_bits_hw(hdr.x & 0xFFFFu), half_bits_hw(hdr.x >> 16));
    constexpr bool Q5 = KIND == Q5_K;
    U4 h0 = {0, 0, 0, 0}, h1 = {0, 0, 0, 0};
    if (Q5) {
      h0 = gm_lds128(p + 16);
      h1 = gm_lds128(p + 32);
    }
    const uint32_t h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
    for (int c = 0; c < 2; c++) {  // 32 bytes: sub-blocks 2c (low nibbles) and 2c + 1 of the half
      const uint32_t qs = p + (Q5 ? 48 : 16) + 64 * u + 32 * c;
      const U4 q0 = gm_lds128(qs), q1 = gm_lds128(qs + 16);
      const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      uint32_t lo[16], hi[16];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int j = 2 * c + e;
        const uint32_t sc = byte_of(scw, j), s0 = sc & 7u, s1 = sc >> 3;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          uint32_t v = (e ? w[i] >> 4 : w[i]) & 0x0F0F0F0Fu;
          if (Q5) v |= ((u ? h[i] >> j : h[i] << (4 - j)) & 0x10101010u);  // bit 4 * u + j
          lo[8 * e + i] = v * s0;
          hi[8 * e + i] = v * s1;
        }
      }
      kt_st16(a + 32 * u + 16 * c, lo);
      kt_st16(a + 64 + 32 * u + 16 * c, hi);
    }
    return d;
  }
}

// Slot of a ring and the parity of its current phase.
struct KtPos {
  int slot = 0;
  uint32_t par = 0;
  __device__ __forceinline__ void advance(int n) {
    if (++slot == n) {
      slot = 0;
      par ^= 1u;
    }
  }
};

template <int KIND, int C>
__global__ void __launch_bounds__(KT_THREADS, 1) kt_kernel(const __grid_constant__ KtParams P) {
  using K = KtKind<KIND>;
  constexpr int OQ = KT_QUADS / C;  // quads of an owner
  extern __shared__ __align__(128) uint8_t smem[];
  // [terms x 2][activation slots][raw slots][row scales][barriers][tensor memory base][abort]
  const int nt = P.nt, nt16 = (nt + 1) >> 1, b_bytes = nt16 * 2 * XT_BLOCK;
  uint8_t* const terms = smem;
  uint8_t* const b_ring = terms + 2 * KT_TERMS;
  uint8_t* const raw_ring = b_ring + P.n_b * b_bytes;
  float2* const side = reinterpret_cast<float2*>(raw_ring + P.n_raw * K::RAW);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(side + KT_SIDE_SLOTS * KT_ROWS);
  float* const exchange = reinterpret_cast<float*>(bars + KT_BARS + 1 + (KT_BARS + 1) % 2);  // pairs only
  uint64_t* const raw_full = bars;
  uint64_t* const raw_empty = raw_full + KT_MAX_SLOTS;
  uint64_t* const b_full = raw_empty + KT_MAX_SLOTS;
  uint64_t* const b_empty = b_full + KT_MAX_SLOTS;
  uint64_t* const a_full = b_empty + KT_MAX_SLOTS;
  uint64_t* const a_empty = a_full + 2;
  uint64_t* const d_full = a_empty + 2;
  uint64_t* const d_empty = d_full + 2;
  uint64_t* const t_full = d_empty + 2;
  uint64_t* const t_empty = t_full + 2;
  uint64_t* const side_full = t_empty + 2;
  uint64_t* const drain = side_full + KT_SIDE_SLOTS;
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  Ring R;  // for its bounded waits
  R.abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  R.err = P.err;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank();
  const int nb = P.cols >> 8, n_st = (nb + C - 1) / C;
  const int cl = blockIdx.x / C, n_cl = gridDim.x / C;
  const int halves = nt16 > 2 ? 2 : 1;                     // MMA groups of at most 32 tokens
  const int n16 = halves == 2 ? 2 : nt16;                  // tokens / 16 of the first
  const int trows = P.pair ? KT_ROWS / 2 : KT_ROWS;        // rows of the row space per tile
  // what the other CTAs send this one in the stage-th stage (counted over its tiles): their blocks of the
  // stage times the quads it owns
  const int my_quads = (4 * nt16 - rank + C - 1) / C;
  auto t_expect = [&](int stage, uint64_t* bar) { mbar_expect_tx(bar, (uint32_t)((min(C, nb - stage % n_st * C) - (stage % n_st * C + rank < nb ? 1 : 0)) * my_quads * KT_ROWS * 16)); };
  if (warp == 2 && P.tma && lane < P.nseg) prefetch_map(&P.map[lane]);
  if (tid < KT_BARS) {  // a thread per barrier
    constexpr int S4 = KT_MAX_SLOTS;
    const int i = tid;
    const int count = i < S4 ? (P.tma ? 1 : 64)   // raw_full
                      : i < 2 * S4 ? 8            // raw_empty
                      : i < 3 * S4 ? 1            // b_full
                      : i < 4 * S4 ? 9            // b_empty
                      : i < 4 * S4 + 2 ? 8        // a_full
                      : i < 4 * S4 + 6 ? 1        // a_empty, d_full
                      : i < 4 * S4 + 8 ? 8        // d_empty
                      : i < 4 * S4 + 10 ? 9       // t_full
                      : i < 4 * S4 + 12 ? 4 * C   // t_empty
                      : i < 4 * S4 + 12 + KT_SIDE_SLOTS ? 4 : 1;  // side_full, drain
    mbar_init(bars + i, count);
    if (i >= 4 * S4 + 8 && i < 4 * S4 + 10) t_expect(i - 4 * S4 - 8, bars + i);
    if (i == 0) *R.abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) tc_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_arrive();  // every CTA's barriers are set up before another CTA writes there: the warps that do wait for it
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  // matrix and first row of a tile
  auto locate = [&](int tile, int& sg, int& r0) {
    sg = 0;
    if (!P.pair)
      while (sg < P.nseg - 1 && tile >= P.tiles_before[sg + 1]) sg++;
    r0 = (tile - P.tiles_before[sg]) * trows;
  };

  if (warp == 0) {
    // ---- activations ----
    KtPos pb;
    bool ok = true;
    int left = P.give_up;
    pdl_wait();
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok; tile += n_cl) {
#pragma unroll 1
      for (int sb = rank; sb < nb; sb += C) {
        ok = kt_wait(R, &b_empty[pb.slot], pb.par ^ 1u);
        if (!ok) break;
        if (elect_one()) {
          mbar_expect_tx(&b_full[pb.slot], (uint32_t)(nt * XT_BLOCK));
          bulk_g2s(b_ring + pb.slot * b_bytes, P.xf + (size_t)sb * P.xf_nt * XT_BLOCK, (uint32_t)(nt * XT_BLOCK), &b_full[pb.slot]);
          if (left && --left == 0) kt_give_up(R);
        }
        __syncwarp();
        pb.advance(P.n_b);
      }
    }
  } else if (warp == 1) {
    // ---- MMAs ----
    const uint32_t idesc = (2u << 4) | (1u << 10) | ((KT_ROWS >> 4) << 24), fdesc = (1u << 4) | ((KT_ROWS >> 4) << 24);
    KtPos pa, pb, pd;
    bool ok = true;
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok; tile += n_cl) {
#pragma unroll 1
      for (int s = 0; s < n_st && ok; s++) {
        if (s * C + rank >= nb) continue;
        ok = kt_wait(R, &b_full[pb.slot], pb.par) && kt_wait(R, &a_full[pa.slot], pa.par);
        if (!ok) break;
        const uint32_t a = tmem + KT_A_BASE + pa.slot * KT_A_COLS, b0 = smem_addr(b_ring + pb.slot * b_bytes);
#pragma unroll 1
        for (int h = 0; h < halves; h++) {
          ok = kt_wait(R, &d_empty[pd.slot], pd.par ^ 1u);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t n = (uint32_t)(2 * (h ? nt16 - 2 : n16)) << 17, d = tmem + pd.slot * KT_D_COLS, bh = b0 + h * 4 * XT_BLOCK;
            const uint64_t db = kt_desc(bh);
            if (KIND != Q6_K) kt_mma_f16(d + 64, a + 128, kt_desc(bh + XT_BSUMS), fdesc | n);
#pragma unroll
            for (int j = 0; j < 8; j++) {
              kt_mma_i8(d, a + 8 * j, db + 16 * j, idesc | n, j);
              kt_mma_i8(d + 32, a + 64 + 8 * j, db + 16 * j, idesc | n, j);
            }
            tc_commit(&d_full[pd.slot]);
            if (h == halves - 1) {
              tc_commit(&a_empty[pa.slot]);
              tc_commit(&b_empty[pb.slot]);
            }
          }
          __syncwarp();
          pd.advance(2);
        }
        pa.advance(2);
        pb.advance(P.n_b);
      }
    }
    // every MMA has finished before the tensor memory and the operands go
    if (elect_one()) tc_commit(drain);
    __syncwarp();
    mbar_wait(drain, 0, P.err);
  } else if (warp < 4) {
    // ---- rows; they do not depend on the previous kernel ----
    const int g = lane >> 2, q = lane & 3;
    KtPos pr;
    bool ok = true;
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok && !(P.tma && warp == 3); tile += n_cl) {
      int sg, r0;
      locate(tile, sg, r0);
#pragma unroll 1
      for (int sb = rank; sb < nb; sb += C) {
        ok = kt_wait(R, &raw_empty[pr.slot], pr.par ^ 1u);
        if (!ok) break;
        const uint32_t dst = smem_addr(raw_ring + pr.slot * K::RAW);
        if (P.tma) {
          const int x = (KIND == Q6_K ? (sb * K::BS) & ~15 : sb * K::BS) >> 2;
          if (elect_one()) {
            mbar_expect_tx(&raw_full[pr.slot], K::RAW);
            tma_load_2d(dst, &P.map[sg], x, r0, &raw_full[pr.slot]);
            if (P.pair) tma_load_2d(dst + K::RAW / 2, &P.map[1], x, r0, &raw_full[pr.slot]);
          }
          __syncwarp();
        } else {  // four lanes per row
#pragma unroll 2
          for (int i = 0; i < KT_ROWS / 16; i++) {
            const int r = (2 * i + warp - 2) * 8 + g;
            const GemvSeg& G = P.seg[P.pair ? r >> 6 : sg];
            // rows past the matrix repeat its last row, their results are dropped
            const int row = min(r0 + (P.pair ? r & 63 : r), G.rows - 1);
            const uint8_t* src = G.w + ((size_t)row * nb + sb) * K::BS;
            if (KIND == Q6_K) src = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15);
#pragma unroll
            for (int j = 0; j < (K::PIECES + 3) / 4; j++)
              if (4 * j + 3 < K::PIECES || 4 * j + q < K::PIECES) cp_async16(dst + r * K::PITCH + 16 * q + 64 * j, src + 16 * q + 64 * j);
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_addr(&raw_full[pr.slot])) : "memory");
        }
        pr.advance(P.n_raw);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp < 12) {
    // ---- unpack ----
    const int row = (tid - 128) & 127, u = (warp - 4) >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    KtPos pr, pa, ps;
    bool ok = true;
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok; tile += n_cl) {
      int sg, r0;
      locate(tile, sg, r0);
      const GemvSeg& G = P.seg[P.pair ? row >> 6 : sg];
      const uint32_t row_at = (uint32_t)(uintptr_t)G.w + (uint32_t)min(r0 + (P.pair ? row & 63 : row), G.rows - 1) * (uint32_t)nb * K::BS;
#pragma unroll 1
      for (int s = 0; s < n_st; s++) {
        const int sb = s * C + rank;
        if (sb >= nb) continue;
        ok = kt_wait(R, &raw_full[pr.slot], pr.par) && kt_wait(R, &a_empty[pa.slot], pa.par ^ 1u);
        if (!ok) break;
        tc_fence_after();
        const float2 d = kt_unpack<KIND>(smem_addr(raw_ring + pr.slot * K::RAW + row * K::PITCH), KIND == Q6_K ? (row_at + sb * K::BS) & 15u : 0u,
                                                        tmem + lanes + KT_A_BASE + pa.slot * KT_A_COLS, u);
        if (u == 0) side[ps.slot * KT_ROWS + row] = d;
        kt_wait_st();
        tc_fence_before();
        __syncwarp();
        if (elect_one()) {
          mbar_arrive(&raw_empty[pr.slot]);
          mbar_arrive(&a_full[pa.slot]);
          if (u == 0) mbar_arrive(&side_full[ps.slot]);
        }
        __syncwarp();
        pr.advance(P.n_raw);
        pa.advance(2);
        ps.advance(KT_SIDE_SLOTS);
      }
    }
  } else if (warp < 20) {
    // ---- terms ----
    cluster_sync_wait();
    const int row = (tid - 384) & 127, e16 = (warp - 12) >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t owner[4];  // terms ring of the CTAs that own this thread's quads 4 * e16 + qd (+ 8h); the barriers lie t_bar after it
#pragma unroll
    for (int qd = 0; qd < 4; qd++) owner[qd] = cluster_map(smem_addr(terms), (4 * e16 + qd) % C);
    const uint32_t t_bar = smem_addr(t_full) - smem_addr(terms);
    KtPos pb, pd, ps, pt;
    bool ok = true;
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok; tile += n_cl) {
#pragma unroll 1
      for (int s = 0; s < n_st; s++) {
        const bool mine = s * C + rank < nb;
        float2 d = make_float2(0.0f, 0.0f);
        if (mine) {
          ok = kt_wait(R, &side_full[ps.slot], ps.par) && kt_wait(R, &b_full[pb.slot], pb.par);
          if (!ok) break;
          d = side[ps.slot * KT_ROWS + row];
        }
        const F2 dd = f2_pack(d.x, d.x), dm = f2_pack(d.y, d.y), minus1 = f2_pack(-1.0f, -1.0f);
        ok = kt_wait<true>(R, &t_empty[pt.slot], pt.par ^ 1u);
        if (!ok) break;
        if (mine) {
          const uint32_t tb = pt.slot * KT_TERMS + (rank * OQ * KT_ROWS + row) * 16, fb = t_bar + 8 * pt.slot, own = smem_addr(terms) + tb;
#pragma unroll
          for (int h = 0; h < KT_MAX_M / 32; h++) {
            if (h >= halves) break;
            ok = kt_wait(R, &d_full[pd.slot], pd.par);
            if (!ok) break;
            tc_fence_after();
            const int t16 = 2 * h + e16;
            const uint32_t at = tmem + lanes + pd.slot * KT_D_COLS + e16 * 16;
            const uint32_t xg = smem_addr(b_ring + pb.slot * b_bytes) + t16 * 2 * XT_BLOCK;
#pragma unroll
            for (int g8 = 0; g8 < 2 && t16 < nt16; g8++) {
              uint32_t lo[8], hi[8], sm[8];
              kt_ld8(at + 8 * g8, lo);
              kt_ld8(at + 32 + 8 * g8, hi);
              if (KIND != Q6_K) kt_ld8(at + 64 + 8 * g8, sm);
              tc_wait_ld();
#pragma unroll
              for (int q2 = 0; q2 < 2; q2++) {
                const int qd = 2 * g8 + q2;
                const uint32_t xq = xg + g8 * XT_BLOCK + q2 * 16;
                const U4 dx = gm_lds128(xq + XT_D);
                U4 sx = {0, 0, 0, 0};
                if (KIND == Q6_K) sx = gm_lds128(xq + XT_SUMS);
                const uint32_t dxs[4] = {dx.x, dx.y, dx.z, dx.w}, sxs[4] = {sx.x, sx.y, sx.z, sx.w};
                float t[4];
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                  const int i = 4 * q2 + e;
                  const F2 x = f2_pack(__uint_as_float(dxs[e]), __uint_as_float(dxs[e + 1]));
                  F2 sumi;
                  if (KIND == Q6_K) {
                    sumi = f2_pack(i2f((int)(lo[i] + sxs[e] + (hi[i] << 8))), i2f((int)(lo[i + 1] + sxs[e + 1] + (hi[i + 1] << 8))));
                  } else {
                    sumi = f2_pack(i2f((int)(lo[i] + (hi[i] << 3))), i2f((int)(lo[i + 1] + (hi[i + 1] << 3))));
                  }
                  F2 v = f2_mul(f2_mul(dd, x), sumi);
                  if (KIND != Q6_K)  // t - m as an fma by -1: a packed sum would be contracted with the product before it
                    v = f2_fma(f2_mul(f2_mul(dm, x), f2_pack(__uint_as_float(sm[i]), __uint_as_float(sm[i + 1]))), minus1, v);
                  f2_unpack(v, t[e], t[e + 1]);
                }
                const uint32_t to = owner[qd] + tb + (8 * h + 4 * e16 + qd) / C * (KT_ROWS * 16);
                if ((4 * e16 + qd) % C != rank) cluster_st128(to, owner[qd] + fb, t);
                else asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(own + (8 * h + 4 * e16 + qd) / C * (KT_ROWS * 16)), "f"(t[0]), "f"(t[1]), "f"(t[2]), "f"(t[3]) : "memory");
              }
            }
            tc_fence_before();
            __syncwarp();
            if (elect_one()) mbar_arrive(&d_empty[pd.slot]);
            __syncwarp();
            pd.advance(2);
          }
          if (!ok) break;
          ps.advance(KT_SIDE_SLOTS);
        }
        __syncwarp();
        if (elect_one()) mbar_arrive(&t_full[pt.slot]);
        __syncwarp();
        if (mine) {
          if (elect_one()) mbar_arrive(&b_empty[pb.slot]);
          __syncwarp();
          pb.advance(P.n_b);
        }
        pt.advance(2);
      }
    }
  } else {
    // ---- sums in block order, and what is done with them ----
    cluster_sync_wait();
    const int row = tid - 640;
    const uint32_t empty_at = cluster_map(smem_addr(t_empty), lane & (C - 1));
    KtPos pt;
    bool ok = true;
    const int stages = (P.n_tiles - cl + n_cl - 1) / n_cl * n_st;
    int stage = 0;
    pdl_wait();
#pragma unroll 1
    for (int tile = cl; tile < P.n_tiles && ok; tile += n_cl) {
      int sg, r0;
      locate(tile, sg, r0);
      F2 acc[OQ][2];
#pragma unroll
      for (int i = 0; i < OQ; i++) acc[i][0] = acc[i][1] = f2_pack(0.0f, 0.0f);
#pragma unroll 1
      for (int s = 0; s < n_st; s++) {
        ok = kt_wait<true>(R, &t_full[pt.slot], pt.par);
        if (!ok) break;
        // (the other three warps' phase cannot end again before they have said that they read this one)
        if (warp == 20 && stage + 2 < stages) {
          if (elect_one()) t_expect(stage + 2, &t_full[pt.slot]);
          __syncwarp();
        }
        stage++;
        const uint32_t at = smem_addr(terms) + pt.slot * KT_TERMS + row * 16;
        // loads in groups of eight, then their sums: a branch for each would wait out its load
        constexpr int CG = C < 8 ? 8 / C : 1;  // quads of a group
        const int cnt = min(C, nb - s * C);
#pragma unroll
        for (int i0 = 0; i0 < OQ; i0 += CG) {
          if (i0 * C + rank >= 4 * nt16) break;
          U4 v[CG][C];
#pragma unroll
          for (int i = 0; i < CG; i++)
#pragma unroll
            for (int c = 0; c < C; c++) v[i][c] = gm_lds128(at + (c * OQ + i0 + i) * (KT_ROWS * 16));
#pragma unroll
          for (int c = 0; c < C; c++) {
            if (c >= cnt) break;
#pragma unroll
            for (int i = 0; i < CG; i++) {
              acc[i0 + i][0] = f2_add(acc[i0 + i][0], f2_pack(__uint_as_float(v[i][c].x), __uint_as_float(v[i][c].y)));
              acc[i0 + i][1] = f2_add(acc[i0 + i][1], f2_pack(__uint_as_float(v[i][c].z), __uint_as_float(v[i][c].w)));
            }
          }
        }
        __syncwarp();
        if (lane < C) cluster_arrive(empty_at + 8 * pt.slot);
        pt.advance(2);
      }
      if (!ok) {
        if (P.pair) kt_meet(1, false);
        break;
      }
      float out[OQ][4];
#pragma unroll
      for (int i = 0; i < OQ; i++) {
        f2_unpack(acc[i][0], out[i][0], out[i][1]);
        f2_unpack(acc[i][1], out[i][2], out[i][3]);
      }
      const GemvSeg& G = P.seg[P.pair ? row >> 6 : sg];
      const int gr = r0 + (P.pair ? row & 63 : row);
      if (P.pair) {
        // threads 0..63 hold gate rows, 64.. the up rows of the same numbers: after an exchange of half of
        // the quads both finish half of the results
        constexpr int HQ = OQ / 2;
        float* const xch = exchange + row * KT_XCH<C>;
        const bool up = row >= 64;
#pragma unroll
        for (int i = 0; i < HQ; i++)
          *reinterpret_cast<float4*>(xch + 4 * i) = up ? make_float4(out[2 * i][0], out[2 * i][1], out[2 * i][2], out[2 * i][3])
                                                       : make_float4(out[2 * i + 1][0], out[2 * i + 1][1], out[2 * i + 1][2], out[2 * i + 1][3]);
        ok = kt_meet(1, true);
        if (!ok) break;
        const float* const other = exchange + (row ^ 64) * KT_XCH<C>;
#pragma unroll
        for (int i = 0; i < HQ; i++) {
          const float4 o = *reinterpret_cast<const float4*>(other + 4 * i);
          const float os[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float gate = up ? os[e] : out[2 * i][e], upv = up ? out[2 * i + 1][e] : os[e];
            const int tok = ((2 * i + up) * C + rank) * 4 + e;
            const size_t at = (size_t)tok * G.rows + gr;
            if (tok < P.m && gr < G.rows) {
              P.seg[0].out[at] = P.epilogue == EPI_SILU_MUL ? silu_mul_exact(gate, upv) : gate;
              P.seg[1].out[at] = upv;
            }
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");  // the next tile writes the exchange again
      } else if (gr < G.rows) {
#pragma unroll
        for (int i = 0; i < OQ; i++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int tok = (i * C + rank) * 4 + e;
            float* const o = G.out + (size_t)tok * G.rows + gr;
            if (tok < P.m) *o = P.epilogue == EPI_ACCUM ? fadd(*o, out[i][e]) : out[i][e];
          }
      }
    }
  }
  __syncwarp();
  if (warp < 12) cluster_sync_wait();
  tc_fence_before();
  __syncthreads();
  cluster_sync_arrive();  // nobody writes into a CTA that has left
  cluster_sync_wait();
  if (warp == 1) {
    // Nothing is written into a CTA that has left. Who has done all its stages has all that was requested and all its
    // terms; after a wait that gave up, whichever warp's, some may be on their way still, and the cluster barrier does
    // not wait for what was sent asynchronously.
    if (*R.abort) {
      for (int i = 0; i < P.n_b; i++) mbar_drain(&b_full[i]);
      for (int i = 0; i < P.n_raw && P.tma; i++) mbar_drain(&raw_full[i]);
      for (int i = 0; i < 2; i++) mbar_drain(&t_full[i]);
    }
    tc_dealloc(tmem, 512);
  }
}

}  // namespace aot

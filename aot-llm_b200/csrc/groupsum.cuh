// Exact sequential-order f32 sums evaluated by a group of warps (device side of seqsum.cuh).
#pragma once
#include "blockmath.cuh"
#include "seqsum.cuh"

namespace aot {

// ---- a group of warps inside a CTA that synchronise on a named barrier ---------------
struct CtaGroup {
  int tid;       // thread index inside the group
  int nthreads;  // multiple of 32
  int bar_id;    // hardware barrier id (0 = the whole CTA, like __syncthreads)
  __device__ __forceinline__ void sync() const {
    if (nthreads == 32) {  // a single warp needs no hardware barrier (there are only 16 of them)
      __syncwarp();
      return;
    }
    asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(nthreads) : "memory");
  }
};

// Optional sub-phase cycle counters (slots 16..31 of the profile array).
struct SubProf {
  unsigned long long* prof;
  long long last;
  __device__ __forceinline__ void mark(int slot) {
    if (prof) {
      long long now = clock64();
      atomicAdd(&prof[slot], (unsigned long long)(now - last));  // fire and forget: no wait for the old value
      last = now;
    }
  }
};

// The form with an item per run and per slow chunk (ties included), however many there are: for
// sums whose terms keep changing binade. Every thread of the group calls it; scratch as above.
__device__ __noinline__ float group_seq_sum_items(const float* p, int n, SeqSumScratch* sc, int gtid, int gthreads, int bar_id) {
  const CtaGroup g{gtid, gthreads, bar_id};
  const int tid = g.tid, lane = tid & 31, warp = tid >> 5, nwarps = g.nthreads >> 5;
  const bool walker = tid == (nwarps - 1) * 32;
  g.sync();
  if (n <= SEQ_HEAD) {
    // short sums: one thread's add chain
    if (walker) {
      float s = 0.0f;
      for (int i = 0; i < n; i++) s = fadd(s, p[i]);
      sc->s = s;
    }
    g.sync();
    return sc->s;
  }
  if (walker) {
    // the opening chain, beside passes 1 and 2 of the warps that own groups
    float s = 0.0f;
    // all loads first, then the chain
    float hv[SEQ_HEAD];
#pragma unroll
    for (int k = 0; k < SEQ_HEAD; k++) hv[k] = p[k];
#pragma unroll
    for (int k = 0; k < SEQ_HEAD; k++) s = fadd(s, hv[k]);
    sc->s = s;
  }
  float approx = 0.0f;  // inexact sum of the passes before this one
  for (int base = 0; base < n; base += SEQ_CHUNKS * SEQ_E) {
    const int len = min(n - base, SEQ_CHUNKS * SEQ_E), nch = (len + SEQ_E - 1) / SEQ_E, ngr = (nch + 31) >> 5;
    // 1. inexact sums: per chunk, prefix inside the group, group totals
    for (int gr = warp; gr < ngr; gr += nwarps) {
      const int c = gr * 32 + lane, i0 = c * SEQ_E;
      float t = 0.0f;
#pragma unroll
      for (int j = 0; j < SEQ_E; j++) t += i0 + j < len ? p[base + i0 + j] : 0.0f;
      float incl = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      sc->excl[c] = incl - t;
      if (lane == 31) sc->gtot[gr] = incl;
    }
    g.sync();
    // 2. predicted exponents, increments, runs, items
    float total = approx;
#pragma unroll
    for (int k = 0; k < SEQ_CHUNKS / 32; k++) total += k < ngr ? sc->gtot[k] : 0.0f;
    for (int gr = warp; gr < ngr; gr += nwarps) {
      const int c = gr * 32 + lane, i0 = c * SEQ_E;
      float before = approx;
#pragma unroll
      for (int k = 0; k < SEQ_CHUNKS / 32; k++) before += k < gr ? sc->gtot[k] : 0.0f;  // all loads issue together
      before += sc->excl[c];
      float t = 0.0f;
      uint32_t vb[SEQ_E];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < SEQ_E; j++) {
        const float v = i0 + j < len ? p[base + i0 + j] : 0.0f;
        vb[j] = f2u(v) & 0x7FFFFFFFu;
        cnt += i0 + j < len ? 1 : 0;
        t += v;
      }
      const int eb = seq_exp_field(before), ea = seq_exp_field(before + t);
      const int head_lanes = base == 0 && gr == 0 ? SEQ_HEAD / SEQ_E : 0;  // chunks of the opening chain
      const bool live = lane >= head_lanes;
      bool bad = ea != eb || eb >= 255;
      int inc = 0;
#pragma unroll
      for (int j = 0; j < SEQ_E; j++) inc += seq_increment(vb[j], eb, bad);
      const bool slow = live && cnt > 0 && bad;
      inc = slow || !live ? 0 : min(inc, SUMFN_SAT);
      const int eb_prev = __shfl_up_sync(0xffffffffu, eb, 1);
      const int slow_prev = __shfl_up_sync(0xffffffffu, (int)slow, 1);
      const bool starts = live && (lane == head_lanes || slow_prev || eb != eb_prev);
      const uint32_t slow_mask = __ballot_sync(0xffffffffu, slow);
      const uint32_t begin = __ballot_sync(0xffffffffu, starts) | slow_mask;  // lanes at which an item begins
      // first chunk of this lane's item: the highest item begin at or below the lane
      const uint32_t below = begin & (0xFFFFFFFFu >> (31 - lane));
      const int rs = below ? 31 - __clz((int)below) : lane;
      // segmented inclusive scan of the increments inside runs
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane - d >= rs) inc = min(inc + o, SUMFN_SAT);
      }
      // the last chunk of an item writes it
      const bool next_begins = lane == 31 || ((begin >> (lane + 1)) & 1u);
      if (live && next_begins) {
        const int first = (gr * 32 + rs) * SEQ_E;
        SeqItem it;
        it.csum = inc;
        it.ep = slow ? -1 : eb;
        it.first = first;
        it.count = max(0, min(len, (c + 1) * SEQ_E) - first);
        sc->item[32 * gr + __popc(below) - 1] = it;
      }
      if (lane == 0) sc->n_items[gr] = __popc(begin);
    }
    g.sync();
    // 3. the walk
    if (walker) {
      sc->s = seqsum_walk(p + base, sc, ngr, sc->s);
    }
    g.sync();
    approx = total;
  }
  return sc->s;
}


// ---- exact sequential-order sum of non-negative floats in shared memory --------------
// (((0 + p[0]) + p[1]) + ...) with the rounding of a scalar f32 loop (seqsum.cuh): lanes own
// chunks of SEQ_E terms, warps own groups of 32 chunks. Pass 1 gives every chunk an inexact
// prefix sum, which predicts the exponent the running sum will have there. Pass 2 turns every
// chunk into the function "mantissa -> mantissa + a[its parity]" for that exponent (exact ties
// included: they only look at the parity) and composes the chunks of a binade, per group, by a
// segmented warp scan; between two binades lies one chunk in which the sum changes exponent.
// One warp then composes the groups of each binade, and walks the binades: one integer step and
// eight real adds each.
//
// What bounds it is the serial end: one warp's dependent instructions. Measured on a row of 2048
// squares: 4.3 K cycles on its own (9.3 K with an item per run, crossing chunk and tie walked one
// by one through shared memory; 11.2 K for a plain chain), 4.0 K inside the decode step (7.8 K).
// A wrong prediction, a sum that goes down in the inexact prefix or more than SEQ_BINADES
// binades are noticed and send the whole sum to group_seq_sum_items.
constexpr int SEQ_BINADES = 8;
constexpr int SEQ_GROUPS = 16;  // groups per round: 4096 terms

struct SeqFastScratch {
  int2 fn[SEQ_BINADES * SEQ_GROUPS];  // composed function of a group's chunks in a binade; x < 0: none
  int cross[SEQ_BINADES];             // 1 + the chunk that leaves the binade; 0: none
  float gtot[SEQ_GROUPS];
  float zero[SEQ_E];                  // eight zeros: the crossing chunk of a binade without one
  int e0;                             // exponent field of binade 0
  int over;
  float s;
};
static_assert(sizeof(SeqFastScratch) <= sizeof(SeqSumScratch), "the scratch is shared with the fallback");

__device__ __forceinline__ void seq_fast_clear(SeqFastScratch* sc, int tid, int nthreads) {
  for (int i = tid; i < SEQ_BINADES * SEQ_GROUPS; i += nthreads) sc->fn[i] = make_int2(-1, 0);
  if (tid < SEQ_BINADES) sc->cross[tid] = 0;
  if (tid < SEQ_E) sc->zero[tid] = 0.0f;
  if (tid == 0) sc->over = 0;
}

// Group `gr` of a round of `len` terms: the lane's eight terms and the inexact sum of everything in
// front of its chunk; `after`: that of everything up to the group's end (the next group's first
// `before`, formed the same way, so that neighbouring chunks agree on the exponent between them).
__device__ __forceinline__ void seq_group_fn(const float (&v)[SEQ_E], float before, float after, int gr, int len, int head_lanes, int e0,
                                             SeqFastScratch* sc) {
  const int lane = threadIdx.x & 31, c = gr * 32 + lane;
  const int eb = seq_exp_field(before), e_after = seq_exp_field(after);
  int ea = __shfl_down_sync(0xffffffffu, eb, 1);
  if (lane == 31) ea = e_after;
  const bool live = lane >= head_lanes && c * SEQ_E < len;
  // The chunk's adds from an even and from an odd mantissa, done as f32 adds in a binade where the
  // unit is 1: rounding (ties included) depends on the fraction and the parity only, so each chain
  // advances by what the running sum advances by, in units of its own last place.
  const float scale = u2f((uint32_t)(277 - eb) << 23);  // 2^(150 - eb): eb in 24 .. 254 below
  float u = 8388608.0f, w = 8388609.0f;
#pragma unroll
  for (int j = 0; j < SEQ_E; j++) {
    const float x = fmul(v[j], scale);
    u = fadd(u, x);
    w = fadd(w, x);
  }
  int a0 = (int)f2u(u) - 0x4B000000, a1 = (int)f2u(w) - 0x4B000001;
  const bool bad = (f2u(u) >> 23) != 150u || (f2u(w) >> 23) != 150u;  // more than a binade
  const bool cross = live && ea != eb;
  const int bi = eb - e0;
  bool over = live && (ea < eb || (bad && !cross) || bi < 0 || bi >= SEQ_BINADES || eb < 24 || eb >= 255);
  if (cross || !live) a0 = a1 = 0;
  const int eb_prev = __shfl_up_sync(0xffffffffu, eb, 1);
  const uint32_t begin = __ballot_sync(0xffffffffu, live && (lane == head_lanes || eb != eb_prev));
  // first chunk of this lane's binade in the group: the highest begin at or below the lane
  const uint32_t below = begin & (0xFFFFFFFFu >> (31 - lane));
  const int rs = below ? 31 - __clz((int)below) : lane;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int p0 = __shfl_up_sync(0xffffffffu, a0, d), p1 = __shfl_up_sync(0xffffffffu, a1, d);
    if (lane - d >= rs) {
      const int c0 = a0, c1 = a1;
      a0 = min(p0 + ((p0 & 1) ? c1 : c0), SUMFN_SAT);
      a1 = min(p1 + ((p1 & 1) ? c0 : c1), SUMFN_SAT);
    }
  }
  const bool last = lane == 31 || ((begin >> (lane + 1)) & 1u) || (c + 1) * SEQ_E >= len;
  if (live && !over) {
    if (cross) over = atomicExch(&sc->cross[bi], c + 1) != 0;
    if (last) sc->fn[bi * SEQ_GROUPS + gr] = make_int2(a0, a1);
  }
  if (__any_sync(0xffffffffu, over) && lane == 0) sc->over = 1;
}

// First f, then g (x < 0: the identity).
__device__ __forceinline__ int2 seq_fn_then(int2 f, int2 g) {
  if (f.x < 0) return g;
  if (g.x < 0) return f;
  return make_int2(min(f.x + ((f.x & 1) ? g.y : g.x), SUMFN_SAT), min(f.y + ((f.y & 1) ? g.x : g.y), SUMFN_SAT));
}

// The walk over the binades of a round, by one whole warp: `s` plus the round's terms, the same in
// every lane. False when a prediction was wrong.
__device__ __forceinline__ bool seq_walk_binades(const float* p, int len, const SeqFastScratch* sc, float& s) {
  const int lane = threadIdx.x & 31, e0 = sc->e0;
  const int4 x0 = *reinterpret_cast<const int4*>(sc->cross), x1 = *reinterpret_cast<const int4*>(sc->cross + 4);
  const int cross[SEQ_BINADES] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
  // lane 4 b + k composes groups 4 k .. 4 k + 3 of binade b
  const int4* fp = reinterpret_cast<const int4*>(sc->fn + (lane >> 2) * SEQ_GROUPS + 4 * (lane & 3));
  const int4 f0 = fp[0], f1 = fp[1];
  int2 f = seq_fn_then(seq_fn_then(make_int2(f0.x, f0.y), make_int2(f0.z, f0.w)), seq_fn_then(make_int2(f1.x, f1.y), make_int2(f1.z, f1.w)));
#pragma unroll
  for (int d = 1; d <= 2; d <<= 1) {
    const int2 g = make_int2(__shfl_down_sync(0xffffffffu, f.x, d), __shfl_down_sync(0xffffffffu, f.y, d));
    if ((lane & 3) + d < 4) f = seq_fn_then(f, g);
  }
  uint32_t bits = f2u(s) & 0x7FFFFFFFu;
  bool ok = true;
#pragma unroll
  for (int h = 0; h < SEQ_BINADES; h += 4) {
    // everything the chain of four binades needs, fetched before it starts
    int a0[4], a1[4];
    float4 t0[4], t1[4];
#pragma unroll
    for (int b = 0; b < 4; b++) {
      a0[b] = __shfl_sync(0xffffffffu, f.x, 4 * (h + b));
      a1[b] = __shfl_sync(0xffffffffu, f.y, 4 * (h + b));
      const float* q = cross[h + b] ? p + (cross[h + b] - 1) * SEQ_E : sc->zero;
      t0[b] = *reinterpret_cast<const float4*>(q);
      t1[b] = *reinterpret_cast<const float4*>(q + 4);
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const bool any = a0[b] >= 0;
      const uint32_t nb = bits + (uint32_t)(any ? ((bits & 1u) ? a1[b] : a0[b]) : 0);
      ok = ok && (!any || ((int)(bits >> 23) == e0 + h + b && (int)(nb >> 23) == e0 + h + b));
      float x = u2f(nb);
      x = fadd(fadd(fadd(fadd(x, t0[b].x), t0[b].y), t0[b].z), t0[b].w);
      x = fadd(fadd(fadd(fadd(x, t1[b].x), t1[b].y), t1[b].z), t1[b].w);
      bits = f2u(x) & 0x7FFFFFFFu;
    }
  }
  s = u2f(bits);
  return ok;
}

// Lane's terms of chunk c of a round (zeros behind it).
__device__ __forceinline__ void seq_chunk(const float* p, int len, int c, float (&v)[SEQ_E]) {
  float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
  if (c * SEQ_E < len) {
    a = *reinterpret_cast<const float4*>(p + c * SEQ_E);
    b = *reinterpret_cast<const float4*>(p + c * SEQ_E + 4);
  }
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ float seq_chunk_sum(const float (&v)[SEQ_E]) {
  return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}
__device__ __forceinline__ float seq_warp_scan(float t) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_up_sync(0xffffffffu, t, o);
    if (lane >= o) t += y;
  }
  return t;
}
// A plain add chain over p[0 .. n), n a multiple of SEQ_E or zero-filled to one; the same in every
// lane. About 5 cycles per term, and up to SEQ_CHAIN_MAX terms quicker than the passes.
constexpr int SEQ_CHAIN_MAX = 768;
__device__ __forceinline__ float seq_chain(const float* p, int n) {
  float s = 0.0f;
#pragma unroll 4
  for (int i = 0; i < n; i += SEQ_E) {
    const float4 a = *reinterpret_cast<const float4*>(p + i), b = *reinterpret_cast<const float4*>(p + i + 4);
    s = fadd(fadd(fadd(fadd(s, a.x), a.y), a.z), a.w);
    s = fadd(fadd(fadd(fadd(s, b.x), b.y), b.z), b.w);
  }
  return s;
}

// Every thread of the group calls it (p 16-byte aligned and zero-filled to a multiple of SEQ_E
// terms). Opens with a barrier; the result in every thread.
__device__ __forceinline__ float group_seq_sum(const float* p, int n, SeqSumScratch* scratch, const CtaGroup& g, unsigned long long* prof = nullptr) {
  SubProf sp{prof, clock64()};
  SeqFastScratch* const sc = reinterpret_cast<SeqFastScratch*>(scratch);
  const int tid = g.tid, lane = tid & 31, warp = tid >> 5, nwarps = g.nthreads >> 5;
  const bool walker = warp == nwarps - 1;
  const int round = min(SEQ_GROUPS, 2 * nwarps) * 32 * SEQ_E;  // at most two groups per warp
  g.sync();
  float s = 0.0f, approx = 0.0f;
  if (walker) s = seq_chain(p, n <= SEQ_CHAIN_MAX ? n : SEQ_HEAD);  // beside the passes of the warps that own groups
  for (int base = 0; base < n && n > SEQ_CHAIN_MAX; base += round) {
    const int len = min(n - base, round), ngr = (len + 32 * SEQ_E - 1) / (32 * SEQ_E), head = base == 0 ? SEQ_HEAD / SEQ_E : 0;
    seq_fast_clear(sc, tid, g.nthreads);
    float excl[2] = {0.0f, 0.0f}, t[2] = {0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int gr = warp + k * nwarps;
      if (gr < ngr) {
        float v[SEQ_E];
        seq_chunk(p + base, len, gr * 32 + lane, v);
        t[k] = seq_chunk_sum(v);
        const float incl = seq_warp_scan(t[k]);
        excl[k] = incl - t[k];
        if (lane == 31) sc->gtot[gr] = incl;
        if (gr == 0 && lane == head) sc->e0 = seq_exp_field(approx + excl[k]);
      }
    }
    g.sync();
    if (prof && tid == 0) sp.mark(26);
    float total = approx;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int gr = warp + k * nwarps;
      if (gr < ngr) {
        float v[SEQ_E];
        seq_chunk(p + base, len, gr * 32 + lane, v);
        float before = approx;
#pragma unroll
        for (int j = 0; j < SEQ_GROUPS; j++) before += j < gr ? sc->gtot[j] : 0.0f;  // all loads issue together
        seq_group_fn(v, before + excl[k], before + sc->gtot[gr], gr, len, gr == 0 ? head : 0, sc->e0, sc);
      }
    }
    if (base + round < n)
      for (int j = 0; j < ngr; j++) total += sc->gtot[j];
    g.sync();
    if (prof && tid == 0) sp.mark(28);
    if (walker && !sc->over) {
      const long long tw = clock64();
      if (!seq_walk_binades(p + base, len, sc, s) && lane == 0) sc->over = 1;
      if (lane == 0) sc->s = s;
      if (prof) atomicAdd(&prof[31], (unsigned long long)(clock64() - tw));
    }
    g.sync();
    if (sc->over) return group_seq_sum_items(p, n, scratch, g.tid, g.nthreads, g.bar_id);  // uniform over the group
    if (base + round < n) g.sync();  // (the flag is cleared next)
    approx = total;
  }
  if (n <= SEQ_CHAIN_MAX) {
    if (walker && lane == 0) sc->s = s;
    g.sync();
  }
  if (prof && tid == 0) sp.mark(29);
  return sc->s;
}

}  // namespace aot

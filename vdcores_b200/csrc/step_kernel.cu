// One token of a model at batch 1, as one persistent kernel.
//
// A step streams every weight once (1 FLOP per byte), so HBM is the floor; what a step costs beyond it are the places where
// every SM needs what all SMs have just computed, five per layer.  Two things make those short here:
//   * The producer warp of a CTA knows every weight row and cache page of the whole step beforehand and copies them through a
//     ring of ~170 KB without looking at the stages: HBM keeps streaming while the other warps wait for activations.
//   * Activations travel as 8-byte entries {payload, tag}.  A consumer polls the entries themselves; no fence, counter or flag
//     stands between a result and the SMs that wait for it.
// The same step as a program of the megakernel (csrc/megakernel.cu) counts barriers down: fence, atomic, poll, then a copy,
// about 7 us per boundary.
//
// Measured against that program (B200): three layers of width 512 109 -> 46 us, eight 8B-shaped bf16 layers and a 128256-row
// vocabulary projection 1012 -> 800, four such layers e4m3 387 -> 230, NVFP4 388 -> 225, four layers of a 30B mixture of experts
// 437 -> 201 (up to 2 % more or less from one GPU to another).
//
// An entry buffer is written again one layer later, when everything that read it must have been read: whoever polls a buffer
// has rows in the same or the following stage, and those rows go into what the next writer of the buffer waits for.
#include "mk_stage.cuh"

namespace vdc {

// Consumer warps; one more warp produces.  All of them execute what a stage's boundary needs and wait there for entries in L2 and,
// instruction by instruction, for the one before: twice as many would execute it all twice as often (four 8B-shaped layers 515 us with
// sixteen, 451 with eight).
constexpr int kStepWarps = 8;
constexpr int kStepThreads = 32 * kStepWarps;
constexpr int kItems = 16;                           // copies in the ring, at most
constexpr int kItemBytes = 32 * 1024;                // bytes of one, at most
constexpr int kPageBytes = VDC_KV_PAGE * VDC_HEAD_DIM * 2;
constexpr int kGroups = kStepWarps / 4;              // of four warps: a page of the cache each
constexpr int kAlone = 4;                            // pages that one SM walks without splitting them
constexpr int kFewSplits = 32;                       // of a head, while that leaves each kAlone pages at most
constexpr int kOutLd = VDC_HEAD_DIM + 4;
constexpr int kPartFloats = 4 * 8 * kOutLd;          // partial sums of rows; also the groups' partial heads
constexpr int kQLd = VDC_HEAD_DIM / 2 + 4;           // words of a query row in shared memory
constexpr int kPLd = VDC_KV_PAGE / 2 + 4;            // words of a row of probabilities
constexpr int kMaxTopK = 16, kMaxExperts = 256;
constexpr int kScaleBytes = kStepThreads * 16;       // four scales of quantised rows per thread
constexpr int kStepSmem = 227 * 1024 - 1024;         // dynamic; the rest is StepShared's barriers

enum { kQkv, kOut, kRouter, kGateUp, kDown, kVocab, kStages };

// How an SM's consumers take a stage's rows: first row and rows; rows of a chunk; a warp's steps along the inputs; the teams and
// the warps along the inputs (log2); the steps of a slice (0: rows whole); and the rows between two sums of them.
struct Plan {
  int r0, n, per, units, lt, lk, slice, most;
};

// An SM's share of the attention: one KV head's pages first .. first + count - 1; `live` splits of the head have pages.  Up to
// kAlone pages stay with one SM: there is nothing to merge then.  Few KV heads leave a head more splits than a warp has lanes;
// they are used once 32 splits would walk more than kAlone pages each.  Eight layers of width 1024 with one KV head at 32000 /
// 128000 positions 373 -> 274 and 839 -> 396 us, two 382 -> 315 and 876 -> 533 (with 8 or 16 pages in place of kAlone one head
// at 32000 positions takes 309 and 386).
struct Pages {
  int h, split, live, first, count;
};
__device__ __forceinline__ Pages pages_of(const vdc_step& s, int pos, int sm) {
  Pages p{sm % s.n_kv, sm / s.n_kv, 0, 0, 0};
  const int n = min(pos / VDC_KV_PAGE + 1, s.max_pages);
  const int per = n <= kAlone ? n : max((n + s.n_splits - 1) / s.n_splits, min((n + kFewSplits - 1) / kFewSplits, kAlone));
  p.live = (n + per - 1) / per;
  if (p.split < p.live) {
    p.first = p.split * per;
    p.count = min(per, n - p.first);
  }
  return p;
}

struct StepShared {
  uint64_t full[kItems], empty[kItems], routed;
  int start[kItems];                                 // offset of an item in the ring
  volatile int fail;
  alignas(16) float red[kStepWarps];
  float best[kStepWarps];
  int best_row[kStepWarps];
  alignas(16) Plan plan[kStages];
  int slot0, head;                                   // experts: the slot of this SM's first gate/up row, its rows there are
  int pos, token, new_row;                           // of the step; the new row's place in the cache pools
  Pages pages;
  int four0, four1;                                  // fours of a head's dims that this SM merges
};
// Behind the ring: what the consumers share.
struct StepLayout {
  int ring, x, h, part, raw, q, rows, p, gm, wl, route, scales;
  int total;
};
__host__ __device__ inline StepLayout step_layout(const vdc_step& s) {
  const int q = s.n_kv * s.group * VDC_HEAD_DIM, act = s.ffn * (s.n_experts ? s.top_k : 1);
  int xw = s.hidden > q ? s.hidden : q;
  if (act > xw) xw = act;
  StepLayout l;
  int at = 0;
  auto take = [&](int bytes) {
    const int r = at;
    at += (bytes + 127) / 128 * 128;
    return r;
  };
  l.x = take(xw * 2);
  l.h = take(s.hidden * 2);
  l.part = take(kPartFloats * 4);
  l.raw = take(10 * VDC_HEAD_DIM * 2);
  l.q = take(8 * kQLd * 4);
  l.rows = take(2 * VDC_HEAD_DIM * 2 + VDC_HEAD_DIM * 2);       // new key and value row; zeros
  l.p = take(kGroups * 8 * kPLd * 4);
  l.gm = take(kGroups * 4 * 8 * 4);
  l.wl = take(kGroups * 5 * 8 * 4);
  l.route = take(kMaxExperts * 4 + 2 * kMaxTopK * 4);
  l.scales = take(s.wfmt ? kScaleBytes : 0);
  l.ring = at;
  l.total = kStepSmem - 128;
  return l;
}

// Entry buffers in the workspace, in 8-byte words; word 0 counts the launches.
struct StepWork {
  size_t h, qkv, rec, ml, attn, act, router, best, words;
};
__host__ __device__ inline StepWork step_work(const vdc_step& s) {
  StepWork w;
  size_t at = 16;
  auto take = [&](size_t n) {
    const size_t r = at;
    at += (n + 15) / 16 * 16;
    return r;
  };
  const size_t heads = (size_t)s.n_kv * s.group;
  w.h = take(s.hidden);                                        // two versions of hidden / 2 entries
  w.qkv = take((heads + 2 * (size_t)s.n_kv) * VDC_HEAD_DIM / 2);
  w.rec = take((size_t)s.n_kv * s.n_splits * s.group * VDC_HEAD_DIM);
  w.ml = take((size_t)s.n_kv * s.n_splits * s.group * 2);
  w.attn = take(heads * VDC_HEAD_DIM / 2);
  w.act = take((size_t)s.ffn * (s.n_experts ? s.top_k : 1) / 2);
  w.router = take(s.n_experts ? s.n_experts : 1);
  w.best = take(2 * (size_t)s.num_sms);
  w.words = at;
  return w;
}

// A stage as the host divides it: the first `more` SMs take each + 1 units of q rows, the others `each`; lt, lk and most for
// either.  A stage's boundary on the device had 1000 to 2300 cycles of integer divisions for this (of 8000 to 11000).
struct Deal {
  int q, each, more, per, units;
  int lt[2], lk[2], slice[2], most[2];
};
// What a launch passes: the step, where its shared memory and its entries lie, how its stages are divided.  From the constant bank
// these cost no registers.
struct StepArgs {
  vdc_step s;
  StepLayout lay;
  StepWork wk;
  Deal deal[kStages];
  float inv_hidden;
  int q_width, qkv_width;
};
// Rows of a stage that one SM takes.
struct Share {
  int r0, n;
};

// ------------------------------------------------------------------------- //
// entries
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void put(uint64_t* p, uint32_t payload, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((uint64_t)tag << 32) | payload) : "memory");
}
__device__ __forceinline__ void put2(uint64_t* p, uint32_t a, uint32_t b, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(((uint64_t)tag << 32) | a),
               "l"(((uint64_t)tag << 32) | b)
               : "memory");
}
struct Two {
  uint64_t a, b;
  __device__ __forceinline__ bool are(uint32_t tag) const { return (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag; }
};
__device__ __forceinline__ Two get2(const uint64_t* p) {
  Two v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
  return v;
}

// A thread's own copies of 8 bytes to shared memory, waited for by the thread itself: loads that hold no registers while they are
// on their way.
__device__ __forceinline__ void copy8_async(void* to, uint64_t from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------------------- //
// dot products of a chunk's rows
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t e4m3_pair(uint32_t pair) {
  uint32_t d;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(d) : "h"((unsigned short)pair));
  return d;
}
__host__ __device__ constexpr int row_bytes(int fmt, int K) { return fmt == 0 ? 2 * K : fmt == 1 ? K : K / 2 + K / 16; }
__host__ __device__ constexpr int unit_of(int fmt) { return fmt == 0 ? 256 : fmt == 1 ? 512 : 1024; }     // inputs of a warp's step

// Weights as the tensor cores take them: four (bf16), four (e4m3) or eight (NVFP4) of a lane's 16 bytes, which is two, one or
// one word of them, as bf16 or f16 pairs.  An NVFP4 weight times its block's scale is exact in f16.
template <int kFmt>
__device__ __forceinline__ void expand(uint32_t (&o)[kFmt == 2 ? 4 : 2], const uint4& v, int part, uint32_t scales) {
  const uint32_t c[4] = {v.x, v.y, v.z, v.w};
  if constexpr (kFmt == 0) {
    o[0] = c[2 * part];
    o[1] = c[2 * part + 1];
  } else if constexpr (kFmt == 1) {
    e4m3x4_to_half2(c[part], o);
  } else {
    const uint32_t sc = __byte_perm(scales, 0, part < 2 ? 0x1010 : 0x3232);
    e2m1x8_to_half2(c[part], o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const __half2 p = __hmul2(*reinterpret_cast<const __half2*>(&o[j]), *reinterpret_cast<const __half2*>(&sc));
      o[j] = *reinterpret_cast<const uint32_t*>(&p);
    }
  }
}

// Models with experts: packed fp32 FMAs of the widened pairs, sums rounded to nearest at every product.  The router's softmax
// is steep enough that the last bits of what stands in front of it can be seen behind it.
template <int kPairs>
__device__ __forceinline__ void dot_fma(float2 (&d)[2 * kPairs], const uint8_t* w, const int (&row)[4], const uint8_t* x, int u, int lane) {
  auto pair = [](uint32_t v) { return make_float2(bf_lo(v), bf_hi(v)); };
  const uint4 xv = lds128(x + u * 512 + lane * 16);
  const float2 xf[4] = {pair(xv.x), pair(xv.y), pair(xv.z), pair(xv.w)};
#pragma unroll
  for (int i = 0; i < 2 * kPairs; ++i) {
    const uint4 v = lds128(w + row[i] + u * 512 + lane * 16);
    d[i] = __ffma2_rn(pair(v.x), xf[0], d[i]);
    d[i] = __ffma2_rn(pair(v.y), xf[1], d[i]);
    d[i] = __ffma2_rn(pair(v.z), xf[2], d[i]);
    d[i] = __ffma2_rn(pair(v.w), xf[3], d[i]);
  }
}

__device__ __forceinline__ void add2(float& a, float& b, float x, float y) {
  const float2 v = __fadd2_rn(make_float2(a, b), make_float2(x, y));
  a = v.x;
  b = v.y;
}

// kSteps steps of a warp (u, u + kw, ...): 16 bytes per lane of kPairs pairs of rows times the same inputs, as products of 16 x 16
// by 16 x 8 tiles.  Row g of a tile is what the four lanes 4g .. 4g + 3 hold of the pair's first row (8 + g: of its second), column
// g what they hold of the inputs: the tile's element (g, g) is the sum of the four lanes' products, the other elements mean nothing.
// A product of tiles is one instruction where FMAs of four rows are 12 (32 KB of bf16 took 0.8 us with those, HBM 0.73).
// All loads of the steps are issued before the first product waits for one: see steps_of.
// The tensor cores cut off what an fp32 sum cannot hold.  So bf16 and e4m3 rows have only two products of tiles (8 of a lane's
// inputs) added up by them, from zero; those sums meet in rounded additions.  Of 32768 sums of 8192 products around two large
// ones that cancel, 2.0 % miss their bf16 rounding (FMAs 2.1 %, all products in one sum of the tensor cores 7.2 %).  Four
// 8B-shaped layers e4m3 325 -> 329 us, eight bf16 the same.  NVFP4 rows keep long sums, two of them in turn: the megakernel's
// program adds 16 of their products up in f16.
template <int kFmt, int kPairs, int kSteps>
__device__ __forceinline__ void dot_steps(float (&d)[kFmt == 2 ? 2 : 1][kPairs][4], const uint8_t* w, const int (&row)[4], bool single, const uint8_t* x,
                                          int u, int kw, int lane, int K) {
  constexpr int kParts = kFmt == 0 ? 2 : 4, kWords = kFmt == 2 ? 4 : 2;       // of a lane's 16 bytes; expanded words of one
  constexpr int kXs = kParts * kWords / 4;                                    // 16-byte pieces of a lane's inputs
  uint4 xs[kSteps][kXs], c[kSteps][2 * kPairs];
  uint32_t sc[kSteps][2 * kPairs];
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    const int v = u + j * kw;
#pragma unroll
    for (int i = 0; i < 2 * kPairs; ++i) {
      const uint8_t* r = w + row[i];
      const bool none = (i & 1) && single;
      c[j][i] = none ? make_uint4(0u, 0u, 0u, 0u) : lds128(r + v * 512 + lane * 16);
      sc[j][i] = kFmt == 2 && !none ? *reinterpret_cast<const uint16_t*>(r + (K >> 1) + v * 64 + lane * 2) : 0u;
    }
#pragma unroll
    for (int i = 0; i < kXs; ++i) xs[j][i] = lds128(x + v * unit_of(kFmt) * 2 + lane * 16 + i * 512);
  }
#pragma unroll
  for (int j = 0; j < kSteps; ++j) {
    float t[kPairs][4];
    if (kFmt == 2) {
#pragma unroll
      for (int i = 0; i < 2 * kPairs; ++i) sc[j][i] = e4m3_pair(sc[j][i]);
    }
#pragma unroll
    for (int part = 0; part < kParts; ++part) {
      const int at = part * kWords;                                             // first expanded word
      const uint4 xq = xs[j][at >> 2];
      const uint32_t xv[4] = {xq.x, xq.y, xq.z, xq.w};
#pragma unroll
      for (int p = 0; p < kPairs; ++p) {
        uint32_t a[kWords], b[kWords];
        expand<kFmt>(a, c[j][2 * p], part, sc[j][2 * p]);
        expand<kFmt>(b, c[j][2 * p + 1], part, sc[j][2 * p + 1]);
        if (kFmt != 2 && (part & 1) == 0) t[p][0] = t[p][1] = t[p][2] = t[p][3] = 0.f;
        float(&sum)[4] = kFmt == 2 ? d[kFmt == 2 ? part & 1 : 0][p] : t[p];
#pragma unroll
        for (int k = 0; k < kWords; k += 2) {
          if (kFmt == 0) mma_bf16(sum, a[k], b[k], a[k + 1], b[k + 1], xv[(at & 3) + k], xv[(at & 3) + k + 1]);
          else mma_f16(sum, a[k], b[k], a[k + 1], b[k + 1], xv[(at & 3) + k], xv[(at & 3) + k + 1]);
        }
        if (kFmt != 2 && (part & 1) != 0) {
          add2(d[0][p][0], d[0][p][1], t[p][0], t[p][1]);
          add2(d[0][p][2], d[0][p][3], t[p][2], t[p][3]);
        }
      }
    }
  }
}
// Steps of a warp whose loads are on their way together.  With one (and the products in the order of the source) a warp took 290
// cycles for a step of four bf16 rows, a chain of a load, two products and an addition.  A step of NVFP4 rows is as many products
// by itself as four of bf16 (four 8B-shaped layers 232 us, 246 with two steps and the registers they spill), and so is one of two
// pairs of e4m3 rows; of one pair four at once (four 8B-shaped layers 237 us with two steps of either, 232.7 so).
__host__ __device__ constexpr int steps_of(int fmt, int pairs) { return fmt == 0 || (fmt == 1 && pairs == 1) ? 4 : 1; }

// Units of q rows; the first SMs' shares are never empty while there are any.
__host__ __device__ inline Share share_of(int rows, int q, int sm, int sms) {
  const int units = rows / q;
  const int each = units / sms, more = units % sms;             // the first `more` SMs take one unit more
  return {(sm * each + (sm < more ? sm : more)) * q, (each + (sm < more ? 1 : 0)) * q};
}
__host__ __device__ constexpr int chunk_rows(int rb) {        // an even number where more than one
  const int n = kItemBytes / rb < 32 ? kItemBytes / rb : 32;
  return n > 1 ? n & ~1 : 1;
}

// How the warps share n rows of K inputs: teams of them take the chunks in turn, so that one's way through a chunk (a few
// hundred cycles of latency) falls into the others'; a team's warps divide the rows, and the inputs (kw of them).
// Dense bf16 rows of which four make more than one copy are cut along the inputs: a copy is `slice` steps of four rows,
// the teams take a group's slices in turn and every warp keeps its sums of the four rows until the group ends.  Four rows read
// the inputs from shared memory once instead of four times, and their sums meet once: a row of 28 KB took a team 2500 cycles,
// 1.15 of what HBM takes to bring it.  Eight 8B-shaped layers 905 -> 887 us (four with e4m3 rows, two of which are a copy, 296 ->
// 306: those stay whole).
struct Split {
  int teams, kw, slice;
};
// Two teams, since a chunk's place in the ring is held for as long as its team works on it.  With 2 / 4 teams: eight 8B-shaped bf16
// layers 799 / 808 us, four e4m3 230 / 238, NVFP4 224 / 224.5, the 30B mixture of experts 198 / 201.  NVFP4 rows and experts keep four
// for their sums' sake: where a chunk has fewer than eight rows two warps keep two sums of each, a team of four four, and there would be
// room for half as many rows (hidden 6912: 1056 gate/up rows of the chosen experts to an SM instead of 2112).
__host__ __device__ inline int teams_of(int fmt, bool experts, int K, int n) {
  const int chunks = n / chunk_rows(row_bytes(fmt, K));
  return (fmt == 2 || experts) && chunks >= 4 ? 4 : chunks >= 2 ? 2 : 1;
}
__host__ __device__ inline Split split_of(int fmt, bool experts, bool vocab, int K, int n) {
  const int units = K / unit_of(fmt), most = kItemBytes / (4 * 512);
  if (fmt == 0 && !experts && units > most && n >= 4 && (vocab || n <= kPartFloats / kStepWarps)) return {2, kStepWarps, most};
  Split s{teams_of(fmt, experts, K, n), 1, 0};
  // Along the inputs only as far as a warp would otherwise have fewer than four rows of a chunk: the sums over its lanes come once
  // per four rows, whatever the inputs.  With the inputs divided as far as possible four 8B-shaped e4m3 layers took 232.6 us, 228.8 so,
  // NVFP4 229.9 and 225.4, the mixture of experts 208.8 and 201.
  const int per = chunk_rows(row_bytes(fmt, K)), rows = n < per ? n : per, warps = kStepWarps / s.teams;
  while (s.kw < warps && 2 * s.kw <= units && rows < 4 * (warps / s.kw)) s.kw *= 2;
  return s;
}

__host__ inline Deal deal_of(const vdc_step& s, int stage) {
  const int k = s.n_experts ? s.top_k : 1, Q = s.n_kv * s.group * VDC_HEAD_DIM;
  const int rows[kStages] = {Q + 2 * s.n_kv * VDC_HEAD_DIM, s.hidden, s.n_experts, 2 * s.ffn * k, s.hidden, s.vocab};
  const int K = stage == kOut ? Q : stage == kDown ? s.ffn : s.hidden, fmt = stage == kVocab ? 0 : s.wfmt;
  Deal d{};
  d.q = stage == kGateUp ? 4 : stage == kRouter ? 1 : 2;
  d.each = rows[stage] / d.q / s.num_sms;
  d.more = rows[stage] / d.q % s.num_sms;
  d.per = chunk_rows(row_bytes(fmt, K));
  d.units = K / unit_of(fmt);
  for (int i = 0; i < 2; ++i) {
    const int n = (d.each + (i == 0)) * d.q;
    const Split sp = split_of(fmt, s.n_experts != 0, stage == kVocab, K, stage == kDown ? n * k : n);
    while (1 << d.lt[i] < sp.teams) ++d.lt[i];
    while (1 << d.lk[i] < sp.kw) ++d.lk[i];
    d.slice[i] = sp.slice;
    const int per = sp.slice ? 4 : d.per;
    d.most[i] = stage == kVocab ? kPartFloats / sp.kw / per * per : n;
  }
  return d;
}

// ------------------------------------------------------------------------- //
// producer
// ------------------------------------------------------------------------- //
// A whole warp: its lanes decide the same and an item's pieces are copied by a lane each.  (One lane alone takes 300 to 400 cycles
// per piece: with four pieces to an item it took longer to ask for a row of 28 KB than HBM to bring it.)
struct Producer {
  StepShared& sh;
  const Waiter& wait;
  uint8_t* ring;
  int cap, lane;
  RingAt at{kItems};       // next item
  int oldest = 0, live = 0, wr = 0, count = 0;
  int mine = 0;            // offset in the ring of item `lane`
  uint32_t oldest_parity = 0u;
  bool wrapped = false, ok = true;

  // Room for one more item of `bytes`, freeing the oldest ones as they are consumed.
  __device__ __forceinline__ uint8_t* room(int bytes) {
    bytes = (bytes + 127) & ~127;
    int first = __shfl_sync(0xffffffffu, mine, oldest);
#pragma unroll 1
    while (ok) {
      if (live < kItems) {
        if (live == 0) {
          wr = 0;
          wrapped = false;
        }
        if (!wrapped && wr + bytes > cap && bytes <= first) {
          wr = 0;
          wrapped = true;
        }
        if (wr + bytes <= (wrapped ? first : cap)) break;
      }
      ok = wait.warp_wait(&sh.empty[oldest], oldest_parity, 0, count);
      const int was = first;
      if (++oldest == kItems) {
        oldest = 0;
        oldest_parity ^= 1u;
      }
      first = __shfl_sync(0xffffffffu, mine, oldest);
      --live;
      if (live > 0 && first < was) wrapped = false;
    }
    uint8_t* p = ring + wr;
    if (lane == at.st) mine = wr;
    if (lane == 0) sh.start[at.st] = wr;
    wr += bytes;
    ++live;
    return p;
  }
  // One item of n pieces of `bytes`, the i-th from this lane's src in lane i.
  __device__ __forceinline__ void item(const uint8_t* src, int n, int bytes) {
    uint8_t* p = room(n * bytes);
    if (!ok) return;
    if (lane == 0) mbar_arrive_expect_tx(&sh.full[at.st], (uint32_t)(n * bytes));
    if (lane < n) bulk_load_1d(p + lane * bytes, src, (uint32_t)bytes, &sh.full[at.st]);
    __syncwarp();
    at.next();
    ++count;
  }
};

// ------------------------------------------------------------------------- //
// consumers
// ------------------------------------------------------------------------- //
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kStepThreads) : "memory"); }

// Whether to look again for entries that are not there yet (it: looks so far): the time of the first such question, 0 when the wait
// was given up.  Everything by value: what a call could reach by its address would have to be in memory.
static __device__ __noinline__ uint64_t look_again(volatile int* fail, vdc_status* status, uint64_t timeout_ns, uint64_t t0, int at, int it) {
  if (*fail) return 0;
  if (ld_relaxed_gpu(&status->abort) == 0) {
    const uint64_t now = globaltimer_ns();
    if (t0 == 0) return now;
    if (now - t0 <= timeout_ns) return t0;
    report(status, VDC_ERR_TIMEOUT, VDC_STEP_KIND, 1, at, it);
  }
  *fail = 1;
  return 0;
}

template <int n>
struct Steps {
  static constexpr int value = n;
};

struct Consumer {
  const StepArgs& args;
  const vdc_step& s;
  const StepLayout& lay;
  StepShared& sh;
  const Waiter& wait;
  uint8_t* base;
  int tid, warp, lane, sm;
  RingAt at{kItems};
  int teams, turn;               // and the chunks until this warp's team is on
  int kw, kg, rw, rg, ld;        // warps along the inputs, this warp's place there; along the rows; rows there is room for
  int per, units, slice;         // rows of a chunk; steps along the inputs, of a slice of them

  __device__ __forceinline__ float* part() const { return reinterpret_cast<float*>(base + lay.part); }
  __device__ __forceinline__ uint32_t* hs() const { return reinterpret_cast<uint32_t*>(base + lay.h); }
  __device__ __forceinline__ uint8_t* x() const { return base + lay.x; }

  __device__ __forceinline__ bool again(const uint64_t* p, uint32_t it, uint64_t& t0) const {
    t0 = look_again(wait.fail, wait.status, wait.timeout_ns, t0, (int)(p - reinterpret_cast<const uint64_t*>(s.work)), (int)it);
    return t0 != 0;
  }
  __device__ __forceinline__ bool poll2(const uint64_t* p, uint32_t tag, Two& v) const {
    uint64_t t0 = 0;
#pragma unroll 1
    for (uint32_t it = 1; !v.are(tag); ++it) {
      if ((it & 63u) == 0 && !again(p, it, t0)) return false;
      v = get2(p);
    }
    return true;
  }
  // Fours j0 .. j0 + kBatch - 1 of this thread (its j-th is number tid + j * kStepThreads of n) from an entry buffer.  All that a
  // thread still misses is looked for at the same time: one after another, each look is a round trip of its own.
  template <int kBatch>
  __device__ __forceinline__ bool take(const uint64_t* buf, int n, int j0, uint32_t tag, uint2* out) const {
    const int i0 = tid + j0 * kStepThreads;
    Two v[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
      if (i0 + j * kStepThreads < n) v[j] = get2(buf + 2 * (i0 + j * kStepThreads));
    uint64_t t0 = 0;
#pragma unroll 1
    for (uint32_t it = 1;; ++it) {
      bool all = true;
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        if (i0 + j * kStepThreads < n) all = all && v[j].are(tag);
      if (all) break;
      if ((it & 63u) == 0 && !again(buf + 2 * i0, it, t0)) return false;
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        if (i0 + j * kStepThreads < n && !v[j].are(tag)) v[j] = get2(buf + 2 * (i0 + j * kStepThreads));
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) out[j] = make_uint2((uint32_t)v[j].a, (uint32_t)v[j].b);
    return true;
  }
  // n 2-byte values (a multiple of 4) of an entry buffer: f(i, values 4i .. 4i + 3 as two words) for this thread's i.  As many at a
  // time as registers allow: with 14 of them for a down projection's inputs instead of two times 7 values were spilled and eight
  // 8B-shaped layers took 865 instead of 813 us, with four 799.
  template <int kBatch, class F>
  __device__ __forceinline__ void collect(const uint64_t* buf, int n, uint32_t tag, F f) const {
#pragma unroll 1
    for (int j0 = 0; tid + j0 * kStepThreads < n / 4; j0 += kBatch) {
      uint2 v[kBatch];
      if (!take<kBatch>(buf, n / 4, j0, tag, v)) return;
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
        if (tid + (j0 + j) * kStepThreads < n / 4) f(tid + (j0 + j) * kStepThreads, v[j].x, v[j].y);
    }
  }
  // Inputs 4i .. 4i + 3 (two bf16 pairs) as the dot products take them: bf16 in order; f16 for quantised rows, a lane's 16-byte
  // pieces of a step 512 bytes apart, so that neighbouring lanes read neighbouring pieces.
  template <int kFmt>
  static __device__ __forceinline__ int input_at(int i, bool plain) {
    if (kFmt == 0 || plain) return i * 8;
    constexpr int kLane = unit_of(kFmt) / 32;
    const int e = i * 4, u = e / unit_of(kFmt), in = e % unit_of(kFmt);
    return u * unit_of(kFmt) * 2 + (in % kLane) / 8 * 512 + in / kLane * 16 + (i & 1) * 8;
  }
  template <int kFmt>
  __device__ __forceinline__ void set_input(int i, uint32_t a, uint32_t b, bool plain) const {
    uint2* to = reinterpret_cast<uint2*>(x() + input_at<kFmt>(i, plain));
    if (kFmt == 0 || plain) {
      *to = make_uint2(a, b);
      return;
    }
    const __half2 ha = __floats2half2_rn(bf_lo(a), bf_hi(a)), hb = __floats2half2_rn(bf_lo(b), bf_hi(b));
    *to = make_uint2(*reinterpret_cast<const uint32_t*>(&ha), *reinterpret_cast<const uint32_t*>(&hb));
  }
  // The hidden state (entries, or a row of the embedding table) into shared memory and, RMS-normalised with the weights w,
  // into the input vector.  Rounded like a bf16 tensor expression.
  template <int kFmt, int kKept>
  __device__ __forceinline__ void hidden(const uint64_t* buf, uint32_t tag, const uint8_t* row, uint64_t w, bool plain) const {
    const int H = s.hidden;
    constexpr int kMost = 8;                                      // hidden <= 8192; the first kKept stay in registers
    uint2 v[kKept];
    // The weights are on their way while the entries are waited for, to the places of the inputs that they make.  The last stage's
    // inputs there have been read: its partial sums are complete.
#pragma unroll 2
    for (int i = tid; i < H / 4; i += kStepThreads) copy8_async(x() + input_at<kFmt>(i, plain), w + (size_t)i * 8);
    float ssq = 0.f;
#pragma unroll 1
    for (int j0 = (H / 4 - 1) / kStepThreads / kKept * kKept; j0 >= 0; j0 -= kKept) {
      if (row != nullptr) {
#pragma unroll
        for (int j = 0; j < kKept; ++j) {
          const int i = tid + (j0 + j) * kStepThreads;
          if (i < H / 4) v[j] = __ldg(reinterpret_cast<const uint2*>(row) + i);
        }
      } else if (!take<kKept>(buf, H / 4, j0, tag, v)) {
        break;
      }
#pragma unroll
      for (int j = 0; j < kKept; ++j) {
        const int i = tid + (j0 + j) * kStepThreads;
        if (i < H / 4) {
          const uint32_t a = v[j].x, b = v[j].y;
          *reinterpret_cast<uint2*>(hs() + 2 * i) = v[j];
          ssq = fmaf(bf_lo(a), bf_lo(a), fmaf(bf_hi(a), bf_hi(a), fmaf(bf_lo(b), bf_lo(b), fmaf(bf_hi(b), bf_hi(b), ssq))));
        }
      }
    }
    ssq = warp_sum(ssq);
    if (lane == 0) sh.red[warp] = ssq;
    consumers_sync();
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < kStepWarps; k += 4) {
      const float4 r = *reinterpret_cast<const float4*>(sh.red + k);
      tot += r.x; tot += r.y; tot += r.z; tot += r.w;
    }
    // 1 / hidden is exact for powers of two; otherwise its rounding stands for the one that the product in the sum has not
    const float rstd = rsqrtf(fmaf(tot, args.inv_hidden, s.eps));
    copies_wait();
#pragma unroll
    for (int j = 0; j < kMost; ++j) {
      const int i = tid + j * kStepThreads;
      if (j >= kKept && H <= j * 4 * kStepThreads) break;
      if (i < H / 4) {
        const uint2 h = j < kKept ? v[j < kKept ? j : 0] : *reinterpret_cast<const uint2*>(hs() + 2 * i);
        const uint2 wv = *reinterpret_cast<const uint2*>(x() + input_at<kFmt>(i, plain));
        set_input<kFmt>(i, scaled(h.x, rstd, wv.x), scaled(h.y, rstd, wv.y), plain);
      }
    }
    consumers_sync();
  }
  // bf16(bf16(x * rstd) * w) of a pair: the product of two bf16 numbers is exact in fp32, so one rounding in the packed product
  // is the same.
  static __device__ __forceinline__ uint32_t scaled(uint32_t x, float rstd, uint32_t w) {
    const __nv_bfloat162 n = __floats2bfloat162_rn(bf_lo(x) * rstd, bf_hi(x) * rstd);
    const __nv_bfloat162 p = __hmul2(n, *reinterpret_cast<const __nv_bfloat162*>(&w));
    return *reinterpret_cast<const uint32_t*>(&p);
  }

  __device__ __forceinline__ void split(const Plan& p) {
    const int lw = 3 - p.lt;                                   // log2 of a team's warps
    static_assert(kStepWarps == 8, "log2");
    teams = 1 << p.lt;
    kw = 1 << p.lk;
    rw = (1 << lw) >> p.lk;                                    // 0 for slices, which all eight warps divide among themselves
    kg = warp & (kw - 1);
    rg = (warp & ((1 << lw) - 1)) >> p.lk;
    turn = warp >> lw;
    ld = kPartFloats >> p.lk;
    slice = p.slice;
    per = p.per;
    units = p.units;
  }
  // This warp's steps along the inputs, kSteps at a time while there are as many.
  template <int kSteps, class F>
  static __device__ __forceinline__ void walk(int u, int kw, int units, F f) {
#pragma unroll 1
    for (; u + (kSteps - 1) * kw < units; u += kSteps * kw) f(Steps<kSteps>{}, u);
#pragma unroll 1
    for (; u < units; u += kw) f(Steps<1>{}, u);
  }
  // The four lanes 4g + t that hold the diagonal of a product of tiles: of lane l's sums the one of row g, and of row 8 + g.
  template <int kFmt, int kPairs>
  __device__ __forceinline__ void diagonal(const float (&d)[kFmt == 2 ? 2 : 1][kPairs][4], int p, float& first, float& second) const {
    const bool diag = (lane >> 3) == (lane & 3), odd = lane & 4;
    first = diag ? (odd ? d[0][p][1] : d[0][p][0]) : 0.f;
    second = diag ? (odd ? d[0][p][3] : d[0][p][2]) : 0.f;
    if constexpr (kFmt == 2) {
      first += diag ? (odd ? d[1][p][1] : d[1][p][0]) : 0.f;
      second += diag ? (odd ? d[1][p][3] : d[1][p][2]) : 0.f;
    }
  }
  // Four sums over the lanes at once: lanes 8i .. 8i + 7 end up with the i-th.
  __device__ __forceinline__ float sum_lanes(float a, float b, float c, float e) const {
    const bool up = lane & 16, right = lane & 8;
    float p = up ? c : a, q = up ? e : b;
    p += __shfl_xor_sync(0xffffffffu, up ? a : c, 16);
    q += __shfl_xor_sync(0xffffffffu, up ? b : e, 16);
    float v = (right ? q : p) + __shfl_xor_sync(0xffffffffu, right ? p : q, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  // n rows in slices: every warp's share of row r to part[warp][row0 + r].
  template <int kFmt>
  __device__ __forceinline__ void sliced(int n, const uint8_t* xp) {
#pragma unroll 1
    for (int r0 = 0; r0 < n; r0 += 4) {
      const int nr = min(4, n - r0);
      float d[1][2][4] = {};
#pragma unroll 1
      for (int u0 = 0; u0 < units; u0 += slice, at.next(), turn ^= 1) {
        if (!wait.warp_wait(&sh.full[at.st], at.parity, 2, r0)) return;
        if (turn == 0) {
          const uint8_t* w = base + lay.ring + sh.start[at.st];
          const int nu = min(slice, units - u0);
          int off[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) off[i] = min(i, nr - 1) * nu * 512;
          const uint8_t* xs = xp + u0 * (unit_of(kFmt) * 2);
          walk<steps_of(kFmt, 2)>(warp & 3, 4, nu, [&](auto steps, int u) { dot_steps<kFmt, 2, decltype(steps)::value>(d, w, off, false, xs, u, 4, lane, 0); });
          // the place's next bytes come through the other proxy, and nothing that depends on these reads is stored before
          fence_proxy_async_smem();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty[at.st]);
      }
      float a, b, c, e;
      diagonal<kFmt, 2>(d, 0, a, b);
      diagonal<kFmt, 2>(d, 1, c, e);
      const float v = sum_lanes(a, b, c, e);
      if ((lane & 7) == 0 && (lane >> 3) < nr) part()[warp * ld + r0 + (lane >> 3)] = v;
    }
  }
  // n rows from the ring times the inputs xp: every warp's share of row r to part[kg][row0 + r], rows side by side for the
  // threads that add the shares up.
  template <int kFmt, bool kFma>
  __device__ __forceinline__ void rows(int K, int n, const uint8_t* xp, int row0) {
    if constexpr (kFmt == 0 && !kFma) {
      if (slice) return sliced<kFmt>(n, xp);
    }
    const int rb = row_bytes(kFmt, K);
#pragma unroll 1
    for (int r0 = 0; r0 < n; r0 += per, at.next()) {
      if (!wait.warp_wait(&sh.full[at.st], at.parity, 2, r0)) return;
      const uint8_t* w = base + lay.ring + sh.start[at.st];
      const bool mine_now = turn == 0;
      turn = mine_now ? teams - 1 : turn - 1;
      const int nr = mine_now ? min(per, n - r0) : 0;      // every warp sees every chunk arrive, one team works on it
#pragma unroll 1
      for (int r = rg; r < nr; r += 4 * rw) {
        int off[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) off[i] = min(r + i * rw, nr - 1) * rb;
        float a, b, c = 0.f, e = 0.f;          // the lane's share of the four rows
        if (kFma && r + 2 * rw < nr) {
          float2 d[4] = {};
#pragma unroll 2
          for (int u = kg; u < units; u += kw) dot_fma<2>(d, w, off, xp, u, lane);
          a = d[0].x + d[0].y; b = d[1].x + d[1].y; c = d[2].x + d[2].y; e = d[3].x + d[3].y;
        } else if (kFma) {
          float2 d[2] = {};
#pragma unroll 2
          for (int u = kg; u < units; u += kw) dot_fma<1>(d, w, off, xp, u, lane);
          a = d[0].x + d[0].y; b = d[1].x + d[1].y;
        } else if (r + 2 * rw < nr) {
          float d[kFmt == 2 ? 2 : 1][2][4] = {};
          walk<steps_of(kFmt, 2)>(kg, kw, units, [&](auto steps, int u) { dot_steps<kFmt, 2, decltype(steps)::value>(d, w, off, false, xp, u, kw, lane, K); });
          diagonal<kFmt, 2>(d, 0, a, b);
          diagonal<kFmt, 2>(d, 1, c, e);
        } else {
          float d[kFmt == 2 ? 2 : 1][1][4] = {};
          walk<steps_of(kFmt, 1)>(kg, kw, units, [&](auto steps, int u) { dot_steps<kFmt, 1, decltype(steps)::value>(d, w, off, r + rw >= nr, xp, u, kw, lane, K); });
          diagonal<kFmt, 1>(d, 0, a, b);
        }
        const float v = sum_lanes(a, b, c, e);
        const int mine = r + (lane >> 3) * rw;
        if ((lane & 7) == 0 && mine < nr) part()[kg * ld + row0 + r0 + mine] = v;
      }
      // every value read went into the sums stored above, so the reads are complete when the place is given back
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.empty[at.st]);
    }
  }
  __device__ __forceinline__ float sum1(int row) const {
    float v = 0.f;
#pragma unroll 4
    for (int j = 0; j < kw; ++j) v += part()[j * ld + row];
    return v;
  }
  __device__ __forceinline__ float2 sum2(int row) const {      // rows row, row + 1 (row even)
    float2 v = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int j = 0; j < kw; ++j) {
      const float2 a = *reinterpret_cast<const float2*>(part() + j * ld + row);
      v.x += a.x; v.y += a.y;
    }
    return v;
  }
  __device__ __forceinline__ float4 sum4(int row) const {      // four rows (row a multiple of 4)
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int j = 0; j < kw; ++j) {
      const float4 a = *reinterpret_cast<const float4*>(part() + j * ld + row);
      v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
    }
    return v;
  }
  __device__ __forceinline__ bool failed() const { return *wait.fail != 0; }

  // Attention of this SM's unit: queries and the new rows from the QKV entries, its pages from the ring, its share of the
  // head's output to the entries `out`.
  __device__ __forceinline__ void attention(int layer, int pos, const Pages& pg, const uint64_t* qkv, uint64_t* rec, uint64_t* ml,
                                            uint64_t* out, uint32_t tag_in, uint32_t tag_rec, uint32_t tag_out) {
    constexpr int D = VDC_HEAD_DIM;
    const int G = s.group;
    uint32_t* raw = reinterpret_cast<uint32_t*>(base + lay.raw);
    uint32_t* qs = reinterpret_cast<uint32_t*>(base + lay.q);
    uint32_t* krow = reinterpret_cast<uint32_t*>(base + lay.rows);
    uint32_t* vrow = krow + D / 2;
    const bool owner = pg.first + pg.count == min(pos / VDC_KV_PAGE + 1, s.max_pages);
    // what the heads' prologue needs besides the entries is on its way before they are waited for
    const int i0 = lane * 2;
    const float* rope = reinterpret_cast<const float*>(s.rope) + (size_t)pos * D;
    const float2 cs = __ldg(reinterpret_cast<const float2*>(rope + i0)), sn = __ldg(reinterpret_cast<const float2*>(rope + 64 + i0));
    uint32_t nw[4] = {0u, 0u, 0u, 0u};            // norm weights of the queries, of the key
    if (s.qk_norm) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(s.qk_norm) + (size_t)layer * D + lane;
#pragma unroll
      for (int j = 0; j < 4; ++j) nw[j] = __ldg(w + 32 * j);
    }
    collect<2>(qkv + (size_t)pg.h * (G + 2) * (D / 2), (G + 2) * D, tag_in,
               [&](int i, uint32_t a, uint32_t b) { *reinterpret_cast<uint2*>(raw + 2 * i) = make_uint2(a, b); });
    consumers_sync();
#pragma unroll 1
    for (int hd = warp; hd < G + 2; hd += kStepWarps) {      // queries, key, value
      uint32_t lo = raw[hd * (D / 2) + lane], hi = raw[hd * (D / 2) + lane + 32];
      if (hd <= G) {
        float a0 = bf_lo(lo), a1 = bf_hi(lo), b0 = bf_lo(hi), b1 = bf_hi(hi);
        if (s.qk_norm) {
          const float rs = rsqrtf(warp_sum(a0 * a0 + a1 * a1 + b0 * b0 + b1 * b1) / (float)D + s.qk_eps);
          const uint32_t nlo = hd < G ? nw[0] : nw[2], nhi = hd < G ? nw[1] : nw[3];
          a0 = bf16_round(bf_lo(nlo) * bf16_round(a0 * rs));
          a1 = bf16_round(bf_hi(nlo) * bf16_round(a1 * rs));
          b0 = bf16_round(bf_lo(nhi) * bf16_round(b0 * rs));
          b1 = bf16_round(bf_hi(nhi) * bf16_round(b1 * rs));
        }
        lo = pack_bf16x2(bf16_round(a0 * cs.x) - bf16_round(b0 * sn.x), bf16_round(a1 * cs.y) - bf16_round(b1 * sn.y));
        hi = pack_bf16x2(bf16_round(b0 * cs.x) + bf16_round(a0 * sn.x), bf16_round(b1 * cs.y) + bf16_round(a1 * sn.y));
      }
      uint32_t* dst = hd < G ? qs + hd * kQLd : hd == G ? krow : vrow;
      dst[lane] = lo;
      dst[lane + 32] = hi;
    }
    consumers_sync();

    const int group = warp >> 2, wq = warp & 3, gid = lane >> 2, t4 = lane & 3;
    uint32_t q[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k][0] = gid < G ? qs[gid * kQLd + 8 * k + t4] : 0u;
      q[k][1] = gid < G ? qs[gid * kQLd + 8 * k + 4 + t4] : 0u;
    }
    float* gm = reinterpret_cast<float*>(base + lay.gm) + group * 32;
    float* wl = reinterpret_cast<float*>(base + lay.wl) + group * 40;
    uint32_t* ps = reinterpret_cast<uint32_t*>(base + lay.p) + group * 8 * kPLd;
    const uint32_t zero = smem_u32(vrow + D / 2);
    const float scale_log2 = 1.4426950408889634f * rsqrtf((float)D);
    const int lr = lane & 7, mi = lane >> 3;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = 0.f;
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory"); };
#pragma unroll 1
    for (int i = 0; i < pg.count; ++i, at.next()) {
      // every warp sees every page arrive (so that no phase of the ring passes unseen); one group of four works on it
      const bool there = wait.warp_wait(&sh.full[at.st], at.parity, 3, i);
      if ((i & (kGroups - 1)) == group) {      // all of a group's warps meet at its barriers, page or no page
        uint8_t* page = base + lay.ring + (there ? sh.start[at.st] : 0);
        const int valid = pos - (pg.first + i) * VDC_KV_PAGE;
        const bool tail = owner && i == pg.count - 1;
        if (tail && there && wq == 0) {
          // the new position's rows, here and in the cache
          const int r = pos % VDC_KV_PAGE, piece = lane & 15;
          const uint4 v = reinterpret_cast<const uint4*>(krow)[lane];
          *reinterpret_cast<uint4*>(page + (lane < 16 ? 0 : kPageBytes) + r * (D * 2) + ((piece ^ (r & 7)) << 4)) = v;
          const size_t row = (size_t)sh.new_row * (D * 2);
          const size_t pool = (size_t)layer * s.max_pages * s.n_kv * kPageBytes + (size_t)pg.h * kPageBytes;
          uint8_t* to = reinterpret_cast<uint8_t*>(lane < 16 ? s.kpool : s.vpool) + pool + row;
          if (!failed()) *reinterpret_cast<uint4*>(to + ((piece ^ (r & 7)) << 4)) = v;
        }
        if (tail) group_sync();
        const uint32_t kb = smem_u32(page), vb = kb + kPageBytes;
        // S^T = K Q^T: this warp's 16 positions on the tile's rows, the query heads on its columns
        float c[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
        const int pk = wq * 16 + lr + 8 * (mi & 1), hk = mi >> 1;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          uint32_t a[4], a2[4];
          ldsm_x4(a, kb + (uint32_t)(pk * 256 + (((2 * k + hk) ^ lr) << 4)));
          ldsm_x4(a2, kb + (uint32_t)(pk * 256 + (((2 * k + 2 + hk) ^ lr) << 4)));
          mma_16816(c, a[0], a[1], a[2], a[3], q[k][0], q[k][1]);
          mma_16816(c2, a2[0], a2[1], a2[2], a2[3], q[k + 1][0], q[k + 1][1]);
        }
        const int p0 = wq * 16 + gid;
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = p0 + 8 * (j >> 1) <= valid ? (c[j] + c2[j]) * scale_log2 : -INFINITY;
        float mx[2] = {fmaxf(e[0], e[2]), fmaxf(e[1], e[3])};
#pragma unroll
        for (int z = 4; z < 32; z <<= 1) {
          mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], z));
          mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], z));
        }
        if (gid == 0) *reinterpret_cast<float2*>(gm + wq * 8 + 2 * t4) = make_float2(mx[0], mx[1]);
        group_sync();
        float al[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float mn = m[j];
#pragma unroll
          for (int w = 0; w < 4; ++w) mn = fmaxf(mn, gm[w * 8 + 2 * t4 + j]);
          const bool none = mn == -INFINITY;
          // of exp2f's numbers exp2_ftz lacks those below 2^-126, which a row's sum (1 at least) cannot hold
          al[j] = none ? 1.f : exp2_ftz(m[j] - mn);
          e[j] = none ? 0.f : exp2_ftz(e[j] - mn);
          e[j + 2] = none ? 0.f : exp2_ftz(e[j + 2] - mn);
          m[j] = mn;
          l[j] = l[j] * al[j] + e[j] + e[j + 2];      // this warp's positions only
        }
        // probabilities enter P V rounded to bf16, as a bf16 attention module hands them over
        ps[gid * kPLd + wq * 8 + t4] = transpose8x8(pack_bf16x2(e[0], e[1]));
        ps[gid * kPLd + wq * 8 + 4 + t4] = transpose8x8(pack_bf16x2(e[2], e[3]));
        group_sync();
        // O^T = V^T P^T: 32 of the head's dims per warp, all positions of the page
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int j = 0; j < 4; ++j) o[d][j] *= al[j & 1];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int pv = k * 16 + lr + 8 * (mi >> 1), hv = mi & 1;
          const uint32_t vr = pv <= valid ? vb + (uint32_t)(pv * 256) : zero;
          const uint32_t b0 = ps[gid * kPLd + k * 8 + t4], b1 = ps[gid * kPLd + k * 8 + 4 + t4];
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            uint32_t va[4];
            ldsm_x4_trans(va, vr + (uint32_t)(((2 * (2 * wq + d) + hv) ^ lr) << 4));
            mma_16816(o[d], va[0], va[1], va[2], va[3], b0, b1);
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.empty[at.st]);
    }
#pragma unroll
    for (int z = 4; z < 32; z <<= 1) {
      l[0] += __shfl_xor_sync(0xffffffffu, l[0], z);
      l[1] += __shfl_xor_sync(0xffffffffu, l[1], z);
    }
    if (gid == 0) {
      *reinterpret_cast<float2*>(wl + wq * 8 + 2 * t4) = make_float2(l[0], l[1]);
      if (wq == 0) *reinterpret_cast<float2*>(wl + 32 + 2 * t4) = make_float2(m[0], m[1]);
    }
    float* po = part() + group * 8 * kOutLd;
#pragma unroll
    for (int d = 0; d < 2; ++d)
#pragma unroll
      for (int j = 0; j < 4; ++j) po[(2 * t4 + (j & 1)) * kOutLd + (2 * wq + d) * 16 + gid + 8 * (j >> 1)] = o[d][j];
    consumers_sync();
    if (failed()) return;

    // the groups' sums: two dims of a head per thread
#pragma unroll 1
    for (int t = tid; t < G * (D / 2); t += kStepThreads) {
      const int g = t / (D / 2), d2 = t % (D / 2);
      const float* w0 = reinterpret_cast<const float*>(base + lay.wl);
      float mm = -INFINITY;
#pragma unroll
      for (int k = 0; k < kGroups; ++k) mm = fmaxf(mm, w0[k * 40 + 32 + g]);
      float n0 = 0.f, n1 = 0.f, den = 0.f;
#pragma unroll
      for (int k = 0; k < kGroups; ++k) {
        const float mk = w0[k * 40 + 32 + g], wt = mk == -INFINITY ? 0.f : exp2_ftz(mk - mm);
        const float2 v = *reinterpret_cast<const float2*>(part() + (k * 8 + g) * kOutLd + 2 * d2);
        n0 = fmaf(wt, v.x, n0);
        n1 = fmaf(wt, v.y, n1);
        den = fmaf(wt, w0[k * 40 + g] + w0[k * 40 + 8 + g] + w0[k * 40 + 16 + g] + w0[k * 40 + 24 + g], den);
      }
      if (pg.live == 1) {
        const float inv = den > 0.f ? 1.f / den : 0.f;       // 0 where no score was a number
        put(out + (size_t)pg.h * G * (D / 2) + t, pack_bf16x2(n0 * inv, n1 * inv), tag_out);
      } else {
        const size_t u = (size_t)pg.h * s.n_splits + pg.split;
        put2(rec + (u * G * (D / 2) + t) * 2, __float_as_uint(n0), __float_as_uint(n1), tag_rec);
        if (d2 == 0) put2(ml + (u * G + g) * 2, __float_as_uint(mm), __float_as_uint(den), tag_rec);
      }
    }
    if (pg.live == 1) return;
    // Four of the head's dims at a time are shared by its units: a lane per split (of 8, 16 or 32 lanes), so that an SM's share is
    // one pass of the warps, as a rule.  Beyond 32 splits a lane takes every 32nd.  The first one by itself: a loop over all of
    // them lets the lanes drift apart while they poll (four 8B-shaped e4m3 layers 330 -> 368 us).
    const int fours = G * (D / 4), lo = sh.four0, hi = sh.four1;
    const int lg = pg.live <= 8 ? 3 : pg.live <= 16 ? 4 : 5, lanes = 1 << lg, mine = lane & (lanes - 1), step = 32 >> lg;
#pragma unroll 1
    for (int i0 = lo + warp * step; i0 < hi; i0 += kStepWarps * step) {
      const int i = i0 + (lane >> lg);
      float mk = -INFINITY, lk = 0.f;
      float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
      bool ok = true;
      auto take = [&](int sp, float4& n, float& mk, float& lk) {
        const size_t u = (size_t)pg.h * s.n_splits + sp;
        const uint64_t *rp = rec + (u * fours + i) * 4, *mp = ml + (u * G + i / (D / 4)) * 2;
        Two a = get2(rp), b = get2(rp + 2), z = get2(mp);
        uint64_t t0 = 0;
#pragma unroll 1
        for (uint32_t it = 1; !(a.are(tag_rec) && b.are(tag_rec) && z.are(tag_rec)); ++it) {
          if ((it & 63u) == 0 && !again(rp, it, t0)) {
            ok = false;
            return;
          }
          a = get2(rp);
          b = get2(rp + 2);
          z = get2(mp);
        }
        n = make_float4(__uint_as_float((uint32_t)a.a), __uint_as_float((uint32_t)a.b), __uint_as_float((uint32_t)b.a), __uint_as_float((uint32_t)b.b));
        mk = __uint_as_float((uint32_t)z.a);
        lk = __uint_as_float((uint32_t)z.b);
      };
      if (i < hi && mine < pg.live) take(mine, n, mk, lk);
#pragma unroll 1
      for (int sp = mine + 32; sp - mine < pg.live; sp += 32) {
        if (sp >= pg.live || !ok) continue;
        float4 n1;
        float m1, l1;
        take(sp, n1, m1, l1);
        if (!ok) continue;
        const float m2 = fmaxf(mk, m1), w0 = mk == -INFINITY ? 0.f : exp2_ftz(mk - m2), w1 = m1 == -INFINITY ? 0.f : exp2_ftz(m1 - m2);
        n = make_float4(fmaf(w0, n.x, w1 * n1.x), fmaf(w0, n.y, w1 * n1.y), fmaf(w0, n.z, w1 * n1.z), fmaf(w0, n.w, w1 * n1.w));
        lk = fmaf(w0, lk, w1 * l1);
        mk = m2;
      }
      if (!__all_sync(0xffffffffu, ok)) break;
      float mm = mk;
#pragma unroll 1
      for (int z = lanes >> 1; z > 0; z >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, z));
      const float wt = mk == -INFINITY ? 0.f : exp2_ftz(mk - mm);
      n = make_float4(wt * n.x, wt * n.y, wt * n.z, wt * n.w);
      float den = wt * lk;
#pragma unroll 1
      for (int z = lanes >> 1; z > 0; z >>= 1) {
        n.x += __shfl_xor_sync(0xffffffffu, n.x, z);
        n.y += __shfl_xor_sync(0xffffffffu, n.y, z);
        n.z += __shfl_xor_sync(0xffffffffu, n.z, z);
        n.w += __shfl_xor_sync(0xffffffffu, n.w, z);
        den += __shfl_xor_sync(0xffffffffu, den, z);
      }
      const float inv = den > 0.f ? 1.f / den : 0.f;
      if (mine == 0 && i < hi) put2(out + ((size_t)pg.h * fours + i) * 2, pack_bf16x2(n.x * inv, n.y * inv), pack_bf16x2(n.z * inv, n.w * inv), tag_out);
    }
  }

  // The router's logits from their entries; every SM selects the experts for itself and tells its producer.
  __device__ __forceinline__ void route(const uint64_t* buf, uint32_t tag) {
    const int E = s.n_experts;
    float* lg = reinterpret_cast<float*>(base + lay.route);
    int* ids = reinterpret_cast<int*>(lg + kMaxExperts);
    float* weights = reinterpret_cast<float*>(ids + kMaxTopK);
    collect<1>(buf, 2 * E, tag, [&](int i, uint32_t a, uint32_t b) {
      lg[2 * i] = __uint_as_float(a);
      lg[2 * i + 1] = __uint_as_float(b);
    });
    consumers_sync();
    if (warp == 0) {
      constexpr int kMost = kMaxExperts / 32;
      float v[kMost], mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < kMost; ++j) {
        v[j] = lane + 32 * j < E ? lg[lane + 32 * j] : -INFINITY;
        mx = fmaxf(mx, v[j]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      // One logit without a number and the softmax's sum has none, nor has any expert's weight, whichever experts are chosen.
      bool none = false;
#pragma unroll
      for (int j = 0; j < kMost; ++j) {
        v[j] = lane + 32 * j < E ? __expf(v[j] - mx) : -1.f;
        none |= v[j] != v[j];
      }
      // The largest, k times over; of equal ones the lowest number.  Their weights are renormalised, so the softmax's own sum does
      // not matter otherwise.
      float all = __any_sync(0xffffffffu, none) ? NAN : 0.f, mine = 0.f;
      int id = 0;
#pragma unroll 1
      for (int k = 0; k < s.top_k; ++k) {
        float bv = -1.f;
        int bi = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < kMost; ++j)
          if (v[j] > bv) {
            bv = v[j];
            bi = lane + 32 * j;
          }
        // a number that was not chosen yet is not negative, so that its bits order it as an integer
        const int top = __reduce_max_sync(0xffffffffu, __float_as_int(bv));
        // logits without a number select nothing: any expert will do
        bi = min((int)__reduce_min_sync(0xffffffffu, __float_as_int(bv) == top ? (unsigned)bi : 0x7fffffffu), E - 1);
#pragma unroll
        for (int j = 0; j < kMost; ++j)
          if (bi == lane + 32 * j) v[j] = -1.f;
        all += __int_as_float(top);
        if (lane == k) {
          mine = __int_as_float(top);
          id = bi;
        }
      }
      if (lane < s.top_k) {
        ids[lane] = id;
        weights[lane] = bf16_round(mine / all);
        if (sm == 0) {
          reinterpret_cast<int*>(s.route)[lane] = id;
          reinterpret_cast<float*>(s.route)[16 + lane] = bf16_round(mine / all);
        }
      }
      __syncwarp();
      if (lane == 0 && !failed()) mbar_arrive(&sh.routed);
    }
    consumers_sync();
  }
};

// ------------------------------------------------------------------------- //
// the step
// ------------------------------------------------------------------------- //
template <int kFmt, bool kExperts>
__global__ void __launch_bounds__(kStepThreads + 32, 1) decode_step(const __grid_constant__ StepArgs args, vdc_status* status,
                                                                    uint64_t timeout_ns) {
  extern __shared__ uint8_t dyn[];
  __shared__ StepShared sh;
  const vdc_step& s = args.s;
  const StepLayout& lay = args.lay;
  const StepWork& wk = args.wk;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sm = blockIdx.x, sms = gridDim.x;
  uint8_t* base = aligned128(dyn);
  const Waiter wait{&sh.fail, status, timeout_ns, VDC_STEP_KIND};
  constexpr int D = VDC_HEAD_DIM;
  if (tid < kStages) {
    const Deal& d = args.deal[tid];
    const int i = sm < d.more ? 0 : 1;
    sh.plan[tid] = Plan{(sm * d.each + min(sm, d.more)) * d.q, (d.each + 1 - i) * d.q, d.per, d.units, d.lt[i], d.lk[i], d.slice[i], d.most[i]};
    if (kExperts && tid == kGateUp) {
      sh.slot0 = sh.plan[tid].r0 / (2 * s.ffn);
      sh.head = (sh.slot0 + 1) * 2 * s.ffn - sh.plan[tid].r0;
    }
  }
  if (tid == 0) {
    for (int i = 0; i < kItems; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], kStepWarps);
    }
    mbar_init(&sh.routed, 1);
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 64 && tid < 64 + D / 2) reinterpret_cast<uint32_t*>(base + lay.rows)[D + tid - 64] = 0u;     // a value row of zeros
  grid_dep_wait();
  grid_dep_launch();
  // Read before the error is looked for: in a launch that fails, SM 0 counts the launch behind the error.  An SM that starts late
  // and took the number from there would leave entries that the next launch takes for its own.
  const uint32_t launches = (uint32_t)ld_acquire_gpu(reinterpret_cast<const int*>(s.work));
  const int* state = reinterpret_cast<const int*>(s.state);
  const int aborted = ld_relaxed_gpu(&status->abort);
  int id = 0;
  bool wrong = false;
  if (tid == 0) {
    const int pos = ld_relaxed_gpu(state + VDC_ST_POS), token = ld_relaxed_gpu(state + VDC_ST_TOKEN);
    sh.new_row = ld_relaxed_gpu(state + VDC_ST_NEWROW);
    sh.pos = pos;
    sh.token = token < 0 || token >= s.vocab ? 0 : token;
    wrong = sh.token != token;
    id = token;
    const Pages pg = pages_of(s, pos, sm);
    sh.pages = pg;
    sh.four0 = s.group * (D / 4) * pg.split / pg.live;
    sh.four1 = s.group * (D / 4) * (pg.split + 1) / pg.live;
  }
  if (__syncthreads_or(aborted)) {      // behind an unread error nothing runs
    if (sm == 0 && tid == 0) red_release_gpu_add(reinterpret_cast<int*>(s.work), 1);
    return;
  }
  if (wrong && sm == 0) report(status, VDC_ERR_TOKEN, VDC_STEP_KIND, 0, 0, id);

  const int H = s.hidden, F = s.ffn, Q = args.q_width, QKV = args.qkv_width, L = s.n_layers, E = kExperts ? s.n_experts : 0;
  const int slots = E ? s.top_k : 1;
  const int rbH = row_bytes(kFmt, H), rbQ = row_bytes(kFmt, Q), rbF = row_bytes(kFmt, F);
  int* ids = reinterpret_cast<int*>(base + lay.route + kMaxExperts * 4);
  float* weights = reinterpret_cast<float*>(ids + kMaxTopK);

  if (warp == kStepWarps) {
    {
      fence_proxy_async();      // the cache rows of the steps before were written with ordinary stores
      Producer p{sh, wait, base + lay.ring, lay.total - lay.ring, lane};
      const int* table = state + VDC_ST_PAGETABLE;
      const Pages pg = sh.pages;
      // stage after stage; a stage is one run of rows or several (experts), the attention one run per page
      int l = 0, stage = kQkv, sub = 0;
#pragma unroll 1
      while (p.ok) {
        asm volatile("" : "+r"(stage), "+r"(sub));
        const uint8_t *src = nullptr, *second = nullptr;
        int rb = rbH, r0 = sh.plan[stage].r0, rows = sh.plan[stage].n;
        bool more = false;                     // the stage goes on
        if (stage == kQkv) {
          src = reinterpret_cast<const uint8_t*>(s.wqkv) + (size_t)l * QKV * rbH;
          if (sub > 0) {                       // page sub - 1
            rows = 0;
            if (sub <= pg.count) {
              const size_t off = ((size_t)l * s.max_pages + ld_relaxed_gpu(table + pg.first + sub - 1)) * s.n_kv * kPageBytes + (size_t)pg.h * kPageBytes;
              src = reinterpret_cast<const uint8_t*>(s.kpool) + off;
              second = reinterpret_cast<const uint8_t*>(s.vpool) + off;
              rows = 1;
              r0 = 0;
              rb = kPageBytes;
            }
          }
          more = sub < pg.count;
        } else if (stage == kOut) {
          rb = rbQ;
          src = reinterpret_cast<const uint8_t*>(s.wo) + (size_t)l * H * rbQ;
        } else if (stage == kRouter) {
          src = reinterpret_cast<const uint8_t*>(s.router) + (size_t)l * E * rbH;
        } else if (stage == kGateUp) {
          src = reinterpret_cast<const uint8_t*>(s.wgu);
          size_t first = (size_t)l * 2 * F;
          if (E) {                             // a slot's rows end where the next slot's begin
            if (sub == 0 && (rows || sh.plan[kDown].n) && !(p.ok = wait.warp_wait(&sh.routed, (uint32_t)l & 1u, 0, l))) break;
            const int end = r0 + rows, slot = sh.slot0 + sub;
            r0 = max(r0, slot * 2 * F);
            rows = min(end, (slot + 1) * 2 * F) - r0;
            more = r0 + rows < end;
            first = rows > 0 ? ((size_t)l * E + ids[slot]) * 2 * F : 0;
            r0 -= slot * 2 * F;
          }
          src += first * rbH;
        } else if (stage == kDown) {
          rb = rbF;
          more = sub + 1 < slots;
          src = reinterpret_cast<const uint8_t*>(s.wd) + (E ? ((size_t)l * E + ids[sub]) * H : (size_t)l * H) * rbF;
          if (!rows) more = false;
        } else {
          rb = H * 2;
          src = reinterpret_cast<const uint8_t*>(s.lm_head);
        }
        const int slice = kExperts || second ? 0 : sh.plan[stage].slice, units = sh.plan[stage].units, per = second ? 1 : sh.plan[stage].per;
        src += (size_t)r0 * rb;
        if (slice) {
#pragma unroll 1
          for (int g = 0; g < rows && p.ok; g += 4, src += 4 * rb)
#pragma unroll 1
            for (int u0 = 0; u0 < units; u0 += slice) p.item(src + lane * rb + u0 * 512, min(4, rows - g), min(slice, units - u0) * 512);
        } else {
#pragma unroll 1
          for (int g = 0; g < rows && p.ok; g += per) p.item(second && lane ? second : src + (size_t)g * rb, second ? 2 : 1, min(per, rows - g) * rb);
        }
        if (stage == kVocab) break;
        ++sub;
        if (more) continue;
        sub = 0;
        if (stage == kDown) stage = ++l == L ? kVocab : kQkv;
        else stage = stage == kOut && !E ? kGateUp : stage + 1;
      }
    }
    __syncwarp();
  } else {
    uint64_t* work = reinterpret_cast<uint64_t*>(s.work);
    const uint32_t tag0 = (launches * (uint32_t)(L + 1) + 1u) * 8u;
    Consumer c{args, s, lay, sh, wait, base, tid, warp, lane, sm};
    // a residual row pair: this SM's rows of a projection added to the hidden state it has in shared memory
    auto residual = [&](int pair, float y0, float y1, uint64_t* out, uint32_t tag) {
      const uint32_t h = c.hs()[pair];
      put(out + pair, pack_bf16x2(bf_lo(h) + bf16_round(y0), bf_hi(h) + bf16_round(y1)), tag);
    };
    // a division: an approximate reciprocal has no denormal results, and 1 / (1 + exp(88)) is one (width 512 46.2 us with it, 47.1
    // so; eight 8B-shaped layers 799.7 and 801)
    auto silu = [&](float g, float u) {
      g = bf16_round(g);
      return bf16_round(g / (1.f + __expf(-g))) * bf16_round(u);
    };
    auto keep_hidden = [&](uint64_t to) {        // SM 0: the hidden state as it came in, for whoever asks
      if (sm == 0 && to && !c.failed())
#pragma unroll 1
        for (int i = tid; i < H / 2; i += kStepThreads) reinterpret_cast<uint32_t*>(to)[i] = c.hs()[i];
    };
    float best;
    int best_row;
    // One loop over the layers' stages, with the vocabulary projection as the first stage behind the last layer: each piece of
    // code is there once, since what falls out of the instruction caches between two stages costs as much as the stage.
#pragma unroll 1
    for (int l = 0, stage = kQkv;;) {
      asm volatile("" : "+r"(stage), "+r"(l));      // the compiler would otherwise make a copy of the loop for every stage
      const uint32_t tag = tag0 + (uint32_t)l * 8u;
      const bool lm = l == L;
      const int K = stage == kOut ? Q : stage == kDown ? F : H;
      const Plan r = sh.plan[lm ? kVocab : stage];
      c.split(r);
      // the scales of this thread's first rows come from HBM while the inputs are waited for
      const float* scales = nullptr;
      const float2* mine = reinterpret_cast<const float2*>(base + lay.scales + tid * 16);
      if (kFmt != 0 && !lm) {
        const uint64_t of = stage == kQkv ? s.s_qkv : stage == kOut ? s.s_o : stage == kGateUp ? s.s_gu : s.s_d;
        scales = reinterpret_cast<const float*>(of) + (size_t)l * (stage == kQkv ? QKV : stage == kGateUp ? 2 * F : H) + r.r0;
        const int each = stage == kGateUp ? 4 : 2;
        if (tid < r.n / each) {
          copy8_async(base + lay.scales + tid * 16, reinterpret_cast<uint64_t>(scales + tid * each));
          if (each == 4) copy8_async(base + lay.scales + tid * 16 + 8, reinterpret_cast<uint64_t>(scales + tid * 4 + 2));
        }
      }
      auto scaled2 = [&](int i) {         // rows 2i, 2i + 1 of this SM
        float2 v = c.sum2(2 * i);
        if (kFmt != 0) {
          const float2 k = i == tid ? *mine : __ldg(reinterpret_cast<const float2*>(scales) + i);
          v.x *= k.x; v.y *= k.y;
        }
        return v;
      };
      // ---- inputs
      bool skip = false;
      if (stage == kQkv || stage == (E ? kRouter : kGateUp)) {
        // whoever has rows of this stage, or of the one that adds to the hidden state, reads it
        skip = !r.n && (lm ? sm != 0 : !sh.plan[kOut].n && (stage == kQkv || !sh.plan[kGateUp].n));
        if (!skip) {
          const uint64_t w = lm ? s.norm_w : (stage == kQkv ? s.ln1 : s.ln2) + (size_t)l * H * 2;
          c.template hidden<kFmt, kExperts ? 4 : 2>(work + wk.h + (stage == kQkv ? H / 2 : 0), stage == kQkv ? tag - 8u + 5u : tag + 4u, l == 0 && stage == kQkv ? reinterpret_cast<const uint8_t*>(s.embed) + (size_t)sh.token * H * 2 : nullptr, w, lm);
          if (stage == kQkv && l > 0 && s.taps) keep_hidden(s.taps + (size_t)(l - 1) * H * 2);
          if (lm) keep_hidden(s.hidden_out);
        }
      } else if (stage == kOut || stage == kDown) {
        skip = !r.n;
        if (!skip) {
          c.template collect<kExperts ? 7 : 4>(work + (stage == kOut ? wk.attn : wk.act), stage == kOut ? Q : F * slots, tag + (stage == kOut ? 3u : 6u),
                    [&](int i, uint32_t a, uint32_t b) { c.template set_input<kFmt>(i, a, b, false); });
          consumers_sync();
        }
      } else if (r.n || sh.plan[kDown].n) {      // kGateUp behind a router: its inputs are there, the experts are not
        c.route(work + wk.router, tag + 7u);
      }
      if (lm) {
        best = -INFINITY;
        best_row = 0x7fffffff;
      }
      // ---- rows, as many at a time as their partial sums have room for
#pragma unroll 1
      for (int r0 = 0; r0 < r.n && !skip; r0 += r.most) {
        const int n = min(r.most, r.n - r0);
        if (lm && kFmt != 0) {
          c.template rows<0, false>(K, n, c.x(), 0);
        } else {
          // experts: a slot's gate/up rows end where the next slot's begin; every slot's down rows have inputs of their own
          const int segs = E && stage == kDown ? slots : 1;
#pragma unroll 1
          for (int e = 0, done = 0; E && stage == kGateUp ? done < n : e < segs; ++e) {
            const int take = E && stage == kGateUp ? min(n - done, done ? 2 * F : sh.head) : n;
            c.template rows<kFmt, kExperts>(K, take, c.x() + (segs > 1 ? (size_t)e * F * 2 : 0), segs > 1 ? e * n : done);
            done += take;
          }
        }
        if (kFmt != 0) copies_wait();
        consumers_sync();
        if (!c.failed()) {
          if (lm) {
#pragma unroll 1
            for (int i = tid; i < n / 2; i += kStepThreads) {
              const int rr = r.r0 + r0 + 2 * i;
              const float2 y = c.sum2(2 * i);
              const uint32_t v = pack_bf16x2(y.x, y.y);
              reinterpret_cast<uint32_t*>(s.logits)[rr >> 1] = v;
              if (bf_lo(v) > best) {
                best = bf_lo(v);
                best_row = rr;
              }
              if (bf_hi(v) > best) {
                best = bf_hi(v);
                best_row = rr + 1;
              }
            }
          } else if (stage == kQkv) {
#pragma unroll 1
            for (int i = tid; i < n / 2; i += kStepThreads) {
              const float2 y = scaled2(i);
              put(work + wk.qkv + (r.r0 >> 1) + i, pack_bf16x2(y.x, y.y), tag + 1u);
            }
          } else if (stage == kRouter) {
            if (tid < n) put(work + wk.router + r.r0 + tid, __float_as_uint(c.sum1(tid)), tag + 7u);
          } else if (stage == kGateUp) {
#pragma unroll 1
            for (int i = tid; i < n / 4; i += kStepThreads) {
              float4 y = c.sum4(4 * i);
              if (kFmt) {
                const float4 k = i == tid ? *reinterpret_cast<const float4*>(mine) : __ldg(reinterpret_cast<const float4*>(scales) + i);
                y.x *= k.x; y.y *= k.y; y.z *= k.z; y.w *= k.w;
              }
              put(work + wk.act + (r.r0 >> 2) + i, pack_bf16x2(silu(y.x, y.y), silu(y.z, y.w)), tag + 6u);
            }
          } else {
#pragma unroll 1
            for (int i = tid; i < n / 2; i += kStepThreads) {
              float2 y = make_float2(0.f, 0.f);
              if (E && stage == kDown) {
#pragma unroll 1
                for (int e = 0; e < slots; ++e) {
                  const float2 v = c.sum2(e * n + 2 * i);
                  y.x = fmaf(weights[e], bf16_round(v.x), y.x);
                  y.y = fmaf(weights[e], bf16_round(v.y), y.y);
                }
              } else {
                y = scaled2(i);
              }
              residual((r.r0 >> 1) + i, y.x, y.y, work + wk.h + (stage == kDown ? H / 2 : 0), tag + (stage == kDown ? 5u : 4u));
            }
          }
        }
        if (lm) consumers_sync();
      }
      if (lm) break;
      if (stage == kQkv && sh.pages.count > 0)
        c.attention(l, sh.pos, sh.pages, work + wk.qkv, work + wk.rec, work + wk.ml, work + wk.attn, tag + 1u, tag + 2u, tag + 3u);
      if (stage == kDown) ++l;
      stage = stage == kDown ? kQkv : stage == kOut ? (E ? kRouter : kGateUp) : stage + 1;
    }
    const uint32_t tag = tag0 + (uint32_t)L * 8u;
    if (s.taps) keep_hidden(s.taps + (size_t)(L - 1) * H * 2);
    auto better = [](float v, int r, float& bv, int& br) {      // the lowest row wins ties
      if (v > bv || (v == bv && r < br)) {
        bv = v;
        br = r;
      }
    };
    auto warp_best = [&](float& bv, int& br) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int orow = __shfl_xor_sync(0xffffffffu, br, o);
        better(ov, orow, bv, br);
      }
    };
    warp_best(best, best_row);
    if (lane == 0) {
      sh.best[warp] = best;
      sh.best_row[warp] = best_row;
    }
    consumers_sync();
    if (warp == 0) {
      best = lane < kStepWarps ? sh.best[lane] : -INFINITY;
      best_row = lane < kStepWarps ? sh.best_row[lane] : 0x7fffffff;
      warp_best(best, best_row);
      if (lane == 0 && !c.failed()) put2(work + wk.best + 2 * sm, __float_as_uint(best), (uint32_t)best_row, tag + 1u);
      if (sm == 0) {
        best = -INFINITY;
        best_row = 0x7fffffff;
        bool ok = true;
#pragma unroll 1
        for (int i = lane; i < sms && ok; i += 32) {
          Two v = get2(work + wk.best + 2 * i);
          ok = c.poll2(work + wk.best + 2 * i, tag + 1u, v);
          if (ok) better(__uint_as_float((uint32_t)v.a), (int)(uint32_t)v.b, best, best_row);
        }
        warp_best(best, best_row);
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) {
          red_release_gpu_add(reinterpret_cast<int*>(s.work), 1);      // the next launch's tags are others, whatever became of this one
          int* st = reinterpret_cast<int*>(s.state);
          if (ok && best_row == 0x7fffffff) {         // no logit is a number: no next token, the state stays
            report(status, VDC_ERR_TOKEN, VDC_STEP_KIND, 1, 0, -1);
          } else if (ok && !c.failed() && !ld_relaxed_gpu(&status->abort)) {
            const int step = st[VDC_ST_STEP], next = sh.pos + 1, page = next / VDC_KV_PAGE;
            reinterpret_cast<int*>(s.log)[step] = best_row;
            st[VDC_ST_TOKEN] = best_row;
            st[VDC_ST_STEP] = step + 1;
            st[VDC_ST_POS] = next;
            st[VDC_ST_NPAGES] = page + 1;
            if (page < st[VDC_ST_MAXPAGES])
              st[VDC_ST_NEWROW] = st[VDC_ST_PAGETABLE + page] * VDC_KV_PAGE * st[VDC_ST_NKVH] + next % VDC_KV_PAGE;
            else
              st[VDC_ST_ERR] = 1;      // out of KV pages: the host must not launch another step
          }
        }
      }
    }
  }
  wait.drain();
}

}  // namespace vdc

// 0 when the kernel can run this step, otherwise why not.
extern "C" const char* vdc_step_refuses(const vdc_step* s, bool pointers) {
  using namespace vdc;
  auto al16 = [](uint64_t p) { return p != 0 && (p & 15) == 0; };
  if (s->num_sms < 1 || s->num_sms > VDC_MAX_SMS || s->n_layers < 1 || s->wfmt < 0 || s->wfmt > 2) return "step: bad shape";
  if ((s->group != 4 && s->group != 8) || s->n_kv < 1 || s->max_pages < 1) return "step: bad heads or pages";
  if (s->n_splits < 1 || s->n_splits > s->num_sms / s->n_kv) return "step: more attention units than SMs";
  const int u = unit_of(s->wfmt), Q = s->n_kv * s->group * VDC_HEAD_DIM;
  if (s->hidden < 512 && s->hidden != 256) return "step: hidden too small";
  if (s->hidden > 8192 || s->hidden % u || s->hidden % 256 || s->ffn < u || s->ffn % u || Q % u || s->vocab < 2 || s->vocab % 2)
    return "step: widths not supported";
  if (row_bytes(0, s->hidden) > kItemBytes || row_bytes(s->wfmt, s->ffn) > kItemBytes || row_bytes(s->wfmt, Q) > kItemBytes)
    return "step: a weight row is longer than a copy";
  if (s->n_experts && (s->wfmt || s->n_experts > kMaxExperts || s->n_experts % 2 || s->top_k < 1 || s->top_k > kMaxTopK || s->top_k > s->n_experts))
    return "step: experts not supported";
  const StepLayout l = step_layout(*s);
  // three copies, or, where weights have scales, what those leave of them: the ring needs room for one
  if (l.total - l.ring + (s->wfmt ? kScaleBytes : 0) < 3 * kItemBytes) return "step: no room for the ring";
  // the partial sums of an SM's rows: of those SMs with the most, and of those with a unit less
  auto fits = [&](int rows, int q, int K, int slots) {
    const int most = share_of(rows, q, 0, s->num_sms).n;
    for (int n = most; n > 0 && n >= most - q; n -= q)
      if (n * slots > kPartFloats / split_of(s->wfmt, s->n_experts != 0, false, K, n * slots).kw) return false;
    return true;
  };
  const int k = s->n_experts ? s->top_k : 1;
  if (!fits(Q + 2 * s->n_kv * VDC_HEAD_DIM, 2, s->hidden, 1) || !fits(s->hidden, 2, Q, 1) ||
      !fits(2 * s->ffn * k, 4, s->hidden, 1) || !fits(s->hidden, 2, s->ffn, k))
    return "step: more rows per SM than partial sums have room for";
  if (!pointers) return nullptr;
  if (!al16(s->embed) || !al16(s->lm_head) || !al16(s->norm_w) || !al16(s->ln1) || !al16(s->ln2) || !al16(s->wqkv) || !al16(s->wo) ||
      !al16(s->wgu) || !al16(s->wd) || !al16(s->kpool) || !al16(s->vpool) || !al16(s->rope) || !al16(s->logits) || !al16(s->hidden_out) ||
      !al16(s->work) || !s->state || (s->state & 3) || !s->log || (s->log & 3) || (s->taps & 15) || (s->qk_norm & 15))
    return "step: null or misaligned pointer";
  if (s->wfmt && (!al16(s->s_qkv) || !al16(s->s_o) || !al16(s->s_gu) || !al16(s->s_d))) return "step: null or misaligned scales";
  if (s->n_experts && (!al16(s->router) || !al16(s->route))) return "step: null or misaligned router";
  return nullptr;
}

extern "C" long long vdc_step_words(const vdc_step* s) { return (long long)vdc::step_work(*s).words; }

extern "C" cudaError_t vdc_step_prepare() {
  const void* fs[] = {(const void*)vdc::decode_step<0, false>, (const void*)vdc::decode_step<0, true>,
                      (const void*)vdc::decode_step<1, false>, (const void*)vdc::decode_step<2, false>};
  for (const void* f : fs)
    if (cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, vdc::kStepSmem)) return e;
  return cudaSuccess;
}

extern "C" cudaError_t vdc_step_launch(const vdc_step* s, vdc_status* status, uint64_t timeout_ns, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)s->num_sms);
  cfg.blockDim = dim3(vdc::kStepThreads + 32);
  cfg.dynamicSmemBytes = vdc::kStepSmem;
  auto f = s->n_experts ? vdc::decode_step<0, true> : s->wfmt == 0 ? vdc::decode_step<0, false>
           : s->wfmt == 1 ? vdc::decode_step<1, false> : vdc::decode_step<2, false>;
  vdc::StepArgs args{*s, vdc::step_layout(*s), vdc::step_work(*s), {}, 1.f / (float)s->hidden, s->n_kv * s->group * VDC_HEAD_DIM, s->n_kv * (s->group + 2) * VDC_HEAD_DIM};
  for (int i = 0; i < vdc::kStages; ++i) args.deal[i] = vdc::deal_of(*s, i);
  return cudaLaunchKernelEx(&cfg, f, args, status, timeout_ns);
}

// Wide stages: a prompt's rows through a layer together (up to VDC_WIDE_ROWS of them), where the stage kernels take 128.
//
// What bounds a prompt in chunks of 128 rows is the weights: a pass over two Llama-3.1-8B-shaped layers reads 0.87 GB, 133 us
// at the copy rate, for 128 rows of arithmetic that the tensor cores finish in 70.  With all rows behind one pass the weights
// are read once and the tensor cores are the bound.
//
// Rows lie in sub-matrices of 128 (the accumulator's lanes), each k-chunk-major like a stage's rows.  A projection leaves
// fp32 sums [K-split][columns / 4][rows][4] (consecutive rows side by side, so that a warp's stores are contiguous), or
// SiLU products; what a bf16 module does behind it (heads, residual add and norm) is a small kernel of its own, which also
// adds the splits up in order: no atomics, the same bits every time.
//
// Measured (B200): two such layers and a small vocabulary, 2048 tokens 5.1 -> 2.2 ms, 77 tokens (two chunks of 64 before)
// 667 -> 465 us.  Gate/up of 2048 rows 352 us (1.37 PFLOP/s; cuBLAS 331), down 166 us (1.45; 155).  A prompt's large projections of
// up to 128 rows are stages of the batched step (csrc/stage_kernels.cu); which, prefill.py decides.
#include "mk_stage.cuh"

namespace vdc {

constexpr int kKc = 64;                 // inputs per chunk
constexpr int kBlk = VDC_STAGE_BLOCK;   // rows of a block of packed weights
constexpr int kWideRing = 8;
constexpr int kWideSmem = 224 * 1024;   // one CTA per SM: a tile's operands are read from L2, and larger tiles read less
constexpr int kWideN = 256;             // columns of an accumulator: two of them fill tensor memory
constexpr int kSub = 128 * kKc * 2;     // bytes of a chunk of 128 rows

// Warps: four producers, one that issues the MMAs, sixteen workers (epilogue; widening of quantised weights).
constexpr int kWideProducers = 4, kWideWorkers = 16, kWideThreads = 32 * (kWideProducers + 1 + kWideWorkers);

struct WideShared {
  uint64_t full[kWideRing], empty[kWideRing], ready[kWideRing], stg_empty[2];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem;
  volatile int fail;
};

// Header of the block a prompt's stages read instead of per-row state: first position, rows, then the page table.
__device__ __forceinline__ int wide_first(const vdc_stage& s) { return ld_relaxed_gpu(reinterpret_cast<const int*>(s.state) + VDC_WIDE_POS); }
__device__ __forceinline__ int wide_rows(const vdc_stage& s) { return ld_relaxed_gpu(reinterpret_cast<const int*>(s.state) + VDC_WIDE_N); }

__host__ __device__ constexpr int wide_stage_bytes(int wfmt, int subs, int n) {
  return subs * kSub + (chunk_bytes(wfmt, n) + 127) / 128 * 128;
}
__host__ __device__ inline int wide_ring(int wfmt, int subs, int n) {
  const int r = (kWideSmem - 128 - (wfmt ? 2 * n * kKc * 2 : 0)) / wide_stage_bytes(wfmt, subs, n);
  return r < kWideRing ? r : kWideRing;
}

struct WideTile {
  int m, n0, N, c0, n_ch, subs, split;
};
// The row tiles of one column tile are neighbours: they run at the same time and read its weights from HBM once.
__device__ __forceinline__ WideTile wide_tile(const vdc_stage& s, int i) {
  WideTile t;
  const int all = s.Bpad / 128, per = s.group, m_tiles = (all + per - 1) / per, chunks = s.K / kKc;
  t.m = i % m_tiles;
  t.split = i / m_tiles % s.splits;
  t.n0 = i / m_tiles / s.splits * s.n_kv;
  t.N = min(s.n_kv, s.M - t.n0);
  t.c0 = chunks * t.split / s.splits;
  t.n_ch = chunks * (t.split + 1) / s.splits - t.c0;
  t.subs = min(per, all - t.m * per);
  return t;
}

// Projection of s.Bpad rows: tiles of s.group sub-matrices of rows (one or two) times s.n_kv weight rows, K shared by s.splits
// tiles.  One CTA per SM walks its tiles; the producer fills the ring for the next tile while the epilogue empties the
// accumulators of this one (two of 256 columns: the tile's two sub-matrices, or this tile's and the next one's).
template <int kFmt>
__global__ void __launch_bounds__(kWideThreads, 1) wide_gemm(const __grid_constant__ vdc_stage s, int n_tiles, vdc_status* status,
                                                                 uint64_t timeout_ns) {
  extern __shared__ uint8_t dyn[];
  __shared__ WideShared sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per = s.group, NT = s.n_kv;
  const int stage_bytes = wide_stage_bytes(kFmt, per, NT), n_ring = wide_ring(kFmt, per, NT);
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn) + 127) & ~(uintptr_t)127);
  uint8_t* staging = ring + n_ring * stage_bytes;
  const Waiter wait{&sh.fail, status, timeout_ns, s.kind};

  if (warp == kWideProducers) tmem_alloc(&sh.tmem, 2 * kWideN);
  if (tid == 0) {
    for (int i = 0; i < kWideRing; ++i) {
      mbar_init(&sh.full[i], 1);
      // the MMAs have read it; and the team that does not widen it has seen it come (the one that does has, for them)
      mbar_init(&sh.empty[i], kFmt != 0 ? 1 + kWideWorkers / 2 : 1);
      mbar_init(&sh.ready[i], kWideWorkers / 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.stg_empty[i], 1);
      mbar_init(&sh.acc_full[i], 1);
      mbar_init(&sh.acc_empty[i], kWideWorkers / per);
    }
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;

  if (warp < kWideProducers) {
    // A chunk of a tile's weights is cut from at most three blocks of packed rows: per block one piece per eight (bf16) or
    // sixteen inputs, NVFP4 one more for the scales.  Lane i of the producers copies piece i of the chunk, the last two lanes
    // the rows.  Four warps, because a warp's lanes issue their copies one after another (one warp: gate/up of 2048 rows 507 us
    // instead of 420).
    constexpr int kPieces = kFmt == 1 ? 4 : 8;
    const int item = lane * kWideProducers + warp;
    bool ok = true;
    RingAt at_ring{n_ring};
    for (int i = blockIdx.x, it = 0; i < n_tiles && ok; i += gridDim.x) {
      const WideTile t = wide_tile(s, i);
      const int seg = item / kPieces, piece = item % kPieces, blk = t.n0 / kBlk + seg, Nb = min(kBlk, s.M - blk * kBlk);
      const int lo = max(t.n0, blk * kBlk), rows = min(t.n0 + t.N, blk * kBlk + Nb) - lo, at = lo - blk * kBlk, to = lo - t.n0;
      uint32_t bytes = 0, dst = 0;
      const uint8_t* src = nullptr;
      if (item < 3 * kPieces && rows > 0) {
        const uint8_t* base = reinterpret_cast<const uint8_t*>(s.w) + (size_t)blk * kBlk * s.K * (kFmt == 0 ? 32 : kFmt == 1 ? 16 : 9) / 16 +
                              (size_t)t.c0 * chunk_bytes(kFmt, Nb);
        if (kFmt == 2) {
          const int g = piece >> 1, sc = piece & 1;
          src = base + g * 9 * Nb + (sc ? 8 * Nb + at : 8 * at);
          dst = (uint32_t)(g * 9 * t.N + (sc ? 8 * t.N + to : 8 * to));
          bytes = (uint32_t)(sc ? rows : 8 * rows);
        } else {
          src = base + (piece * Nb + at) * 16;
          dst = (uint32_t)((piece * t.N + to) * 16);
          bytes = (uint32_t)rows * 16u;
        }
      }
      const size_t wstep = (size_t)chunk_bytes(kFmt, Nb);
      const int sub = lane == 31 ? warp : per;               // lane 31 of the first two warps: a sub-matrix of rows
      const uint8_t* x = reinterpret_cast<const uint8_t*>(s.x) + ((size_t)(t.m * per + (sub < per ? sub : 0)) * s.K + (size_t)t.c0 * kKc) * 256;
      const uint32_t tx = (uint32_t)(t.subs * kSub + chunk_bytes(kFmt, t.N));
      auto weights = [&](int c, int st) {
        if (item == 0) mbar_arrive_expect_tx(&sh.full[st], tx);
        if (bytes) bulk_load_1d(ring + st * stage_bytes + per * kSub + dst, src + (size_t)c * wstep, bytes, &sh.full[st]);
      };
      auto rows_in = [&](int c, int st) {
        if (sub < t.subs) bulk_load_1d(ring + st * stage_bytes + sub * kSub, x + (size_t)c * kSub, kSub, &sh.full[st]);
      };
      int c = 0;
      if (it == 0) {
        // weights depend on nothing: the first ones are on their way before the rows' producer has ended
        const int early = min(t.n_ch, n_ring);
        for (; c < early; ++c) weights(c, c);
        grid_dep_wait();
        fence_proxy_async();
        for (c = 0; c < early; ++c, at_ring.next()) rows_in(c, c);
        it = early;
      }
      for (; c < t.n_ch; ++c, ++it, at_ring.next()) {
        const int st = at_ring.st;
        if (it >= n_ring && !(ok = wait.warp_wait(&sh.empty[st], at_ring.parity ^ 1u, 0, it))) break;
        weights(c, st);
        rows_in(c, st);
      }
    }
    grid_dep_launch();
  } else if (warp == kWideProducers) {
    if (lane == 0) {
      // What this thread does per chunk beside its MMAs is time the tensor cores stand still once their short queue is empty:
      // no divisions, descriptors advanced by constants (gate/up of 2048 rows 427 -> 354 us).
      bool ok = true;
      uint32_t used[2] = {0u, 0u};          // times an accumulator was taken
      RingAt at{n_ring};
      const uint32_t stage16 = (uint32_t)stage_bytes >> 4;
      const uint64_t a0 = umma_desc(smem_u32(ring), 2048u, 128u);
      for (int i = blockIdx.x, it = 0, j = 0; i < n_tiles && ok; i += gridDim.x, ++j) {
        const WideTile t = wide_tile(s, i);
        const uint32_t idesc = umma_idesc_bf16_m128(t.N), lbo_b = (uint32_t)t.N * 16u, step_b = (2u * lbo_b) >> 4;
        const uint64_t b0 = umma_desc(smem_u32(kFmt != 0 ? staging : ring + per * kSub), lbo_b, 128u);
        const uint32_t stg16 = (uint32_t)(NT * kKc * 2) >> 4;
        const int slot0 = per == 2 ? 0 : j & 1;
        for (int c = 0; c < t.n_ch; ++c, ++it, at.next()) {
          const int st = at.st;
          // widened weights stand for the chunk's arrival too: the warps that widened them have seen it
          ok = wait(kFmt != 0 ? &sh.ready[st] : &sh.full[st], at.parity, 1, it);
          if (!ok) break;
          if (c == 0) {
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if (u >= slot0 && u < slot0 + t.subs) {
                if (used[u] > 0 && ok) ok = wait(&sh.acc_empty[u], (used[u] - 1u) & 1u, 1, it);
                ++used[u];
              }
            if (!ok) break;
          }
          tc_fence_after();
          const uint64_t ad = a0 + st * stage16, bd = b0 + (kFmt != 0 ? (it & 1) * stg16 : st * stage16);
          for (int u = 0; u < t.subs; ++u) {
            const uint32_t d = tmem + (uint32_t)((slot0 + u) * kWideN);
#pragma unroll
            for (int k = 0; k < kKc / 16; ++k)
              umma_bf16(d, ad + u * (kSub >> 4) + k * 256, bd + k * step_b, idesc, (uint32_t)((c | k) != 0));
          }
          umma_commit(&sh.empty[st]);
          if (kFmt != 0) umma_commit(&sh.stg_empty[it & 1]);
        }
        if (ok)
          for (int u = 0; u < t.subs; ++u) umma_commit(&sh.acc_full[slot0 + u]);
      }
    }
  } else {
    const int worker = warp - kWideProducers - 1, quarter = warp & 3, group = worker >> 2, t512 = tid - 32 * (kWideProducers + 1);
    bool skip = false, first = true;
    const float* scales = reinterpret_cast<const float*>(s.scales);
    int uses = 0;
    RingAt at_ring{n_ring};
    for (int i = blockIdx.x, j = 0, it = 0; i < n_tiles; i += gridDim.x, ++j) {
      const WideTile t = wide_tile(s, i);
      bool seen = true;
      if (kFmt != 0) {
        for (int c = 0; c < t.n_ch; ++c, ++it, at_ring.next()) {
          const int st = at_ring.st;
          // Two teams take the chunks in turn: one's wait for the tensor cores to leave its buffer falls into the other's
          // work.  Both see every chunk arrive, so that no phase of a ring's barrier passes unseen.
          const bool mine = (it & 1) == (worker >> 3);
          seen = wait(&sh.full[st], at_ring.parity, 3, it) &&
                 (!mine || it < 2 || wait(&sh.stg_empty[it & 1], (uint32_t)((it >> 1) - 1) & 1u, 3, it));
          if (!(seen = __all_sync(0xffffffffu, seen))) break;
          if (!mine) {
            if (lane == 0) mbar_arrive(&sh.empty[st]);
            continue;
          }
          uint8_t* dst = staging + (it & 1) * (NT * kKc * 2);
          const uint8_t* src = ring + st * stage_bytes + per * kSub;
          for (int g = 0, row = t512 & 255; g < 4; row += 256) {       // consecutive threads take consecutive rows
            for (; g < 4 && row >= t.N; ++g) row -= t.N;
            if (g < 4) widen16<kFmt>(dst, src, t.N, row, g);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.ready[st]);
        }
        if (!seen) break;
      }
      if (first) {
        grid_dep_wait();                                       // the outputs' last readers have ended
        skip = ld_relaxed_gpu(&status->abort) != 0;            // behind an unread error nothing is written
        first = false;
      }
      // a sub-matrix's columns are shared by its two (of two sub-matrices) or four groups of four warps
      const int which = per == 2 ? group >> 1 : 0, share = per == 2 ? group & 1 : group, shares = 4 / per;
      if (which >= t.subs) continue;
      const int slot = per == 2 ? which : j & 1, sub = t.m * per + which;
      const int wide = (t.N / 16 + shares - 1) / shares * 16;
      const int lo = share * wide, hi = min(lo + wide, t.N);
      const int use = per == 2 ? uses++ : j >> 1;
      if (!wait.warp_wait(&sh.acc_full[slot], (uint32_t)use & 1u, 2, i)) break;
      tc_fence_after();
      const int b = quarter * 32 + lane;
      for (int n = lo; n < hi; n += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * kWideN + n), r);
        if (skip) continue;
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[e]);
        const int col = t.n0 + n;
        if (kFmt != 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 sc = __ldg(reinterpret_cast<const float4*>(scales + col) + e);
            v[4 * e] *= sc.x; v[4 * e + 1] *= sc.y; v[4 * e + 2] *= sc.z; v[4 * e + 3] *= sc.w;
          }
        }
        if (s.mode == VDC_STAGE_SILU) {
          float o[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float g = bf16_round(v[2 * e]), u = bf16_round(v[2 * e + 1]);
            o[e] = bf16_round(g / (1.f + __expf(-g))) * u;
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + (size_t)sub * 128 * (s.M / 2) * 2 + kc_piece(128, b, col >> 1)) = pack8(o);
        } else {
          float4* out = reinterpret_cast<float4*>(s.out) + ((size_t)t.split * (s.M >> 2) + (col >> 2)) * s.Bpad + sub * 128 + b;
#pragma unroll
          for (int e = 0; e < 4; ++e) out[(size_t)e * s.Bpad] = make_float4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.acc_empty[slot]);
    }
  }
  __syncwarp();
  wait.drain();
  __syncthreads();
  if (warp == kWideProducers) tmem_dealloc(tmem, 2 * kWideN);
}

// Sum of the K-splits' partial sums of four columns, in order.
__device__ __forceinline__ float4 wide_sum4(const vdc_stage& s, int M, int quad, int row) {
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4* p = reinterpret_cast<const float4*>(s.x) + (size_t)quad * s.Bpad + row;
  for (int i = 0; i < s.splits; ++i) {
    const float4 v = __ldcg(p + (size_t)i * (M >> 2) * s.Bpad);
    a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
  }
  return a;
}

// Embedding rows of the prompt; rows past its end take its last id.  An id outside the table is reported, row 0 taken.
__global__ void __launch_bounds__(128) wide_embed(const __grid_constant__ vdc_stage s, vdc_status* status) {
  const int b = blockIdx.x;
  grid_dep_wait();
  grid_dep_launch();
  const int n = wide_rows(s);
  int token = ld_relaxed_gpu(reinterpret_cast<const int*>(s.log) + min(b, n - 1));
  if (ld_relaxed_gpu(&status->abort)) return;
  if (token < 0 || (s.M > 0 && token >= s.M)) {
    if (threadIdx.x == 0) report(status, VDC_ERR_TOKEN, s.kind, 0, b, token);
    token = 0;
  }
  const uint4* row = reinterpret_cast<const uint4*>(s.w) + (size_t)token * (s.K / 8);
  uint8_t* out = reinterpret_cast<uint8_t*>(s.hid) + (size_t)(b / 128) * 128 * s.K * 2;
  for (int p = threadIdx.x; p < s.K / 8; p += 128) *reinterpret_cast<uint4*>(out + kc_piece(128, b % 128, p * 8)) = __ldg(row + p);
}

// hid += the projection's sums (x; 0: none), then (out) its RMSNorm, both rounded like a bf16 tensor expression.  Two rows per
// block: the two share the 32-byte sectors of the matrix; 256 threads each, so that few rows are many loads at a time.  A row's
// first kKept pieces of a thread stay in registers between the sum of squares and the products, and their norm weights are on
// their way while the projection ends: 600 rows of two 8B-shaped layers NVFP4 1012 -> 996 us, e4m3 1034 -> 1022.
constexpr int kNormThreads = 512;
__global__ void __launch_bounds__(kNormThreads, 2) wide_norm(const __grid_constant__ vdc_stage s, vdc_status* status) {
  constexpr int kStep = kNormThreads / 2, kKept = 2;
  __shared__ float red[kNormThreads / 32][2];
  const int tid = threadIdx.x, r = tid & 1, b = (int)blockIdx.x * 2 + r, t = tid >> 1, pieces = s.K / 8;
  const size_t sub = (size_t)(b / 128) * 128 * s.K * 2;
  uint8_t* hid = reinterpret_cast<uint8_t*>(s.hid) + sub;
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  uint4 kept[kKept], w[kKept];
#pragma unroll
  for (int q = 0; q < kKept; ++q)
    w[q] = s.out && t + q * kStep < pieces ? __ldg(reinterpret_cast<const uint4*>(s.norm_w) + t + q * kStep) : none;
  grid_dep_wait();
  grid_dep_launch();
  const int aborted = ld_relaxed_gpu(&status->abort);
  float ssq = 0.f;
  const float4* sums = reinterpret_cast<const float4*>(s.x) + b;
  const size_t split = (size_t)(s.K >> 2) * s.Bpad;
  // kKept pieces from k0 on: the hidden state with the sums added, its squares
  auto add = [&](int k0, uint4 (&h)[kKept]) {
    float4 y[kKept][2];
#pragma unroll
    for (int q = 0; q < kKept; ++q) {
      const int k8 = k0 + q * kStep;
      h[q] = k8 < pieces ? __ldcg(reinterpret_cast<const uint4*>(hid + kc_piece(128, b % 128, k8 * 8))) : none;
      y[q][0] = y[q][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (s.x) {
#pragma unroll 4
      for (int i = 0; i < s.splits; ++i)
#pragma unroll
        for (int q = 0; q < kKept; ++q)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int k8 = k0 + q * kStep;
            const float4 v = k8 < pieces ? __ldcg(sums + i * split + (size_t)(2 * k8 + e) * s.Bpad) : make_float4(0.f, 0.f, 0.f, 0.f);
            y[q][e].x += v.x; y[q][e].y += v.y; y[q][e].z += v.z; y[q][e].w += v.w;
          }
    }
#pragma unroll
    for (int q = 0; q < kKept; ++q) {
      const int k8 = k0 + q * kStep;
      if (k8 >= pieces) break;
      const uint32_t hv[4] = {h[q].x, h[q].y, h[q].z, h[q].w};
      const float yv[8] = {y[q][0].x, y[q][0].y, y[q][0].z, y[q][0].w, y[q][1].x, y[q][1].y, y[q][1].z, y[q][1].w};
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] = bf_lo(hv[j]);
        v[2 * j + 1] = bf_hi(hv[j]);
      }
      if (s.x) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j] + bf16_round(yv[j]));
        h[q] = pack8(v);
        if (!aborted) *reinterpret_cast<uint4*>(hid + kc_piece(128, b % 128, k8 * 8)) = h[q];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ssq = fmaf(v[j], v[j], ssq);
    }
  };
  add(t, kept);
  for (int k0 = t + kKept * kStep; k0 < pieces; k0 += kKept * kStep) {
    uint4 h[kKept];
    add(k0, h);
  }
  if (!s.out || __syncthreads_or(aborted)) return;
#pragma unroll
  for (int x = 2; x < 32; x <<= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, x);
  if ((tid & 31) < 2) red[tid >> 5][r] = ssq;
  __syncthreads();
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kNormThreads / 32; ++i) sum += red[i][r];
  const float rstd = rsqrtf(sum / (float)s.K + s.eps);
  auto scale = [&](int k8, const uint4& h, const uint4& w) {
    const uint32_t hv[4] = {h.x, h.y, h.z, h.w}, wv[4] = {w.x, w.y, w.z, w.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o[j] = pack_bf16x2(bf16_round(bf_lo(hv[j]) * rstd) * bf_lo(wv[j]), bf16_round(bf_hi(hv[j]) * rstd) * bf_hi(wv[j]));
    *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + sub + kc_piece(128, b % 128, k8 * 8)) = make_uint4(o[0], o[1], o[2], o[3]);
  };
#pragma unroll
  for (int q = 0; q < kKept; ++q)
    if (t + q * kStep < pieces) scale(t + q * kStep, kept[q], w[q]);
  for (int k8 = t + kKept * kStep; k8 < pieces; k8 += kStep)
    scale(k8, ldcg128(hid + kc_piece(128, b % 128, k8 * 8)), __ldg(reinterpret_cast<const uint4*>(s.norm_w) + k8));
}

// Heads of the QKV projection's sums, eight rows to a block and a warp to a row: q/k norm, rotation, query rows and cache
// rows.  A block takes one KV head's G + 2 heads, with the next one's sums on their way while it finishes one, or a single head
// where that would be few blocks (heads_per_block).
__host__ __device__ inline int heads_per_block(const vdc_stage& s) { return s.Bpad * s.n_kv >= 8 * 512 ? s.group + 2 : 1; }
__global__ void __launch_bounds__(256) wide_heads(const __grid_constant__ vdc_stage s, vdc_status* status) {
  constexpr int kLd = VDC_HEAD_DIM + 4;
  __shared__ alignas(16) float tile[2][8][kLd];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, heads = heads_per_block(s), parts = s.n_kv * (s.group + 2) / heads;
  const int first = (int)blockIdx.x % parts * heads, b0 = (int)blockIdx.x / parts * 8;
  grid_dep_wait();
  grid_dep_launch();
  const int row = tid & 7, quad = tid >> 3;
  float4 next = wide_sum4(s, s.M, first * (VDC_HEAD_DIM / 4) + quad, b0 + row);
  const int n = wide_rows(s), b = b0 + warp, pos = wide_first(s) + min(b, n - 1);
  const int page = ld_relaxed_gpu(reinterpret_cast<const int*>(s.state) + VDC_ST_PAGETABLE + pos / VDC_KV_PAGE);
  if (b0 >= n || __syncthreads_or(ld_relaxed_gpu(&status->abort))) return;
  for (int i = 0; i < heads; ++i) {
    *reinterpret_cast<float4*>(&tile[i & 1][row][quad * 4]) = next;
    __syncthreads();
    if (i + 1 < heads) next = wide_sum4(s, s.M, (first + i + 1) * (VDC_HEAD_DIM / 4) + quad, b0 + row);
    const float* in = tile[i & 1][warp];
    const float2 lo = *reinterpret_cast<const float2*>(in + lane * 2), hi = *reinterpret_cast<const float2*>(in + lane * 2 + 64);
    float x[4] = {lo.x, lo.y, hi.x, hi.y};
    if (b < n) head_row(s, x, b, first + i, lane, pos, page * VDC_KV_PAGE * s.n_kv + pos % VDC_KV_PAGE, true);
  }
}

// The rows of a prompt's last chunk (s.B of them from row s.M; past the prompt's end its last row again) into the chunk's
// hidden matrix, with their sums of squares: the stages behind find what the chunk's own stages would have left.
__global__ void __launch_bounds__(128) wide_tail(const __grid_constant__ vdc_stage s, vdc_status* status) {
  __shared__ float red[4];
  const int b = blockIdx.x, tid = threadIdx.x;
  grid_dep_wait();
  grid_dep_launch();
  if (__syncthreads_or(ld_relaxed_gpu(&status->abort))) return;
  const int from = min(s.M + b, wide_rows(s) - 1);
  const uint8_t* x = reinterpret_cast<const uint8_t*>(s.x) + (size_t)(from / 128) * 128 * s.K * 2;
  float ssq = 0.f;
  for (int k8 = tid; k8 < s.K / 8; k8 += 128) {
    const uint4 v = ldcg128(x + kc_piece(128, from % 128, k8 * 8));
    const uint32_t xv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) ssq = fmaf(bf_lo(xv[j]), bf_lo(xv[j]), fmaf(bf_hi(xv[j]), bf_hi(xv[j]), ssq));
    *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.hid) + kc_piece(s.Bpad, b, k8 * 8)) = v;
  }
  ssq = warp_sum(ssq);
  if ((tid & 31) == 0) red[tid >> 5] = ssq;
  __syncthreads();
  if (tid == 0) reinterpret_cast<float*>(s.stats_out)[b] = red[0] + red[1] + red[2] + red[3];
}

}  // namespace vdc

extern "C" cudaError_t vdc_wide_prepare() {
  const void* gemms[] = {(const void*)vdc::wide_gemm<0>, (const void*)vdc::wide_gemm<1>, (const void*)vdc::wide_gemm<2>};
  for (const void* f : gemms)
    if (cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, vdc::kWideSmem)) return e;
  return cudaSuccess;
}

// CTAs of a wide stage.  Projections: one per SM at most (sms), each with its share of the tiles.
extern "C" int vdc_wide_grid(const vdc_stage* s, int sms, int* tiles) {
  *tiles = 0;
  switch (s->kind) {
    case VDC_STAGE_WIDE_EMBED: return s->Bpad;
    case VDC_STAGE_WIDE_NORM: return s->Bpad / 2;
    case VDC_STAGE_WIDE_HEADS: return s->Bpad / 8 * s->n_kv * (s->group + 2) / vdc::heads_per_block(*s);
    case VDC_STAGE_WIDE_TAIL: return s->B;
    default: break;
  }
  const int per = s->group, m = (s->Bpad / 128 + per - 1) / per, n = (s->M + s->n_kv - 1) / s->n_kv;
  *tiles = m * n * s->splits;
  return *tiles < sms ? *tiles : sms;
}

extern "C" cudaError_t vdc_wide_launch(const vdc_stage* s, int sms, vdc_status* status, uint64_t timeout_ns, cudaStream_t stream) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int tiles;
  cfg.gridDim = dim3((unsigned)vdc_wide_grid(s, sms, &tiles));
  switch (s->kind) {
    case VDC_STAGE_WIDE_GEMM: {
      auto f = s->wfmt == 0 ? vdc::wide_gemm<0> : s->wfmt == 1 ? vdc::wide_gemm<1> : vdc::wide_gemm<2>;
      cfg.blockDim = dim3(vdc::kWideThreads);
      cfg.dynamicSmemBytes = vdc::kWideSmem;
      return cudaLaunchKernelEx(&cfg, f, *s, tiles, status, timeout_ns);
    }
    case VDC_STAGE_WIDE_EMBED: cfg.blockDim = dim3(128); return cudaLaunchKernelEx(&cfg, vdc::wide_embed, *s, status);
    case VDC_STAGE_WIDE_NORM: cfg.blockDim = dim3(vdc::kNormThreads); return cudaLaunchKernelEx(&cfg, vdc::wide_norm, *s, status);
    case VDC_STAGE_WIDE_HEADS: cfg.blockDim = dim3(256); return cudaLaunchKernelEx(&cfg, vdc::wide_heads, *s, status);
    case VDC_STAGE_WIDE_TAIL: cfg.blockDim = dim3(128); return cudaLaunchKernelEx(&cfg, vdc::wide_tail, *s, status);
    default: return cudaErrorInvalidValue;
  }
}

// The tile of a projection for the least estimated time, in ns (measured, B200): a chunk of 64 inputs takes 200 + 1.05 per
// sub-matrix and column (480 at 1 x 256, 740 at 2 x 256) and 440 at least, 40 more where tiles cut blocks of packed weights
// (more and smaller copies), and what widening takes where that is longer (e4m3 1130 at 224 columns, NVFP4 1280); a tile's
// epilogue 4 us, beside the next tile where that is of one sub-matrix; the weights come at 5.6 TB/s; fp32 sums are written
// and read once per split.
extern "C" void vdc_wide_choose(int rows, int M, int K, int wfmt, int sms, int whole, int* out) {
  const int subs_all = rows / 128, chunks = K / 64;
  const double wbytes = (double)M * K * (wfmt == 0 ? 2.0 : wfmt == 1 ? 1.0 : 0.5625), widen = wfmt == 0 ? 0.0 : wfmt == 1 ? 2.4 : 3.2;
  double best = 0.0;
  int most = chunks / 4 < 8 ? chunks / 4 : 8;
  if (most > 2048 / rows) most = 2048 / rows;
  if (whole || most < 1) most = 1;
  for (int subs = 1; subs <= 2 && subs <= subs_all; ++subs)
    for (int cols = 64; cols <= 256; cols += 16) {
      double chunk = 200 + 1.05 * subs * cols + (cols % 128 ? 40 : 0);
      if (chunk < 440) chunk = 440;
      if (wfmt && chunk < 560 + widen * cols) chunk = 560 + widen * cols;
      for (int ks = 1; ks <= most; ++ks) {
        const int tiles = (subs_all + subs - 1) / subs * ((M + cols - 1) / cols) * ks, waves = (tiles + sms - 1) / sms;
        double t = waves * ((chunks + ks - 1) / ks * chunk + (subs == 2 ? 4000 : 0)) + 4000;
        if (t < wbytes / 5600 + 4000) t = wbytes / 5600 + 4000;
        if (!whole) t += (double)ks * rows * M * 8 / 5000;
        if (best == 0.0 || t < best) {
          best = t;
          out[0] = subs;
          out[1] = cols;
          out[2] = ks;
        }
      }
    }
}

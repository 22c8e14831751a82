// Stage kernels: the batched decode step and the chunked prefill as one kernel per stage.
//
// A step of 2..128 rows runs, per layer: QKV projection (with per-head norm, rotation and the cache append in its
// epilogue), attention, output projection, gate/up projection, down projection.  The rows sit on the 128 lanes of a
// tcgen05 accumulator, a block of 128 weight rows on its columns; with quantised weights, which are widened into tensor
// memory as the A operand, it is the other way round: 32 rows took 68 KB of shared-memory traffic per 8 KB of e4m3 weights
// when they were widened into shared memory, 24 KB so (two layers 321.5 -> 303.4 us).  Why kernels and not tasks of the megakernel: with
// many rows a projection block needs a K-split whose partial sums meet (here through distributed shared memory inside
// one cluster, in the megakernel through fp32 atomics in L2 and a last arrival that ran the block's epilogue alone), and
// a stage boundary needs no spinning: programmatic dependent launch starts the next kernel's CTAs while this one drains,
// and they fill their shared memory with weights before they wait for its results (427 -> 384 us for two layers and a
// 128256-row vocabulary projection at 3 rows).
//
// Measured against the megakernel's program, two Llama-3.1-8B-shaped layers and a small vocabulary (B200): 3 rows at
// 1000 positions 416 -> 235 us, 32 rows with e4m3 weights 759 -> 276, 64 rows at 2100 positions 929 -> 402, 128 rows
// 1024 -> 397 (up to 4 % more or less from one GPU to another).
#include "mk_stage.cuh"

namespace vdc {

constexpr int kBlk = VDC_STAGE_BLOCK;   // weight rows of a projection block: accumulator columns
constexpr int kKc = 64;                 // inputs per chunk
constexpr int kMaxRing = 16;
constexpr int kBufs = 4;                // of widened weights
constexpr int kRowCols = 128;           // tensor memory: sums in columns 0 .. 127, widened weights behind them
constexpr int kGemmThreads = 320;       // producer warp, MMA warp, eight warps that convert weights and run the epilogue
constexpr int kEpiThreads = 256;
// Shared memory of one CTA.  Two CTAs fit an SM (the register budget allows it too), so that one streams while the
// other is in its prologue or epilogue, and the next stage's CTAs move in while the last ones of this stage finish.
constexpr int kGemmSmem = 110 * 1024;
constexpr int kCol4 = kBlk / 4;         // groups of four columns in the fp32 exchange tile

// ------------------------------------------------------------------------- //
// projection: D[b, n] = sum_k X[b, k] W[n, k] for one block of weight rows, K shared by the CTAs of a cluster
// ------------------------------------------------------------------------- //
struct GemmShared {
  uint64_t full[kMaxRing], empty[kMaxRing];
  uint64_t ready[kMaxRing];     // weights converted
  uint64_t done;
  uint32_t tmem;
  volatile int fail;
  int skip;                     // an earlier stage failed: what this one computes is not written
  float ssq[128];
  unsigned long long key[128];
};

// One ring stage: the rows' chunk, then the weights' chunk.
__host__ __device__ constexpr int stage_size(int wfmt, int bpad) {
  return bpad * kKc * 2 + (chunk_bytes(wfmt, kBlk) + 127) / 128 * 128;
}
__host__ __device__ inline int ring_stages(int wfmt, int bpad) {
  const int n = (kGemmSmem - 2048 - 128) / stage_size(wfmt, bpad), most = wfmt ? kMaxRing : 8;
  return n >= most ? most : wfmt ? n & ~1 : n;      // even where weights are converted, see kTeams
}
// Quantised weights are converted by two teams of warps that take the chunks in turn, so that a team's waits fall into the other's
// conversion.  The ring's length is even then: a team sees every round of its places (it would otherwise meet a place two rounds
// on, and the barrier's parity cannot tell those apart).
constexpr int kTeams = 2, kTeam = kEpiThreads / kTeams;
static_assert(kTeam == 128, "a thread of a team for every lane of tensor memory");
static_assert((kGemmSmem - 2048 - 128) / stage_size(1, 128) >= kBufs && kBufs % kTeams == 0,
              "a place for every buffer of widened weights (128 rows of e4m3 weights are the largest places)");

// The exchange tile of a CTA: [source CTA][four columns][its row, one spare][4] fp32.  Every CTA of the cluster writes the
// sums of its K-range straight from tensor memory into the tile of the CTA that finishes the row (consecutive rows lie
// side by side, so a warp's store is contiguous; the spare row spreads the column groups over the banks); what is then
// read is local.  Pulling the sums instead cost one remote round trip per source and item.
__device__ __forceinline__ uint32_t tile_at(uint32_t tile, int src, int nb, int col4, int row) {
  return tile + (uint32_t)(((src * kCol4 + col4) * (nb + 1) + row) * 16);
}
// Eight fp32 sums (columns col .. col+7 of the CTA's row bl) over the cluster's K-ranges, in rank order.
__device__ __forceinline__ void sum8(float (&v)[8], const uint8_t* tile, int splits, int nb, int bl, int col) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  for (int r = 0; r < splits; ++r) {
    const uint8_t* p = tile + (size_t)((r * kCol4 + (col >> 2)) * (nb + 1) + bl) * 16;
    const float4 a = *reinterpret_cast<const float4*>(p), c = *reinterpret_cast<const float4*>(p + (nb + 1) * 16);
    v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    v[4] += c.x; v[5] += c.y; v[6] += c.z; v[7] += c.w;
  }
}
// One head of the QKV projection, one warp per row: the sums over the cluster's K-ranges, then the rest of the head.
__device__ __forceinline__ void qkv_head(const vdc_stage& s, const uint8_t* tile, int splits, int nb, int bl, int b, int block,
                                         int lane) {
  const int n0 = block * kBlk, i0 = lane * 2;
  float x[4] = {0.f, 0.f, 0.f, 0.f};
  for (int r = 0; r < splits; ++r) {
    const uint8_t* p = tile + (size_t)((r * kCol4 + (i0 >> 2)) * (nb + 1) + bl) * 16 + (i0 & 3) * 4;
    const float2 lo = *reinterpret_cast<const float2*>(p), hi = *reinterpret_cast<const float2*>(p + (size_t)(16 * (nb + 1)) * 16);
    x[0] += lo.x; x[1] += lo.y; x[2] += hi.x; x[3] += hi.y;
  }
  const float* scales = reinterpret_cast<const float*>(s.scales);
  if (scales != nullptr) {
    const float2 lo = __ldg(reinterpret_cast<const float2*>(scales + n0 + i0));
    const float2 hi = __ldg(reinterpret_cast<const float2*>(scales + n0 + i0 + 64));
    x[0] *= lo.x; x[1] *= lo.y; x[2] *= hi.x; x[3] *= hi.y;
  }
  const int* st = reinterpret_cast<const int*>(s.state) + (size_t)b * s.state_stride;
  // rows past a prompt's end repeat its last position: the first of them writes the cache row, since their sums of squares
  // (atomics) may differ in the last bit
  const int new_row = ld_relaxed_gpu(st + VDC_ST_NEWROW);
  const bool first = b == 0 || ld_relaxed_gpu(st - s.state_stride + VDC_ST_NEWROW) != new_row;
  head_row(s, x, b, block, lane, ld_relaxed_gpu(st + VDC_ST_POS), new_row, first);
}

// The exchange of a block whose weight rows lie on the accumulator's lanes: [source CTA][kPiece of its rows][128 columns][kPiece]
// fp32, so that a lane has a piece of consecutive rows and a warp stores 32 of them side by side.  A store to another CTA costs what
// the pieces cost into which it falls.  Eight CTAs to a block, 128 rows, e4m3: 4096 x 1024 17.1 us with a lane storing single words of
// the layout of tile_at, 12.6 with sixteen lanes exchanging sixteen values each in front of the stores, 12.5 so; 2048 x 4096 16.3, 13.1
// and 12.7; of 32 rows 9.1, 8.8 and 8.4.  kPiece is 2 where a CTA finishes two rows.
template <int kPiece>
__device__ __forceinline__ uint32_t piece_at(uint32_t tile, int src, int nb, int row, int col) {
  return tile + (uint32_t)(((src * nb + row) / kPiece * kBlk + col) * kPiece) * 4u;
}
// This warp's accumulator columns (rows row0 .. row0 + 15 of a lane's weight row n) to the CTAs that finish them.
template <int kPiece>
__device__ __forceinline__ void send_pieces(const uint32_t (&r)[16], uint32_t tile, int rank, int nb, int row0, int n) {
  const int lg = 31 - __clz(nb);
#pragma unroll
  for (int j = 0; j < 16; j += kPiece) {
    const uint32_t to = peer_smem(piece_at<kPiece>(tile, rank, nb, (row0 + j) & (nb - 1), n), (uint32_t)((row0 + j) >> lg));
    if constexpr (kPiece == 4) st_cluster4(to, r[j], r[j + 1], r[j + 2], r[j + 3]);
    else st_cluster2(to, r[j], r[j + 1]);
  }
}
static_assert(128 * kBlk * 4 + kCol4 * (64 + 1) * 16 <= kGemmSmem - 128, "pieces of 128 rows, and behind them the sums of a CTA's 64");
// The sums over the cluster's K-ranges, in rank order, from pieces to the layout of tile_at (one source; rows and columns of a warp's
// stores lie in different banks).
template <int kPiece>
__device__ __forceinline__ void sum_pieces(uint8_t* to, const uint8_t* from, int splits, int nb, int N, int t) {
  using Piece = typename std::conditional<kPiece == 4, float4, float2>::type;
  for (int i = t; i < nb / kPiece * kBlk; i += kEpiThreads) {
    const int n = i & (kBlk - 1), row = i / kBlk * kPiece;
    if (n >= N) continue;
    float v[kPiece];
#pragma unroll
    for (int j = 0; j < kPiece; ++j) v[j] = 0.f;
    for (int src = 0; src < splits; ++src) {
      const Piece p = *reinterpret_cast<const Piece*>(from + (size_t)piece_at<kPiece>(0u, src, nb, row, n));
      v[0] += p.x; v[1] += p.y;
      if constexpr (kPiece == 4) { v[2] += p.z; v[3] += p.w; }
    }
    float* out = reinterpret_cast<float*>(to + tile_at(0u, 0, nb, n >> 2, row)) + (n & 3);
#pragma unroll
    for (int j = 0; j < kPiece; ++j) out[4 * j] = v[j];
  }
}

template <int kFmt>
__global__ void __launch_bounds__(kGemmThreads, 2) stage_gemm(const __grid_constant__ vdc_stage s, int first_block, int n_ring,
                                                              vdc_status* status, uint64_t timeout_ns) {
  extern __shared__ uint8_t dyn[];
  __shared__ GemmShared sh;
  constexpr int kTmem = kFmt != 0 ? kRowCols + kBufs * kKc / 2 : kBlk;
  static_assert(kTmem == 128 || kTmem == 256, "a power of two");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = s.splits;
  const int rank = splits > 1 ? (int)cluster_rank() : 0;
  const int block = first_block + (int)blockIdx.x / splits;
  const int n0 = block * kBlk, N = min(kBlk, s.M - n0);
  const int chunks = s.K / kKc, c0 = chunks * rank / splits, n_ch = chunks * (rank + 1) / splits - c0;
  const int xbytes = s.Bpad * kKc * 2, wbytes = chunk_bytes(kFmt, N);
  const int stage_bytes = stage_size(kFmt, s.Bpad);
  uint8_t* ring = aligned128(dyn);
  const Waiter wait{&sh.fail, status, timeout_ns, s.kind};

  if (warp == 1) tmem_alloc(&sh.tmem, kTmem);
  if (tid == 0) {
    for (int i = 0; i < n_ring; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 1);
      mbar_init(&sh.ready[i], kTeam / 32);
    }
    mbar_init(&sh.done, 1);
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 64 && tid < 192) {
    sh.ssq[tid - 64] = 0.f;
    sh.key[tid - 64] = 0ull;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;

  if (warp == 0) {
    if (lane == 0) {
      const uint8_t* w = reinterpret_cast<const uint8_t*>(s.w) + (size_t)n0 * s.K * (kFmt == 0 ? 32 : kFmt == 1 ? 16 : 9) / 16 +
                         (size_t)c0 * wbytes;
      const uint8_t* x = reinterpret_cast<const uint8_t*>(s.x) + (size_t)c0 * xbytes;
      const uint32_t tx = (uint32_t)(xbytes + wbytes);
      auto load_weights = [&](int i, int st) {
        mbar_arrive_expect_tx(&sh.full[st], tx);
        bulk_load_1d(ring + st * stage_bytes + xbytes, w + (size_t)i * wbytes, (uint32_t)wbytes, &sh.full[st]);
      };
      // the weights depend on nothing: they are on their way before the previous stage's results are waited for
      const int first = min(n_ch, n_ring);
      for (int i = 0; i < first; ++i) load_weights(i, i);
      grid_dep_wait();
      fence_proxy_async();
      for (int i = 0; i < first; ++i) bulk_load_1d(ring + i * stage_bytes, x + (size_t)i * xbytes, (uint32_t)xbytes, &sh.full[i]);
      const int aborted = ld_relaxed_gpu(&status->abort);    // looked at below, when it has long arrived
      RingAt at{n_ring};
      for (int i = first; i < n_ch; ++i, at.next()) {       // chunk i takes the place of chunk i - n_ring
        const int st = at.st;
        if (!wait(&sh.empty[st], at.parity, 0, i)) break;
        load_weights(i, st);
        bulk_load_1d(ring + st * stage_bytes, x + (size_t)i * xbytes, (uint32_t)xbytes, &sh.full[st]);
      }
      sh.skip = aborted;
      grid_dep_launch();     // not earlier: waiting CTAs of the stages behind would hold the shared memory of this one's
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_bf16_m128(kFmt != 0 ? s.Bpad : N);
      const uint32_t lbo_x = (uint32_t)s.Bpad * 16u, lbo_w = (uint32_t)N * 16u;
      // No divisions per chunk and descriptors advanced by constants, here and in the other roles: what this thread does beside
      // its MMAs the tensor cores wait for.  A step of 32 rows with e4m3 weights 338 -> 319 us, 16 rows NVFP4 364 -> 358, 3 rows
      // bf16 245 -> 242.
      const uint64_t x0 = umma_desc(smem_u32(ring), lbo_x, 128u), w0 = umma_desc(smem_u32(ring + xbytes), lbo_w, 128u);
      const uint32_t stage16 = (uint32_t)stage_bytes >> 4, step_x = (2u * lbo_x) >> 4, step_w = (2u * lbo_w) >> 4;
      // A finished wait is 145 cycles here, a commit 140 and an MMA 75, more than the tensor cores take for it: the descriptors are
      // made in front of the wait, converted weights stand for the chunk's arrival too (the warps that converted them have seen
      // it), and one commit gives back the chunk's place and the buffer.
      RingAt at{n_ring};
      for (int i = 0; i < n_ch; ++i, at.next()) {
        const int st = at.st;
        uint64_t xd[kKc / 16], wd[kKc / 16];
#pragma unroll
        for (int k = 0; k < kKc / 16; ++k) {
          xd[k] = x0 + st * stage16 + k * step_x;
          wd[k] = kFmt != 0 ? tmem + kRowCols + (i & (kBufs - 1)) * (kKc / 2) + k * 8 : w0 + st * stage16 + k * step_w;
          asm volatile("" : "+l"(xd[k]), "+l"(wd[k]));
        }
        if (!wait(kFmt != 0 ? &sh.ready[st] : &sh.full[st], at.parity, 1, i)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kKc / 16; ++k) {
          if (kFmt != 0) umma_bf16_ta(tmem, (uint32_t)wd[k], xd[k], idesc, (uint32_t)((i | k) != 0));
          else umma_bf16(tmem, xd[k], wd[k], idesc, (uint32_t)((i | k) != 0));
        }
        umma_commit(&sh.empty[st]);
      }
      umma_commit(&sh.done);
      wait(&sh.done, 0u, 1, n_ch);
      tc_fence_before();     // the warps that read the accumulators learn of their completion from this thread's next barrier
    }
  } else {
    const int t = tid - 64;
    if (kFmt != 0) {
      // A warp widens the rows whose lanes of tensor memory it reaches; rows past N are whatever lies there, for sums that nobody
      // reads.
      const int quarter = warp & 3, row = quarter * 32 + lane;
      const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + kRowCols;
      // `old`: the place of the chunk whose buffer chunk i takes, kBufs chunks back.  It cannot be given back a second time before
      // chunk i is converted, since the ring has kBufs places at least.
      RingAt at{n_ring}, old{n_ring};
      if (t >= kTeam) {
        at.next();
        old.next();
      }
      for (int i = t / kTeam; i < n_ch; i += kTeams) {
        const int st = at.st, buf = i & (kBufs - 1);
        const bool seen = wait(&sh.full[st], at.parity, 2, i) && (i < kBufs || wait(&sh.empty[old.st], old.parity, 2, i));
        if (!__all_sync(0xffffffffu, seen)) break;      // as in warp_wait, one vote for both
        tc_fence_after();
        const uint8_t* src = ring + st * stage_bytes + xbytes;
        // all loads before the first store to tensor memory, which no later load passes
        constexpr int kGroups = kKc / 16;
        Narrow<kFmt == 0 ? 1 : kFmt> w[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g)
          w[g].load(src, N, min(row, N - 1), g);
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          uint32_t o[8];
          w[g].widen(o);
          tmem_st8(to + buf * (kKc / 2) + g * 8, o);
        }
        tmem_st_wait();
        tc_fence_before();
        fence_proxy_async_smem();      // the place's next weights come through the other proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.ready[st]);   // one arrival per warp: one per thread would queue on the barrier's word
        at.next();
        at.next();
        if (i >= kBufs) {
          old.next();
          old.next();
        }
      }
    }
    grid_dep_wait();
  }
  __syncwarp();
  // lane 0 of warp 1 saw the last commit: the accumulators are complete, and the rings free, in every CTA of the cluster
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  tc_fence_after();
  const bool failed = sh.fail != 0 || sh.skip != 0;
  const uint32_t tile = smem_u32(ring);
  const int nb = s.Bpad / splits;                    // rows this CTA finishes: a power of two
  if (warp >= 2 && !failed) {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int b = quarter * 32 + lane, ng = N >> 4;
    if (kFmt != 0) {
      // A lane has a weight row, its columns the rows.
      const int n = quarter * 32 + lane;
      for (int g = half; g < s.Bpad / 16; g += 2) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(g * 16), r);
        if (n < N) {
          if (splits == 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) st_shared1(tile_at(tile, 0, nb, n >> 2, g * 16 + j) + (uint32_t)(n & 3) * 4u, r[j]);
          } else if (nb >= 4) {
            send_pieces<4>(r, tile, rank, nb, g * 16, n);
          } else {
            send_pieces<2>(r, tile, rank, nb, g * 16, n);
          }
        }
        __syncwarp();
      }
    } else if (quarter * 32 < s.Bpad) {
      for (int gi = half ? (ng + 1) / 2 : 0; gi < (half ? ng : (ng + 1) / 2); ++gi) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(gi * 16), r);
        if (b < s.Bpad) {
          const uint32_t at = tile_at(tile, rank, nb, gi * 4, b & (nb - 1)), step = (uint32_t)(nb + 1) * 16u;
          const uint32_t to = splits > 1 ? peer_smem(at, (uint32_t)(b / nb)) : at;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (splits > 1) st_cluster4(to + j * step, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            else st_shared4(to + j * step, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          }
        }
        __syncwarp();      // at 16 rows half a warp has none: it comes back before the next load of all lanes
      }
    }
    tc_fence_before();
  }
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }

  // ---- epilogue: this CTA finishes Bpad / splits of the rows, all columns of the block
  if (warp >= 2 && !failed) {
    const int t = tid - 64;
    const int b_lo = rank * nb;
    const uint8_t* sums = ring;       // laid out as tile_at has it, from `parts` sources
    int parts = splits;
    if (kFmt != 0 && splits > 1) {
      uint8_t* to = ring + s.Bpad * kBlk * 4;
      if (nb >= 4) sum_pieces<4>(to, ring, splits, nb, N, t);
      else sum_pieces<2>(to, ring, splits, nb, N, t);
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      sums = to;
      parts = 1;
    }
    const float* scales = reinterpret_cast<const float*>(s.scales);
    if (s.mode == VDC_STAGE_QKV) {
      for (int bl = warp - 2; bl < nb; bl += kEpiThreads / 32)
        if (b_lo + bl < s.B) qkv_head(s, sums, parts, nb, bl, b_lo + bl, block, lane);
    } else {
      const int bl = t & (nb - 1), b = b_lo + bl;      // nb is a power of two, at most 128
      const int f0 = t / nb, fstep = kEpiThreads / nb;
      if (b < s.B) {
        if (s.mode == VDC_STAGE_RESID) {
          float ssq = 0.f;
          for (int f = f0; f < N / 8; f += fstep) {
            float v[8];
            sum8(v, sums, parts, nb, bl, f * 8);
            scale8(v, scales ? scales + n0 + f * 8 : nullptr);
            uint4* hp = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.hid) + kc_piece(s.Bpad, b, n0 + f * 8));
            const uint4 h = *hp;
            const uint32_t hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[2 * j] = bf16_round(bf_lo(hv[j]) + bf16_round(v[2 * j]));
              v[2 * j + 1] = bf16_round(bf_hi(hv[j]) + bf16_round(v[2 * j + 1]));
              ssq = fmaf(v[2 * j], v[2 * j], fmaf(v[2 * j + 1], v[2 * j + 1], ssq));
            }
            *hp = pack8(v);
          }
          atomicAdd(&sh.ssq[bl], ssq);
        } else if (s.mode == VDC_STAGE_SILU) {
          for (int f = f0; f < N / 16; f += fstep) {
            float o[8];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float v[8];
              sum8(v, sums, parts, nb, bl, f * 16 + h * 8);
              scale8(v, scales ? scales + n0 + f * 16 + h * 8 : nullptr);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float g = bf16_round(v[2 * j]), u = bf16_round(v[2 * j + 1]);
                o[4 * h + j] = bf16_round(g / (1.f + __expf(-g))) * u;
              }
            }
            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + kc_piece(s.Bpad, b, (n0 >> 1) + f * 8)) = pack8(o);
          }
        } else if (s.mode == VDC_STAGE_SUMS) {
          for (int f = f0; f < N / 8; f += fstep) {
            float v[8];
            sum8(v, sums, parts, nb, bl, f * 8);
            scale8(v, scales ? scales + n0 + f * 8 : nullptr);
            float4* to = reinterpret_cast<float4*>(s.out) + (size_t)((n0 >> 2) + f * 2) * s.Bpad + b;
            to[0] = make_float4(v[0], v[1], v[2], v[3]);
            to[s.Bpad] = make_float4(v[4], v[5], v[6], v[7]);
          }
        } else {   // VDC_STAGE_ARGMAX over bf16 logits, the lowest row wins ties
          float best = -INFINITY;
          int row = 0x7fffffff;
          for (int f = f0; f < N / 8; f += fstep) {
            float v[8];
            sum8(v, sums, parts, nb, bl, f * 8);
            scale8(v, scales ? scales + n0 + f * 8 : nullptr);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float l = bf16_round(v[j]);
              if (l > best) {
                best = l;
                row = n0 + f * 8 + j;
              }
            }
          }
          if (row != 0x7fffffff) {
            uint32_t u = __float_as_uint(best);
            u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);   // order-preserving map of the float
            atomicMax(&sh.key[bl], ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)row));
          }
        }
      }
      __syncwarp();
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      if (t < nb && b_lo + t < s.B) {
        if (s.mode == VDC_STAGE_RESID) atomicAdd(reinterpret_cast<float*>(s.stats_out) + b_lo + t, sh.ssq[t]);
        if (s.mode == VDC_STAGE_ARGMAX) atomicMax(reinterpret_cast<unsigned long long*>(s.keys) + b_lo + t, sh.key[t]);
      }
    }
  }
  wait.drain();
  if (warp == 1) tmem_dealloc(tmem, kTmem);
}

// ------------------------------------------------------------------------- //
// attention of a batched step: one row (sequence) and KV head per cluster, its pages shared by the cluster's CTAs
// ------------------------------------------------------------------------- //
// Bound by HBM: 6.1 TB/s at 64 rows and 6.5 TB/s at 128 rows of 2048 positions (the megakernel's units, each walking its
// pages alone with 192 MMAs per page, were bound by the warps at 1.3 us per page and SM).  A page is two bulk copies;
// three of them in flight in each of two CTAs keep 192 KB per SM on their way.
constexpr int kPageBytes = VDC_KV_PAGE * VDC_HEAD_DIM * 2;
constexpr int kAttnRing = 3;
constexpr int kAttnThreads = 160;      // four consumer warps (16 positions of a page each), one producer warp
constexpr int kAttnSmem = kAttnRing * 2 * kPageBytes + 128;
constexpr int kRecLd = VDC_HEAD_DIM + 4;

struct AttnShared {
  uint64_t full[kAttnRing], empty[kAttnRing];
  volatile int fail;
  alignas(16) float m[64], l[64];            // a row's maximum and sum over this CTA's pages
  alignas(16) uint4 zero[16];
  float wm[4][8], wl[4][8];
};

// Producer warp: streams the K and V pages first .. first + count - 1 of one KV head through the ring.  Pages in front of
// `settled` hold no row that the projection in front of this stage writes: their copies start before its end is waited
// for.  (Reading the state blocks that early is safe for the same reason: the stage in front triggers this launch only
// behind its own wait, when everything before it, the last step's advance included, is complete.)  Two layers and a
// 128256-row vocabulary projection: 374 -> 370 us at 3 rows, 501 -> 496 at 32, 558 -> 553 at 64.
__device__ __forceinline__ void stream_pages(AttnShared& sh, const Waiter& wait, uint8_t* ring, const int* table, int first,
                                             int count, const uint8_t* k0, const uint8_t* v0, size_t page_stride, int settled, int lane) {
  int ids = 0;
  bool waited = false;
  for (int i = 0; i < count; ++i) {
    if (!waited && first + i >= settled) {
      grid_dep_wait();
      fence_proxy_async();   // the new cache rows were written with ordinary stores
      waited = true;
    }
    if ((i & 31) == 0) ids = i + lane < count ? ld_relaxed_gpu(table + first + i + lane) : 0;
    const size_t off = (size_t)__shfl_sync(0xffffffffu, ids, i & 31) * page_stride;
    int ok = 1;
    if (lane == 0) {
      const int st = i % kAttnRing;
      if (i >= kAttnRing) ok = wait(&sh.empty[st], (uint32_t)(i / kAttnRing - 1) & 1u, 0, i);
      if (ok) {
        uint8_t* at = ring + st * 2 * kPageBytes;
        mbar_arrive_expect_tx(&sh.full[st], 2 * kPageBytes);
        bulk_load_1d(at, k0 + off, kPageBytes, &sh.full[st]);
        bulk_load_1d(at + kPageBytes, v0 + off, kPageBytes, &sh.full[st]);
      }
    }
    if (!__shfl_sync(0xffffffffu, ok, 0)) break;
  }
  if (!waited) grid_dep_wait();
  grid_dep_launch();
}

// A warp is done with a page.  Its loads (generic proxy) have to be complete before the next bulk copy (async proxy) may
// write there: without the fence the last loads of V, dims 64 and up, could still be on their way when the warp had arrived,
// and when page i + 3 then came in before page i + 1 they read it (a unit in some thousands, 5 % off in the step's hidden
// row).  Fenced by every lane, since each has read for itself, then one arrival for the warp.
__device__ __forceinline__ void page_consumed(uint64_t* empty, int lane) {
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) mbar_arrive(empty);
}

__device__ __forceinline__ void attn_setup(AttnShared& sh, int tid) {
  if (tid == 0) {
    for (int i = 0; i < kAttnRing; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 4);
    }
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid >= 64 && tid < 80) sh.zero[tid - 64] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
}

// The cluster's last step: output rows are sums of the CTAs' unnormalised rows, weighted by their maxima.
// rows: query rows of the tile; row r of this tile is out row `row_b(r)`, head column `row_h(r)`.
template <class Dst>
__device__ __forceinline__ void attn_merge(AttnShared& sh, uint32_t tile, int splits, int rank, int rows, int t, int nt, Dst dst) {
  const uint32_t m_at = smem_u32(sh.m), l_at = smem_u32(sh.l);
  const int per = VDC_HEAD_DIM / 8;
  for (int it = rank * nt + t; it < rows * per; it += splits * nt) {
    const int r = it / per, d = (it % per) * 8;
    // every CTA's share is requested before the first one is used: two remote round trips instead of two per CTA
    float mk[8], m = -INFINITY, den = 0.f, v[8];
    float4 a[8], c[8];
    float lk[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      mk[k] = -INFINITY;
      lk[k] = 0.f;
      a[k] = c[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < splits) {
        mk[k] = ld_cluster1(peer_smem(m_at + r * 4, k));
        lk[k] = ld_cluster1(peer_smem(l_at + r * 4, k));
        const uint32_t p = peer_smem(tile + (uint32_t)(r * kRecLd + d) * 4u, k);
        a[k] = ld_cluster4(p);
        c[k] = ld_cluster4(p + 16);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) m = fmaxf(m, mk[k]);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float w = mk[k] == -INFINITY ? 0.f : exp2f(mk[k] - m);
      den = fmaf(w, lk[k], den);
      v[0] = fmaf(w, a[k].x, v[0]); v[1] = fmaf(w, a[k].y, v[1]); v[2] = fmaf(w, a[k].z, v[2]); v[3] = fmaf(w, a[k].w, v[3]);
      v[4] = fmaf(w, c[k].x, v[4]); v[5] = fmaf(w, c[k].y, v[5]); v[6] = fmaf(w, c[k].z, v[6]); v[7] = fmaf(w, c[k].w, v[7]);
    }
    const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] *= inv;
    uint4* at = dst(r, d);
    if (at != nullptr) *at = pack8(v);
  }
}

__global__ void __launch_bounds__(kAttnThreads, 2) stage_attn(const __grid_constant__ vdc_stage s, int first_unit, vdc_status* status,
                                                              uint64_t timeout_ns) {
  extern __shared__ uint8_t dyn[];
  __shared__ AttnShared sh;
  constexpr int D = VDC_HEAD_DIM;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = s.splits, rank = splits > 1 ? (int)cluster_rank() : 0;
  const int unit = first_unit + (int)blockIdx.x / splits, h = unit % s.n_kv, b = unit / s.n_kv, G = s.group;
  uint8_t* ring = aligned128(dyn);
  const Waiter wait{&sh.fail, status, timeout_ns, s.kind};
  attn_setup(sh, tid);
  const int* st = reinterpret_cast<const int*>(s.state) + (size_t)b * s.state_stride;
  const int pos = ld_relaxed_gpu(st + VDC_ST_POS);
  const int n_pages = min(pos / VDC_KV_PAGE + 1, s.n_pages);
  const int per = (n_pages + splits - 1) / splits, first = rank * per;
  const int count = max(0, min(per, n_pages - first));

  const int gid = lane >> 2, t4 = lane & 3;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[i][j] = 0.f;

  if (warp == 4) {
    const size_t head_off = (size_t)h * kPageBytes;
    stream_pages(sh, wait, ring, st + VDC_ST_PAGETABLE, first, count, reinterpret_cast<const uint8_t*>(s.kpool) + head_off,
                 reinterpret_cast<const uint8_t*>(s.vpool) + head_off, (size_t)s.n_kv * kPageBytes, pos / VDC_KV_PAGE, lane);
  } else {
    grid_dep_wait();
    // S^T = K Q^T and O^T = V^T P^T: the warp's 16 positions (then 16 dims at a time) on the tile's rows, the query
    // heads of the group on its 8 columns.  8 + 8 MMAs per warp and page, none of them on padding for a group of 8.
    uint32_t q[8][2];
    const uint32_t* qp = reinterpret_cast<const uint32_t*>(s.q) + ((size_t)b * s.n_kv * G + (size_t)h * G + gid) * (D / 2) + t4;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k][0] = gid < G ? ldcg32(qp + 8 * k) : 0u;
      q[k][1] = gid < G ? ldcg32(qp + 8 * k + 4) : 0u;
    }
    const float scale_log2 = 1.4426950408889634f * rsqrtf((float)D);
    const uint32_t zero = smem_u32(sh.zero), ring_s = smem_u32(ring);
    const int lr = lane & 7, mi = lane >> 3;
    const int pk = warp * 16 + lr + 8 * (mi & 1), hk = mi >> 1;      // ldmatrix rows of K: position, upper k half
    const int pv = warp * 16 + lr + 8 * (mi >> 1), hv = mi & 1;      // of V (transposed): position, upper dim half
    for (int i = 0; i < count; ++i) {
      const int stg = i % kAttnRing;
      if (!wait.warp_wait(&sh.full[stg], (uint32_t)(i / kAttnRing) & 1u, 1, i)) break;
      const uint32_t kb = ring_s + (uint32_t)(stg * 2 * kPageBytes), vb = kb + kPageBytes;
      const int valid = pos - (first + i) * VDC_KV_PAGE;             // last position that exists, within the page
      float c[4] = {0.f, 0.f, 0.f, 0.f}, c2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        uint32_t a[4], a2[4];
        ldsm_x4(a, kb + (uint32_t)(pk * 256 + (((2 * k + hk) ^ lr) << 4)));
        ldsm_x4(a2, kb + (uint32_t)(pk * 256 + (((2 * k + 2 + hk) ^ lr) << 4)));
        mma_16816(c, a[0], a[1], a[2], a[3], q[k][0], q[k][1]);
        mma_16816(c2, a2[0], a2[1], a2[2], a2[3], q[k + 1][0], q[k + 1][1]);
      }
      // V goes to registers before the softmax, which hides the loads, and the page's place is free that much sooner
      const uint32_t vrow = pv <= valid ? vb + (uint32_t)(pv * 256) : zero;
      uint32_t va[8][4];
#pragma unroll
      for (int d = 0; d < 8; ++d) ldsm_x4_trans(va[d], vrow + (uint32_t)(((2 * d + hv) ^ lr) << 4));
      page_consumed(&sh.empty[stg], lane);
      const int p0 = warp * 16 + gid;
      float e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) e[j] = p0 + 8 * (j >> 1) <= valid ? (c[j] + c2[j]) * scale_log2 : -INFINITY;
      float mx[2] = {fmaxf(e[0], e[2]), fmaxf(e[1], e[3])};
#pragma unroll
      for (int x = 4; x < 32; x <<= 1) {
        mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], x));
        mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], x));
      }
      float al[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float mn = fmaxf(m[j], mx[j]);
        const bool none = mn == -INFINITY;
        al[j] = none ? 1.f : exp2f(m[j] - mn);
        e[j] = none ? 0.f : exp2f(e[j] - mn);
        e[j + 2] = none ? 0.f : exp2f(e[j + 2] - mn);
        m[j] = mn;
        l[j] = l[j] * al[j] + e[j] + e[j + 2];       // this lane's positions only: summed over the lanes at the end
      }
      // probabilities enter P V rounded to bf16, as a bf16 attention module hands them over
      const uint32_t b0 = transpose8x8(pack_bf16x2(e[0], e[1])), b1 = transpose8x8(pack_bf16x2(e[2], e[3]));
#pragma unroll
      for (int d = 0; d < 8; ++d) {
#pragma unroll
        for (int j = 0; j < 4; ++j) o[d][j] *= al[j & 1];
        mma_16816(o[d], va[d][0], va[d][1], va[d][2], va[d][3], b0, b1);
      }
    }
#pragma unroll
    for (int x = 4; x < 32; x <<= 1) {
      l[0] += __shfl_xor_sync(0xffffffffu, l[0], x);
      l[1] += __shfl_xor_sync(0xffffffffu, l[1], x);
    }
    if (gid == 0) {
      sh.wm[warp][2 * t4] = m[0];
      sh.wm[warp][2 * t4 + 1] = m[1];
      sh.wl[warp][2 * t4] = l[0];
      sh.wl[warp][2 * t4 + 1] = l[1];
    }
  }
  __syncthreads();                       // pages are consumed: their shared memory takes the warps' partial outputs
  const bool failed = sh.fail != 0;
  float* part = reinterpret_cast<float*>(ring);                 // [warp][8 heads][kRecLd]
  float* rec = part + 4 * 8 * kRecLd;                           // [head][kRecLd]: this CTA's sum
  if (warp < 4 && !failed) {
#pragma unroll
    for (int d = 0; d < 8; ++d)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        part[(warp * 8 + 2 * t4 + (j & 1)) * kRecLd + d * 16 + gid + 8 * (j >> 1)] = o[d][j];
  }
  __syncthreads();
  if (warp < 4 && !failed) {
    for (int g = 0; g < G; ++g) {
      float mm = -INFINITY;
#pragma unroll
      for (int w = 0; w < 4; ++w) mm = fmaxf(mm, sh.wm[w][g]);
      float sum = 0.f, den = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float wt = sh.wm[w][g] == -INFINITY ? 0.f : exp2f(sh.wm[w][g] - mm);
        sum = fmaf(wt, part[(w * 8 + g) * kRecLd + tid], sum);
        den = fmaf(wt, sh.wl[w][g], den);
      }
      rec[g * kRecLd + tid] = sum;
      if (tid == 0) {
        sh.m[g] = mm;
        sh.l[g] = den;
      }
    }
  }
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp < 4 && !failed)
    attn_merge(sh, smem_u32(rec), splits, rank, G, tid, 128, [&](int r, int d) {
      return reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + kc_piece(s.Bpad, b, (h * G + r) * D + d));
    });
  wait.drain();
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  }
}

// ------------------------------------------------------------------------- //
// attention of a prefill chunk: 64 query rows (64 / G consecutive positions x G heads) of one KV head per cluster
// ------------------------------------------------------------------------- //
constexpr int kRows = 64;

// kWide: the rows are a whole prompt's (up to VDC_WIDE_ROWS), their number and first position in the block `state`; the tiles
// with the longest walks start first.
template <bool kWide>
__global__ void __launch_bounds__(kAttnThreads, 2) stage_attn_prefill(const __grid_constant__ vdc_stage s, int first_unit, vdc_status* status,
                                                                      uint64_t timeout_ns) {
  extern __shared__ uint8_t dyn[];
  __shared__ AttnShared sh;
  constexpr int D = VDC_HEAD_DIM;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = s.splits, rank = splits > 1 ? (int)cluster_rank() : 0;
  const int* st = reinterpret_cast<const int*>(s.state);
  const int unit = first_unit + (int)blockIdx.x / splits, h = unit % s.n_kv, G = s.group, per_tile = kRows / G;
  const int rows = kWide ? ld_relaxed_gpu(st + VDC_WIDE_N) : s.B;
  const int b0 = (kWide ? s.Bpad / per_tile - 1 - unit / s.n_kv : unit / s.n_kv) * per_tile;
  if (kWide && b0 >= rows) return;
  // rounded up as a number: with the registers that known shared memory takes here, 24 bytes are spilled (2048 positions +0.5 %)
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn) + 127) & ~(uintptr_t)127);
  const Waiter wait{&sh.fail, status, timeout_ns, s.kind};
  attn_setup(sh, tid);
  const int pos0 = ld_relaxed_gpu(st + (kWide ? VDC_WIDE_POS : VDC_ST_POS));
  auto row_b = [&](int r) { return min(b0 + r / G, rows - 1); };
  auto pos_of = [&](int r) { return kWide ? pos0 + row_b(r) : ld_relaxed_gpu(st + (size_t)row_b(r) * s.state_stride + VDC_ST_POS); };
  const int pos_hi = pos_of(kRows - 1), pos_lo = pos_of(0);          // the rows' positions never decrease
  const int n_pages = min(pos_hi / VDC_KV_PAGE + 1, s.n_pages);
  const int per = (n_pages + splits - 1) / splits, first = rank * per;
  const int count = max(0, min(per, n_pages - first));

  const int gid = lane >> 2, t4 = lane & 3;
  const int r0 = warp * 16 + gid;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[i][j] = 0.f;

  if (warp == 4) {
    const size_t head_off = (size_t)h * kPageBytes;
    stream_pages(sh, wait, ring, st + VDC_ST_PAGETABLE, first, count, reinterpret_cast<const uint8_t*>(s.kpool) + head_off,
                 reinterpret_cast<const uint8_t*>(s.vpool) + head_off, (size_t)s.n_kv * kPageBytes, pos0 / VDC_KV_PAGE, lane);
  } else {
    grid_dep_wait();
    uint32_t q[8][4];
    const int pos[2] = {pos_of(r0), pos_of(r0 + 8)};
    const uint32_t* qa = reinterpret_cast<const uint32_t*>(s.q) + ((size_t)row_b(r0) * s.n_kv * G + (size_t)h * G + r0 % G) * (D / 2) + t4;
    const uint32_t* qb = reinterpret_cast<const uint32_t*>(s.q) + ((size_t)row_b(r0 + 8) * s.n_kv * G + (size_t)h * G + (r0 + 8) % G) * (D / 2) + t4;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      q[k][0] = ldcg32(qa + 8 * k);
      q[k][1] = ldcg32(qb + 8 * k);
      q[k][2] = ldcg32(qa + 8 * k + 4);
      q[k][3] = ldcg32(qb + 8 * k + 4);
    }
    const float scale_log2 = 1.4426950408889634f * rsqrtf((float)D);
    const uint32_t zero = smem_u32(sh.zero), ring_s = smem_u32(ring);
    const int lr = lane & 7, mi = lane >> 3;
    for (int i = 0; i < count; ++i) {
      const int stg = i % kAttnRing;
      if (!wait.warp_wait(&sh.full[stg], (uint32_t)(i / kAttnRing) & 1u, 1, i)) break;
      const uint32_t kb = ring_s + (uint32_t)(stg * 2 * kPageBytes), vb = kb + kPageBytes;
      const int page0 = (first + i) * VDC_KV_PAGE;
      float c[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[n][j] = 0.f;
#pragma unroll
      for (int k = 0; k < 8; k += 2)
#pragma unroll
        for (int n = 0; n < 8; ++n) {         // one load: eight positions, dims 32 (k / 2) .. + 31
          uint32_t a[4];
          ldsm_x4(a, kb + (uint32_t)((n * 8 + lr) * 256 + (((2 * k + mi) ^ lr) << 4)));
          mma_16816(c[n], q[k][0], q[k][1], q[k][2], q[k][3], a[0], a[1]);
          mma_16816(c[n], q[k + 1][0], q[k + 1][1], q[k + 1][2], q[k + 1][3], a[2], a[3]);
        }
      // Four instructions per score (maximum, fused scale and subtraction, exponential, sum) and nothing that only some pages
      // need: the mask at the diagonal, the rows' rescaling when a maximum moved.  The walk is bound by instructions issued
      // (two warps per scheduler): 2048 positions 178 -> 167 us with 1065 -> 840 per warp and page.
      float mx[2] = {-INFINITY, -INFINITY};
      if (page0 + VDC_KV_PAGE - 1 > pos_lo) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (page0 + n * 8 + 2 * t4 + (j & 1) > pos[j >> 1]) c[n][j] = -INFINITY;
      }
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) mx[j >> 1] = fmaxf(mx[j >> 1], c[n][j]);
      float al[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 1));
        mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 2));
        const float mn = fmaxf(m[j], mx[j] * scale_log2);
        al[j] = mn == -INFINITY ? 1.f : exp2_ftz(m[j] - mn);
        m[j] = mn;
        mx[j] = mn == -INFINITY ? 0.f : mn;                           // a row with no key here: every exponent is -inf
      }
      if (__any_sync(0xffffffffu, al[0] != 1.f || al[1] != 1.f)) {
#pragma unroll
        for (int j = 0; j < 2; ++j) l[j] *= al[j];
#pragma unroll
        for (int d = 0; d < 16; ++d)
#pragma unroll
          for (int j = 0; j < 4; ++j) o[d][j] *= al[j >> 1];
      }
      uint32_t p[8][2];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[n][j] = exp2_ftz(fmaf(c[n][j], scale_log2, -mx[j >> 1]));
          l[j >> 1] += c[n][j];
        }
        p[n][0] = pack_bf16x2(c[n][0], c[n][1]);
        p[n][1] = pack_bf16x2(c[n][2], c[n][3]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {            // 16 positions at a time
        const int pv = k * 16 + lr + 8 * (mi & 1);
        const uint32_t vrow = page0 + pv <= pos_hi ? vb + (uint32_t)(pv * 256) : zero;
#pragma unroll
        for (int d = 0; d < 16; d += 2) {      // one load: the positions' dims 8 d .. 8 d + 15
          uint32_t a[4];
          ldsm_x4_trans(a, vrow + (uint32_t)(((d + (mi >> 1)) ^ lr) << 4));
          mma_16816(o[d], p[2 * k][0], p[2 * k][1], p[2 * k + 1][0], p[2 * k + 1][1], a[0], a[1]);
          mma_16816(o[d + 1], p[2 * k][0], p[2 * k][1], p[2 * k + 1][0], p[2 * k + 1][1], a[2], a[3]);
        }
      }
      page_consumed(&sh.empty[stg], lane);
    }
  }
  __syncthreads();
  const bool failed = sh.fail != 0;
  float* rec = reinterpret_cast<float*>(ring);     // [64 rows][kRecLd]
  if (warp < 4 && !failed) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      l[j] += __shfl_xor_sync(0xffffffffu, l[j], 1);
      l[j] += __shfl_xor_sync(0xffffffffu, l[j], 2);
      if (t4 == 0) {
        sh.m[r0 + 8 * j] = m[j];
        sh.l[r0 + 8 * j] = l[j];
      }
#pragma unroll
      for (int d = 0; d < 16; ++d)
        *reinterpret_cast<float2*>(rec + (r0 + 8 * j) * kRecLd + d * 8 + 2 * t4) = make_float2(o[d][2 * j], o[d][2 * j + 1]);
    }
  }
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp < 4 && !failed)
    attn_merge(sh, smem_u32(rec), splits, rank, kRows, tid, 128, [&](int r, int d) -> uint4* {
      const int b = b0 + r / G, col = (h * G + r % G) * D + d;
      if (b >= rows) return nullptr;
      const size_t at = kWide ? (size_t)(b / 128) * 128 * s.n_kv * G * D * 2 + kc_piece(128, b % 128, col) : kc_piece(s.Bpad, b, col);
      return reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + at);
    });
  wait.drain();
  if (splits > 1) {
    cluster_arrive();
    cluster_wait();
  }
}

// ------------------------------------------------------------------------- //
// first and last kernel of a step
// ------------------------------------------------------------------------- //
// Behind an error that the host has not read yet a step writes nothing that outlives it: the embedding, the projections'
// epilogues and the advance return, so that no state moves on past the failed step.

// Embedding row of one sequence: the hidden state and its sum of squares; and zeros for the sums that the step's residual
// adds accumulate.  An id outside the table (M rows, 0: only its sign is known) is reported and row 0 taken in its place.
__global__ void __launch_bounds__(256) stage_embed(const __grid_constant__ vdc_stage s, int first_row, vdc_status* status) {
  __shared__ float red[8];
  const int b = first_row + (int)blockIdx.x, tid = threadIdx.x;
  grid_dep_wait();
  grid_dep_launch();
  int token = ld_relaxed_gpu(reinterpret_cast<const int*>(s.state) + (size_t)b * s.state_stride + VDC_ST_TOKEN);
  if (__syncthreads_or(ld_relaxed_gpu(&status->abort))) return;
  if (token < 0 || (s.M > 0 && token >= s.M)) {
    if (tid == 0) report(status, VDC_ERR_TOKEN, s.kind, 0, b, token);
    token = 0;
  }
  const uint8_t* row = reinterpret_cast<const uint8_t*>(s.w) + (size_t)token * s.K * 2;
  float ssq = 0.f;
  for (int p = tid; p < s.K / 8; p += 256) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(row) + p);
    const uint32_t xv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) ssq = fmaf(bf_lo(xv[j]), bf_lo(xv[j]), fmaf(bf_hi(xv[j]), bf_hi(xv[j]), ssq));
    *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.hid) + kc_piece(s.Bpad, b, p * 8)) = v;
  }
  ssq = warp_sum(ssq);
  if ((tid & 31) == 0) red[tid >> 5] = ssq;
  __syncthreads();
  float* stats = reinterpret_cast<float*>(s.stats_out);
  if (tid == 0) {
    float t = 0.f;
    for (int w = 0; w < 8; ++w) t += red[w];
    stats[b] = t;
  }
  for (int i = 1 + tid; i < s.n_stats; i += 256) stats[(size_t)i * 128 + b] = 0.f;
}

// RMSNorm of the hidden rows into a matrix of their own, rounded like a bf16 tensor expression: bf16(w * bf16(x * rstd)).
// A stage of its own, once per projection, instead of in every block of the projection that reads the rows: two layers and
// a 128256-row vocabulary projection 382 -> 374 us at 3 rows, 617 -> 574 at 64, 1070 -> 821 at 128 (normalising inside
// the projection, a block's warps rewrote every chunk in shared memory between its arrival and the tensor cores).
__global__ void __launch_bounds__(256) stage_norm(const __grid_constant__ vdc_stage s, int first_block) {
  const int p = (first_block + (int)blockIdx.x) * 256 + (int)threadIdx.x;      // 16-byte piece: eight inputs of one row
  const int k8 = p / s.Bpad, b = p & (s.Bpad - 1);
  const bool live = k8 < s.K / 8;
  const uint4 w = live ? __ldg(reinterpret_cast<const uint4*>(s.norm_w) + k8) : make_uint4(0u, 0u, 0u, 0u);
  grid_dep_wait();
  grid_dep_launch();
  if (!live) return;
  // piece (k8, b) of a k-chunk-major matrix is its p-th piece
  const uint4 v = ldcg128(reinterpret_cast<const uint8_t*>(s.x) + (size_t)p * 16);
  const float rstd = rsqrtf(__ldcg(reinterpret_cast<const float*>(s.stats_in) + b) / (float)s.K + s.eps);
  const uint32_t xv[4] = {v.x, v.y, v.z, v.w}, wv[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    o[j] = pack_bf16x2(bf16_round(bf_lo(xv[j]) * rstd) * bf_lo(wv[j]), bf16_round(bf_hi(xv[j]) * rstd) * bf_hi(wv[j]));
  *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(s.out) + (size_t)p * 16) = make_uint4(o[0], o[1], o[2], o[3]);
}

// Next token, token log and state advance of every sequence.  A row whose logits held no number has no key: that is
// reported, its block marked, and id 0 stored.
__global__ void __launch_bounds__(128) stage_advance(const __grid_constant__ vdc_stage s, vdc_status* status) {
  grid_dep_wait();
  grid_dep_launch();
  const int b = threadIdx.x;
  const bool live = b < s.B;
  int* state = reinterpret_cast<int*>(s.state) + (size_t)(live ? b : 0) * s.state_stride;
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(s.keys);
  const unsigned long long key = live ? __ldcg(keys + b) : 0ull;
  const int step = state[VDC_ST_STEP], pos = state[VDC_ST_POS] + 1, page = pos / VDC_KV_PAGE;
  if (__syncthreads_or(ld_relaxed_gpu(&status->abort)) || !live) return;
  const int token = key != 0ull ? (int)(0xFFFFFFFFu - (uint32_t)(key & 0xFFFFFFFFull)) : 0;
  keys[b] = 0ull;
  reinterpret_cast<int*>(s.log)[(size_t)b * s.log_stride + step] = token;
  state[VDC_ST_TOKEN] = token;
  state[VDC_ST_STEP] = step + 1;
  state[VDC_ST_POS] = pos;
  state[VDC_ST_NPAGES] = page + 1;
  if (page < state[VDC_ST_MAXPAGES])
    state[VDC_ST_NEWROW] = state[VDC_ST_PAGETABLE + page] * VDC_KV_PAGE * state[VDC_ST_NKVH] + pos % VDC_KV_PAGE;
  else
    state[VDC_ST_ERR] = 1;   // out of KV pages: the host must not launch another step
  if (key == 0ull) {
    state[VDC_ST_ERR] = 1;
    report(status, VDC_ERR_TOKEN, s.kind, 0, b, -1);
  }
}

}  // namespace vdc

// ------------------------------------------------------------------------- //
// host entry used by the C ABI
// ------------------------------------------------------------------------- //
extern "C" cudaError_t vdc_stage_prepare() {
  const void* gemms[] = {(const void*)vdc::stage_gemm<0>, (const void*)vdc::stage_gemm<1>, (const void*)vdc::stage_gemm<2>};
  for (const void* f : gemms)
    if (cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, vdc::kGemmSmem)) return e;
  const void* attns[] = {(const void*)vdc::stage_attn, (const void*)vdc::stage_attn_prefill<false>, (const void*)vdc::stage_attn_prefill<true>};
  for (const void* f : attns)
    if (cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, vdc::kAttnSmem)) return e;
  return cudaSuccess;
}

// A stage's grid: `units` of `splits` CTAs each, and how many units one launch takes.
struct Grid {
  int units, splits, slice;
};
static Grid stage_grid(const vdc_stage* s, int max_ctas) {
  const bool attn = s->kind == VDC_STAGE_ATTN || s->kind == VDC_STAGE_ATTN_PREFILL || s->kind == VDC_STAGE_WIDE_ATTN;
  const int tile = attn ? vdc::kRows / s->group : 1;       // rows of a prefill unit
  Grid g{1, s->kind == VDC_STAGE_GEMM || attn ? s->splits : 1, 0};
  switch (s->kind) {
    case VDC_STAGE_GEMM: g.units = (s->M + vdc::kBlk - 1) / vdc::kBlk; break;
    case VDC_STAGE_ATTN: g.units = s->n_kv * s->B; break;
    case VDC_STAGE_ATTN_PREFILL: g.units = s->n_kv * ((s->B + tile - 1) / tile); break;
    case VDC_STAGE_WIDE_ATTN: g.units = s->n_kv * (s->Bpad / tile); break;
    case VDC_STAGE_NORM: g.units = (s->Bpad * (s->K / 8) + 255) / 256; break;
    case VDC_STAGE_EMBED: g.units = s->B; break;
  }
  g.slice = max_ctas ? max_ctas / g.splits : g.units;
  return g;
}

extern "C" void vdc_stage_slices(const vdc_stage* s, int max_ctas, int* launches, int* largest) {
  const Grid g = stage_grid(s, max_ctas);
  *launches = (g.units + g.slice - 1) / g.slice;
  *largest = (g.units < g.slice ? g.units : g.slice) * g.splits;
}

// max_ctas 0: the stage's grid in one launch, with programmatic stream serialisation.  Otherwise at most that many CTAs run
// at any time: the grid goes in slices of whole clusters, and a launch starts early only where it and the one in front of it
// (*front CTAs, -1: not known) fit the limit together.  No third launch joins them: each lets the next one start behind its
// own wait, when the one in front of it has ended.  24 layers of width 512, two rows, on 132 SMs: 1319 us with every launch
// behind the end of the last, 878 us so.
extern "C" cudaError_t vdc_stage_launch(const vdc_stage* s, int max_ctas, int* front, vdc_status* status, uint64_t timeout_ns,
                                        cudaStream_t stream) {
  if (s->kind == VDC_STAGE_COPY) *front = -1;
  if (s->kind == VDC_STAGE_COPY)
    return cudaMemcpyAsync((void*)s->out, (const void*)s->x, (size_t)s->M * s->K, cudaMemcpyDeviceToDevice, stream);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  cfg.stream = stream;
  cfg.attrs = attr;
  const bool gemm = s->kind == VDC_STAGE_GEMM, attn = s->kind == VDC_STAGE_ATTN || s->kind == VDC_STAGE_ATTN_PREFILL || s->kind == VDC_STAGE_WIDE_ATTN;
  const Grid g = stage_grid(s, max_ctas);
  if (g.splits > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)g.splits;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  cudaLaunchAttribute& early = attr[cfg.numAttrs++];
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  cfg.blockDim = dim3(gemm ? vdc::kGemmThreads : attn ? vdc::kAttnThreads : s->kind == VDC_STAGE_ADVANCE ? 128 : 256);
  cfg.dynamicSmemBytes = gemm ? vdc::kGemmSmem : attn ? vdc::kAttnSmem : 0;
  for (int first = 0; first < g.units; first += g.slice) {
    const int ctas = (g.units - first < g.slice ? g.units - first : g.slice) * g.splits;
    cfg.gridDim = dim3((unsigned)ctas);
    early.val.programmaticStreamSerializationAllowed = max_ctas == 0 || (*front >= 0 && *front + ctas <= max_ctas);
    *front = ctas;
    cudaError_t e;
    switch (s->kind) {
      case VDC_STAGE_GEMM: {
        auto f = s->wfmt == 0 ? vdc::stage_gemm<0> : s->wfmt == 1 ? vdc::stage_gemm<1> : vdc::stage_gemm<2>;
        e = cudaLaunchKernelEx(&cfg, f, *s, first, vdc::ring_stages(s->wfmt, s->Bpad), status, timeout_ns);
        break;
      }
      case VDC_STAGE_ATTN: e = cudaLaunchKernelEx(&cfg, vdc::stage_attn, *s, first, status, timeout_ns); break;
      case VDC_STAGE_WIDE_ATTN: e = cudaLaunchKernelEx(&cfg, vdc::stage_attn_prefill<true>, *s, first, status, timeout_ns); break;
      case VDC_STAGE_ATTN_PREFILL: e = cudaLaunchKernelEx(&cfg, vdc::stage_attn_prefill<false>, *s, first, status, timeout_ns); break;
      case VDC_STAGE_NORM: e = cudaLaunchKernelEx(&cfg, vdc::stage_norm, *s, first); break;
      case VDC_STAGE_EMBED: e = cudaLaunchKernelEx(&cfg, vdc::stage_embed, *s, first, status); break;
      case VDC_STAGE_ADVANCE: e = cudaLaunchKernelEx(&cfg, vdc::stage_advance, *s, status); break;
      default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Helpers of the stage kernels: programmatic dependent launch, clusters, bounded waits, the pieces of a projection's epilogue.
#pragma once
#include "mk_umma.cuh"

#include "../../include/vdcores.h"

namespace vdc {

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_smem(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster4(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void st_shared4(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void st_cluster2(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared::cluster.v2.b32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void st_shared1(uint32_t a, uint32_t x) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory"); }
__device__ __forceinline__ float ld_cluster1(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// Dynamic shared memory from its first multiple of 128 bytes.  An offset and no cast, so that the compiler still knows whose memory
// it is: through a pointer rounded up as a number every access would be a generic one.
__device__ __forceinline__ uint8_t* aligned128(uint8_t* dyn) { return dyn + (-(int)smem_u32(dyn) & 127); }

// The first error since the host last looked goes to the status block.
static __device__ void report(vdc_status* status, int code, int kind, int role, int at, int aux) {
  if (atomicCAS(&status->abort, 0, 1) == 0) {
    status->code = code;
    status->sm = (int)blockIdx.x;
    status->role = role;
    status->pc = at;
    status->opcode = kind;
    status->bar = -1;
    status->aux = aux;
    __threadfence();
  }
}

// Bounded wait on an mbarrier of this CTA: after `timeout_ns` the status block says so, the CTA's `fail` word stops
// every other role, and all of them leave through the ordinary exit (cluster barriers and tensor memory included).
static __device__ __noinline__ bool stage_wait_slow(uint64_t* bar, uint32_t parity, volatile int* fail, vdc_status* status,
                                                    uint64_t timeout_ns, int kind, int role, int at) {
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 15u) != 0) continue;
    if (*fail) return false;
    if (globaltimer_ns() - t0 > timeout_ns) {
      report(status, VDC_ERR_TIMEOUT, kind, role, at, (int)it);
      *fail = 1;
      return false;
    }
  }
}

struct Waiter {
  volatile int* fail;
  vdc_status* status;
  uint64_t timeout_ns;
  int kind;
  __device__ __forceinline__ bool operator()(uint64_t* bar, uint32_t parity, int role, int at) const {
    return mbar_try_wait(bar, parity) || stage_wait_slow(bar, parity, fail, status, timeout_ns, kind, role, at);
  }
  // The same for a whole warp: all 32 lanes leave together and with one answer, true only if every lane saw the barrier.
  // What follows such a wait (ldmatrix, mma, full-mask shuffles, one arrival for the warp) needs all lanes.
  __device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int role, int at) const {
    return __all_sync(0xffffffffu, (*this)(bar, parity, role, at));
  }
  // copies that may still be in flight after a wait was given up get a bounded time to land
  __device__ __forceinline__ void drain() const {
    if (*fail) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
  }
};

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 2^x as one instruction: results below the smallest normal number become zero.
__device__ __forceinline__ float exp2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(v));
  return d;
}

// Place in the ring and parity of the phase a role is at.
struct RingAt {
  int n, st = 0;
  uint32_t parity = 0u;
  __device__ __forceinline__ void next() {
    if (++st == n) {
      st = 0;
      parity ^= 1u;
    }
  }
};

__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}
__device__ __forceinline__ void scale8(float (&v)[8], const float* sc) {
  if (sc != nullptr) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(sc)), c = __ldg(reinterpret_cast<const float4*>(sc) + 1);
    v[0] *= a.x; v[1] *= a.y; v[2] *= a.z; v[3] *= a.w;
    v[4] *= c.x; v[5] *= c.y; v[6] *= c.z; v[7] *= c.w;
  }
}

// Bytes of a chunk of n weight rows x 64 inputs as stored: bf16, e4m3, or e2m1 pairs with one e4m3 scale per 16.
__host__ __device__ constexpr int chunk_bytes(int wfmt, int n) { return wfmt == 0 ? n * 128 : wfmt == 1 ? n * 64 : n * 36; }

// 16 weights of a row (inputs 16 g16 .. + 15 of a chunk of N rows) as stored, and as bf16 (exact for e4m3 and for e2m1 code times
// block scale).
template <int kFmt>
struct Narrow {
  uint32_t v[kFmt == 1 ? 4 : 2], scale;
  __device__ __forceinline__ void load(const uint8_t* src, int N, int row, int g16) {
    if constexpr (kFmt == 1) {
      const uint4 w = lds128(src + (g16 * N + row) * 16);
      v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
    } else {
      const uint8_t* g = src + g16 * 9 * N;
      const uint2 w = *reinterpret_cast<const uint2*>(g + row * 8);
      v[0] = w.x; v[1] = w.y;
      scale = g[8 * N + row];
    }
  }
  __device__ __forceinline__ void widen(uint32_t (&o)[8]) const {
    if constexpr (kFmt == 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 lo = e4m3x2_to_float2(v[j] & 0xFFFFu), hi = e4m3x2_to_float2(v[j] >> 16);
        o[2 * j] = pack_bf16x2(lo.x, lo.y);
        o[2 * j + 1] = pack_bf16x2(hi.x, hi.y);
      }
    } else {
      // Conversions of a quarter (e2m1) and half of a pipe's rate.  Nine integer instructions for eight codes instead (byte
      // permutations whose selectors the packed codes are) are slower: two layers of 16 rows 291 us, 304 with those.
      const __half_raw hr = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)scale, __NV_E4M3);
      const __half2 sc = __half2half2(*reinterpret_cast<const __half*>(&hr));
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t h[4];
        e2m1x8_to_half2(v[j], h);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __half22float2(__hmul2(*reinterpret_cast<const __half2*>(&h[i]), sc));
          o[4 * j + i] = pack_bf16x2(f.x, f.y);
        }
      }
    }
  }
};
// The same as pieces of the tensor cores' operand layout in shared memory.
template <int kFmt>
__device__ __forceinline__ void widen16(uint8_t* dst, const uint8_t* src, int N, int row, int g16) {
  uint32_t o[8];
  Narrow<kFmt> w;
  w.load(src, N, row, g16);
  w.widen(o);
  *reinterpret_cast<uint4*>(dst + ((2 * g16) * N + row) * 16) = make_uint4(o[0], o[1], o[2], o[3]);
  *reinterpret_cast<uint4*>(dst + ((2 * g16 + 1) * N + row) * 16) = make_uint4(o[4], o[5], o[6], o[7]);
}

// One head of one row of the QKV projection, one warp: optional RMSNorm over the head, half-rotation, then a query row to
// the query matrix or (append) a key / value row to cache row new_row.  Every product is rounded as a bf16 tensor expression
// rounds it.  Lane i holds dims 2i, 2i+1 and their rotation partners 64 further.
__device__ __forceinline__ void head_row(const vdc_stage& s, float (&x)[4], int b, int block, int lane, int pos, int new_row,
                                         bool append) {
  constexpr int D = VDC_HEAD_DIM;
  const int G = s.group, kvh = block / (G + 2), part = block % (G + 2);
  const int i0 = lane * 2;
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = bf16_round(x[j]);
  if (part <= G) {   // a query head or the key head
    if (s.qk_norm) {
      const float ss = warp_sum(x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3]);
      const float rs = rsqrtf(ss / (float)D + s.qk_eps);
      const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(s.qk_norm) + (part == G ? D : 0);
      const uint32_t wl = *reinterpret_cast<const uint32_t*>(w + i0), wh = *reinterpret_cast<const uint32_t*>(w + i0 + 64);
      x[0] = bf16_round(bf_lo(wl) * bf16_round(x[0] * rs));
      x[1] = bf16_round(bf_hi(wl) * bf16_round(x[1] * rs));
      x[2] = bf16_round(bf_lo(wh) * bf16_round(x[2] * rs));
      x[3] = bf16_round(bf_hi(wh) * bf16_round(x[3] * rs));
    }
    const float* rope = reinterpret_cast<const float*>(s.rope) + (size_t)pos * D;
    const float2 cs = __ldg(reinterpret_cast<const float2*>(rope + i0));
    const float2 sn = __ldg(reinterpret_cast<const float2*>(rope + 64 + i0));
    const float a0 = x[0], a1 = x[1], b0 = x[2], b1 = x[3];
    x[0] = bf16_round(a0 * cs.x) - bf16_round(b0 * sn.x);
    x[1] = bf16_round(a1 * cs.y) - bf16_round(b1 * sn.y);
    x[2] = bf16_round(b0 * cs.x) + bf16_round(a0 * sn.x);
    x[3] = bf16_round(b1 * cs.y) + bf16_round(a1 * sn.y);
  }
  const uint32_t lo = pack_bf16x2(x[0], x[1]), hi = pack_bf16x2(x[2], x[3]);
  if (part < G) {
    uint32_t* dst = reinterpret_cast<uint32_t*>(s.out) + ((size_t)b * s.n_kv * G + (size_t)kvh * G + part) * (D / 2) + lane;
    dst[0] = lo;
    dst[32] = hi;
    return;
  }
  if (!append) return;
  // the row's 16-byte pieces lie at (piece XOR (row mod 8)), the page-row order the attention reads
  const int sw = pos & 7;
  uint8_t* row = reinterpret_cast<uint8_t*>(part == G ? s.kpool : s.vpool) + (size_t)kvh * (VDC_KV_PAGE * D * 2) +
                 (size_t)new_row * (D * 2);
  *reinterpret_cast<uint32_t*>(row + (((i0 >> 3) ^ sw) << 4) + (i0 & 7) * 2) = lo;
  *reinterpret_cast<uint32_t*>(row + (((8 + (i0 >> 3)) ^ sw) << 4) + (i0 & 7) * 2) = hi;
}

}  // namespace vdc

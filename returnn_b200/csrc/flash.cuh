// Building blocks of the fused attention kernels (sdpa_flash.cu, rel_pos_flash.cu): [128, 64] operand tiles in shared memory (128-byte
// swizzle), products of 64-wide tiles, rows of tensor memory in registers, and the life of a CTA (barriers, tensor memory, abort flag).
#pragma once
#include "tcgen05.cuh"

namespace rbf {

using namespace rbt;

constexpr int kRows = 128;   // rows of a CTA
constexpr int kTile = 64;    // width of a score tile, and the head dim
constexpr int kBig = kRows * 128;   // bytes of a [128, 64] bf16 tile
constexpr int kSmall = kTile * 128;  // ... [64, 64]
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void tmem_ld64(uint32_t addr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  tmem_ld32(addr, r);
  tmem_ld32(addr + 32, r + 32);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// 64 values -> row `row` of a swizzled [rows, 64] bf16 tile
__device__ __forceinline__ void store_row64(uint8_t* tile, int row, const float* v) {
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    *reinterpret_cast<uint4*>(tile + row * 128 + ((c ^ (row & 7)) << 4)) =
        make_uint4(pack2(v[8 * c], v[8 * c + 1]), pack2(v[8 * c + 2], v[8 * c + 3]), pack2(v[8 * c + 4], v[8 * c + 5]), pack2(v[8 * c + 6], v[8 * c + 7]));
  }
}

// 64 values -> row `row` of two swizzled [rows, 32] fp32 tiles of kBig bytes, one behind the other (columns 0 .. 31 and 32 .. 63)
__device__ __forceinline__ void store_row64_f32(uint8_t* tile, int row, const float* v) {
#pragma unroll
  for (int c = 0; c < 16; ++c)
    *reinterpret_cast<float4*>(tile + (c >> 3) * kBig + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}

// product of row `row` of two such fp32 tiles with that of a bf16 tile, both [rows, 64]
__device__ __forceinline__ float dot_row64(const uint8_t* f32, const uint8_t* bf, int row) {
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint4 b = *reinterpret_cast<const uint4*>(bf + row * 128 + ((j ^ (row & 7)) << 4));
    const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c = (2 * j + half) & 7;
      const float4 a = *reinterpret_cast<const float4*>(f32 + (j >> 2) * kBig + row * 128 + ((c ^ (row & 7)) << 4));
      s = fmaf(a.x, __uint_as_float(w[2 * half] << 16), s);
      s = fmaf(a.y, __uint_as_float(w[2 * half] & 0xffff0000u), s);
      s = fmaf(a.z, __uint_as_float(w[2 * half + 1] << 16), s);
      s = fmaf(a.w, __uint_as_float(w[2 * half + 1] & 0xffff0000u), s);
    }
  }
  return s;
}

// barriers, tensor memory and the abort flag of a CTA
struct Cta {
  uint64_t* full;    // [2] loads of a stage
  uint64_t* done;    // products of an iteration
  uint64_t* extra;   // one more load
  uint32_t tmem;
  volatile int* abort_flag;
};

template <uint32_t COLS>
__device__ __forceinline__ Cta cta_begin(uint8_t* tail) {
  Cta c;
  c.full = reinterpret_cast<uint64_t*>(tail);
  c.done = c.full + 2;
  c.extra = c.full + 3;
  uint32_t* slot = reinterpret_cast<uint32_t*>(c.full + 4);
  c.abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(c.full + i, 1);
    *c.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  c.tmem = *slot;
  return c;
}

template <uint32_t COLS>
__device__ __forceinline__ void cta_end(const Cta& c) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*c.abort_flag && threadIdx.x == 0) {
    for (uint32_t i = 0; i < (1u << 12); ++i) __nanosleep(256);  // copies still in flight land before the shared memory goes away
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(COLS) : "memory");
  }
}

__device__ __forceinline__ void mbar_arrive_local(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait; a wait that gives up marks the CTA and the status word
__device__ __forceinline__ bool wait_or_abort(const Cta& c, uint64_t* bar, uint32_t parity, int* status, int code) {
  const bool ok = mbar_wait(bar, parity, c.abort_flag);
  if (!ok) {
    *c.abort_flag = 1;
    if (status) atomicCAS(status, 0, (8 << 24) | code);
  }
  return ok;
}

// ---- life of a CTA with warps of rows and one that issues ---------------------------------------------------------------------------
// The warp behind those of the rows issues loads and products; the rows' warps meet it at mbarriers and each other nowhere. Scores
// are in registers as soon as they are read, so the products of the next tile run while the row work of this one does. With thread 0 issuing
// between barriers of the whole CTA, a tile was product (1000 to 1400 cycles), row work, barrier (500), one after the other: 3600, 2800 and 4500
// cycles in the three kernels.
struct Pipe {
  Cta c;
  uint64_t *scores, *out, *taken, *put;  // scores of a tile are there, products with P / dS are done; rows have taken the scores, put P / dS
};
// WARPS: of rows; OUT: arrivals that complete a phase of `out`
template <uint32_t COLS, int WARPS, int OUT = 1>
__device__ __forceinline__ Pipe pipe_begin(uint8_t* tail) {
  Pipe p;
  p.c.full = reinterpret_cast<uint64_t*>(tail);
  p.c.extra = p.c.full + 2;
  p.scores = p.c.full + 3;
  p.c.done = p.out = p.c.full + 4;
  p.taken = p.c.full + 5;
  p.put = p.c.full + 6;
  uint32_t* slot = reinterpret_cast<uint32_t*>(p.c.full + 7);
  p.c.abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 7; ++i) mbar_init(p.c.full + i, i >= 5 ? WARPS : i == 4 ? OUT : 1);
    *p.c.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  p.c.tmem = *slot;
  return p;
}
// all lanes of a warp: the wait of one that gave up is the wait of all
__device__ __forceinline__ bool pipe_wait(const Pipe& p, uint64_t* bar, int phase, int* status, int code) {
  const bool ok = __all_sync(0xffffffffu, wait_or_abort(p.c, bar, phase & 1, status, code));
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return ok;
}
// D[128, 64] (+)= A[128, 64] B by one lane of a converged warp: A K-major; B K-major [n, k] or, `B_MN`, stored [k, n]
template <bool B_MN>
__device__ __forceinline__ void mma64_warp(uint32_t d, const uint8_t* a, const uint8_t* b, bool accumulate) {
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  const uint32_t da = desc_lo(smem_u32(a), 16), db = desc_lo(smem_u32(b), B_MN ? 8192 : 16);
  umma_f16_warp(d, da, db, idesc, accumulate ? 1u : 0u);
#pragma unroll
  for (int kk = 1; kk < 4; ++kk) umma_f16_warp(d, da + 2 * kk, db + (B_MN ? 128 : 2) * kk, idesc, 1u);
}
// a warp of rows is through with its accesses to tensor memory and shared memory (those to the latter made visible by each lane before)
__device__ __forceinline__ void pipe_arrive(uint64_t* bar) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive_local(bar);
}
template <int THREADS>
__device__ __forceinline__ void rows_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}
// The issuing warp, over n tiles: `load(t)` into stage t & 1 (its barrier: full[t & 1]), `first(t)` products that give scores, `second(t)` those with
// what the rows have put, `after(t)` what else is to be done with that. Tiles 0 and 1 are being loaded.
template <typename Load, typename First, typename Second, typename After>
__device__ __forceinline__ void pipe_issue(const Pipe& p, int n, int* status, Load load, First first, Second second, After after) {
  bool ok = pipe_wait(p, &p.c.full[0], 0, status, 1);
  if (ok) {
    first(0);
    umma_commit_warp(p.scores);
  }
  for (int t = 0; t < n && ok; ++t) {
    if (t + 1 < n) {
      ok = pipe_wait(p, p.taken, t, status, 2) && pipe_wait(p, &p.c.full[(t + 1) & 1], (t + 1) >> 1, status, 3);
      if (!ok) break;
      first(t + 1);
      umma_commit_warp(p.scores);
    }
    ok = pipe_wait(p, p.put, t, status, 4);
    if (!ok) break;
    second(t);
    umma_commit_warp(p.out);
    after(t);
    if (t + 2 < n) {
      ok = pipe_wait(p, p.out, t, status, 5);  // stage t & 1 has been read
      if (ok) load(t + 2);
    }
  }
}

// The same with tile t + 2 being loaded while tile t's rows are at work, not after: what only `first` reads has two places, what `second` reads three.
template <typename Load, typename First, typename Second, typename After>
__device__ __forceinline__ void pipe_issue_ahead(const Pipe& p, int n, int* status, Load load, First first, Second second, After after) {
  bool ok = pipe_wait(p, &p.c.full[0], 0, status, 1);
  if (ok) {
    first(0);
    umma_commit_warp(p.scores);
  }
  for (int t = 0; t < n && ok; ++t) {
    if (t + 1 < n) {
      ok = pipe_wait(p, p.taken, t, status, 2) && pipe_wait(p, &p.c.full[(t + 1) & 1], (t + 1) >> 1, status, 3);
      if (!ok) break;
      first(t + 1);
      umma_commit_warp(p.scores);
    }
    if (t + 2 < n) {  // the products of tile t that give scores and all of tile t - 1 are done
      ok = t == 0 || pipe_wait(p, p.out, t - 1, status, 5);
      if (!ok) break;
      load(t + 2);
    }
    ok = pipe_wait(p, p.put, t, status, 4);
    if (!ok) break;
    second(t);
    umma_commit_warp(p.out);
    after(t);
  }
}

// The output of a forward pass stays in tensor memory; where a row's maximum grows, the warp takes its rows of the output out, scales them and puts them
// back, in every tile and by any amount: P refers to the exact maximum, so that the largest weight of a row is 1 and is not rounded. (A maximum that
// lags by up to 2^8 spares most of that, but rounds the largest weight too, an error common to the row that the sum of the weights, taken before the
// rounding, does not have: the output of peaked rows was off by 2^-9, three times as much as with the exact maximum.)
__device__ __forceinline__ void tmem_scale64(uint32_t addr, float factor) {
#pragma unroll 1
  for (int part = 0; part < 4; ++part) {
    uint32_t o[16];
    tmem_ld16(addr + 16 * part, o);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * factor);
    tmem_st16(addr + 16 * part, o);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

}  // namespace rbf

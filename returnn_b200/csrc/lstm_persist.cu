// Persistent LSTM recurrence: ONE kernel runs all T steps of a direction. The recurrent matrix never leaves the chip: CTA c
// keeps the rows of W_rec that produce the four gates of its hidden units in shared memory (forward), or the columns
// that those units feed (backward), for the whole sequence. Per step a CTA multiplies the small [B, K] activation matrix (read
// from L2, where the other CTAs wrote it in the previous step) with its resident slice on the tensor cores, applies the cell
// for its units, publishes its slice of h_t (or dz_t) and waits for those of the others. The per-step executor in lstm.cu needs two
// launches of latency-bound kernels per step (about 22 us); here a step of both directions, forward and backward together, takes about 7.4 us
// (16 rows, H = 1024; 9.6 with flags and a barrier in front of the backward step's fetch, 17.5 with 128 narrow CTAs per direction that met at a
// counter after storing what the backward pass keeps).
//
// The step product has only B <= 48 rows: the warp-level mma (m16n8k16, bf16 -> fp32) fits this shape (three 16-row tiles);
// a tcgen05 tile is at least 64 rows by one CTA and its operands would have to be re-staged through TMA every step. The
// warps of a CTA split the contraction; their partial sums meet in shared memory.
//
// Launched cooperatively (all CTAs resident). Every wait is bounded: a CTA that gives up raises the abort word, all
// CTAs leave the time loop, and the host reports RB_ERR_TIMEOUT.
//
// Semantics, gate order (i, f, g, o), masking and the tensors saved for backward are those of lstm.cu
// (reference: returnn/native_op.py:1029-1179 NativeLstm2, returnn/torch/frontend/_backend.py:2796-2810).
#include "common.cuh"
#include "gemm.h"
#include <cooperative_groups.h>

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kMaxRows = 48;   // batch rows (three m16 tiles)
constexpr int kPad = 32;       // row padding of the resident slice: pitch = 64 bytes mod 128 (conflict-free 16-byte fragment loads)
constexpr int kRedPad = 8;      // row padding of the partial-sum slots
constexpr int kMaxCtas = 160;   // CTAs of one direction
constexpr uint32_t kSpinLimit = 1u << 22;

// How a direction is spread over the GPU: U hidden units per CTA, W warps that split the contraction, room for 16 * MT batch rows.
// Narrow: two CTAs per SM for the two directions of a layer (one direction: one per SM). Wide: one CTA per SM with twice the units. All
// CTAs read the whole exchanged matrix in every step, so half the CTAs halve that L2 traffic (H = 1024, 16 rows, backward: 17 instead of
// 34 MB per step) and the flags of a barrier, and with 16 warps a warp has all of its operand loads in flight at once. Three row tiles do
// not fit the 128 registers of a 512-thread CTA: batches above 32 rows take the narrow form.
template <int UNITS, int WARPS, int TILES, int PF_FWD, int PF_BWD>
struct Shape {
  static constexpr int U = UNITS, W = WARPS, MT = TILES, Threads = 32 * WARPS, Rows = 16 * TILES, Slots = WARPS / 2;
  static constexpr int PrefetchFwd = PF_FWD, PrefetchBwd = PF_BWD;  // blocks of 32 k whose loads a warp has in flight
  static constexpr int PerThread = (Rows * UNITS + Threads - 1) / Threads;  // (row, unit) pairs of a thread
};
using Narrow = Shape<8, 8, 3, 4, 4>;
using NarrowPair = Shape<8, 8, 3, 2, 2>;
using Wide1 = Shape<16, 16, 1, 2, 8>;
using Wide2 = Shape<16, 16, 2, 2, 4>;

__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + __expf(-x)); }

__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Barrier of the CTAs of one direction, in two halves: a CTA announces that its slice of the exchanged matrix is written by storing the
// step number into its own flag word (no atomic: adds of all CTAs onto one counter are served one after the other), does what the others
// need not wait for, and then waits for all flags, one thread per flag. Only the exchanged slice is stored before the announcement, so the
// fence in it does not wait for the tensors that are kept for the backward pass.
// Narrow form with more than kFlagCtas CTAs (H > 512): all CTAs add onto one counter instead, and one thread of each looks at it with pauses.
// 128 threads in each of up to 256 CTAs that read flags all the time take the issue slots of the other CTA of their SM and the L2 requests of
// the operand loads: H = 1024, T = 100, one direction, 16 rows, forward 760 us with flags, 566 with the counter; both directions, 33 rows,
// training 3409 and 2480. Up to 64 CTAs the flags are ahead: one direction, H = 512, 16 rows, forward 428 and 460.
constexpr int kFlagCtas = 64;

template <typename S>
__device__ __forceinline__ bool counts(int n_cta) {
  return S::U == 8 && n_cta > kFlagCtas;
}

template <typename S>
__device__ __forceinline__ void barrier_arrive(uint32_t* flags, int cta, int n_cta, uint32_t step) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (counts<S>(n_cta)) atomicAdd(flags, 1u);
    else asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(flags + cta), "r"(step) : "memory");
  }
}
// false (for every thread of every CTA, eventually) when someone timed out
template <typename S>
__device__ __forceinline__ bool barrier_wait(uint32_t* flags, int n_cta, uint32_t step, int* abort_word, int* status) {
  const bool count = counts<S>(n_cta);
  const uint32_t target = count ? step * (uint32_t)n_cta : step;
  int ok = 1;
  if ((int)threadIdx.x < (count ? 1 : n_cta)) {
    uint32_t spins = 0;
    while ((int32_t)(ld_relaxed_gpu(flags + threadIdx.x) - target) < 0) {
      ++spins;
      if (count) __nanosleep(64);
      if (spins > kSpinLimit || ((spins & 255u) == 0 && *reinterpret_cast<volatile int*>(abort_word))) {
        ok = 0;
        atomicExch(abort_word, 1);
        if (status) atomicCAS(status, 0, (5 << 24) | (int)(blockIdx.x & 0xFFFF));
        break;
      }
    }
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

template <typename S, int NOUT>
__device__ __forceinline__ void store_partials(float (&acc)[S::MT][NOUT / 8][4], int m_tiles, float* __restrict__ red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  // The partial sums of the warps meet in shared memory without atomics (warps adding 48 values per lane onto the
  // same words was the largest batch-dependent part of a forward step): the upper half of the warps store theirs into slot warp - W/2, the
  // lower half add their own onto that slot, the caller sums the W/2 slots (red_sum). Row pitch NOUT + 8 floats: the 8-byte accesses
  // of a half warp fall on distinct banks.
  constexpr int RP = NOUT + kRedPad;
  float* slot = red + (warp & (S::Slots - 1)) * (S::Rows * RP);
  if (warp >= S::Slots) {
#pragma unroll
    for (int m = 0; m < S::MT; ++m) {
      if (m >= m_tiles) continue;
      const int r0 = m * 16 + g, r1 = r0 + 8;
#pragma unroll
      for (int n = 0; n < NOUT / 8; ++n) {
        const int c = n * 8 + 2 * t;
        *reinterpret_cast<float2*>(&slot[r0 * RP + c]) = make_float2(acc[m][n][0], acc[m][n][1]);
        *reinterpret_cast<float2*>(&slot[r1 * RP + c]) = make_float2(acc[m][n][2], acc[m][n][3]);
      }
    }
  }
  __syncthreads();
  if (warp < S::Slots) {
#pragma unroll
    for (int m = 0; m < S::MT; ++m) {
      if (m >= m_tiles) continue;
      const int r0 = m * 16 + g, r1 = r0 + 8;
#pragma unroll
      for (int n = 0; n < NOUT / 8; ++n) {
        const int c = n * 8 + 2 * t;
        float2* q0 = reinterpret_cast<float2*>(&slot[r0 * RP + c]);
        float2* q1 = reinterpret_cast<float2*>(&slot[r1 * RP + c]);
        const float2 v0 = *q0, v1 = *q1;
        *q0 = make_float2(v0.x + acc[m][n][0], v0.y + acc[m][n][1]);
        *q1 = make_float2(v1.x + acc[m][n][2], v1.y + acc[m][n][3]);
      }
    }
  }
}

// red[row][n] += sum_k A[row][k] * Bs[n][k] for rows < n_rows; A in global (written by other CTAs: read through L2), Bs resident
// in shared memory with row pitch K + kPad. The contraction is cut into blocks of 32 k; the warp w of S::W takes the blocks
// [w*nblk/W, (w+1)*nblk/W).
//
// Operand fetch: all CTAs read the same small A matrix at the same time, so the number of L2 requests, not the bytes, sets the
// step time. A lane therefore fetches 16 contiguous bytes (8 k) per row and block instead of four 4-byte fragment words: the
// order of the k inside a block is free as long as A and B agree, so the lane t of a quad owns k [8t, 8t+8) of the block, its
// words 0/1 feed the first m16n8k16 (as the fragment halves "k 2t.." and "k 2t+8..") and its words 2/3 the second one. The B
// fragments come from shared memory with the same 16-byte pattern (row pitch = 64 bytes mod 128: conflict-free quarter warps).
template <typename S, int NOUT, int kPrefetch>
__device__ __forceinline__ void step_matmul(const bf16* __restrict__ A, int n_rows, int K, const bf16* __restrict__ Bs, float* __restrict__ red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int pitch = K + kPad;
  float acc[S::MT][NOUT / 8][4];
#pragma unroll
  for (int m = 0; m < S::MT; ++m)
#pragma unroll
    for (int n = 0; n < NOUT / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
  const int m_tiles = (n_rows + 15) / 16;
  auto load_a = [&](int k0, uint4 (&a)[S::MT][2]) {
#pragma unroll
    for (int m = 0; m < S::MT; ++m) {
      const int r0 = m * 16 + g, r1 = r0 + 8;
      a[m][0] = r0 < n_rows ? __ldcg(reinterpret_cast<const uint4*>(A + (size_t)r0 * K + k0 + 8 * t)) : make_uint4(0u, 0u, 0u, 0u);
      a[m][1] = r1 < n_rows ? __ldcg(reinterpret_cast<const uint4*>(A + (size_t)r1 * K + k0 + 8 * t)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  // chunks of kPrefetch blocks: all operand loads of a chunk are issued before its first multiply, so a chunk costs one L2 round
  // trip (as many as the registers hold: wide, 16 rows: one trip at H = 1024 in both passes; narrow with two CTAs per SM: 2 and 8 trips)
  const int nblk = K >> 5;
  const int b_begin = warp * nblk / S::W, b_end = (warp + 1) * nblk / S::W;
  for (int bc = b_begin; bc < b_end; bc += kPrefetch) {
    uint4 a[kPrefetch][S::MT][2];
#pragma unroll
    for (int i = 0; i < kPrefetch; ++i)
      if (bc + i < b_end) load_a((bc + i) << 5, a[i]);
#pragma unroll
    for (int i = 0; i < kPrefetch; ++i) {
      if (bc + i >= b_end) break;
      const int k0 = (bc + i) << 5;
#pragma unroll
      for (int n = 0; n < NOUT / 8; ++n) {
        const uint4 b = *reinterpret_cast<const uint4*>(Bs + (size_t)(n * 8 + g) * pitch + k0 + 8 * t);
#pragma unroll
        for (int m = 0; m < S::MT; ++m) {
          if (m >= m_tiles) continue;
          const uint32_t f0[4] = {a[i][m][0].x, a[i][m][1].x, a[i][m][0].y, a[i][m][1].y};
          mma16816(acc[m][n], f0, b.x, b.y);
          const uint32_t f1[4] = {a[i][m][0].z, a[i][m][1].z, a[i][m][0].w, a[i][m][1].w};
          mma16816(acc[m][n], f1, b.z, b.w);
        }
      }
    }
  }
  store_partials<S, NOUT>(acc, m_tiles, red);
}

// sum over the slots that step_matmul leaves (after a __syncthreads)
template <typename S, int NOUT>
__device__ __forceinline__ float red_sum(const float* __restrict__ red, int row, int col) {
  constexpr int RP = NOUT + kRedPad;
  const float* q = red + row * RP + col;
  float v[S::Slots];
#pragma unroll
  for (int i = 0; i < S::Slots; ++i) v[i] = q[i * S::Rows * RP];
#pragma unroll
  for (int d = S::Slots / 2; d > 0; d >>= 1)
#pragma unroll
    for (int i = 0; i < d; ++i) v[i] += v[i + d];
  return v[0];
}

struct FwdArgs {
  const bf16* z_in;     // [T,B,4H]
  const bf16* w_rec;    // [4H,H]
  const int* lens;      // [B] or null
  const float *h0, *c0; // [B,H]
  int T, B, H, reverse;
  bf16* y;              // [T,B,H]
  float* c_all;         // [T,B,H]
  bf16* gates;          // [T,B,4H]
  bf16* hprev_all;      // [T,B,H]
  float *h_final, *c_final;
  bf16* hbuf;           // [2,B,H] exchange buffer of the hidden state (wide form: null, hprev_all is the exchanged matrix)
  uint32_t* flags;      // one word per CTA (or the counter), zeroed before the launch
  int* abort_word;      // zeroed before the launch
  int* status;          // receives (5 << 24) | cta when a barrier wait ran out
};

// The exchange of the wide forms has no barrier: the matrix of a step has a place of its own in memory (h_t in hprev_all, dz_t in dz, which the
// passes leave anyway), the launcher fills it with kUnwritten, and a warp that needs values loads them until none of them is that. One trip
// through L2 per step (store, load) takes the place of store, fence, flag, poll and load, a warp waits only for the CTAs whose units it
// multiplies, and only vectors that were not complete are loaded again. kUnwritten is a NaN that no conversion gives (theirs is 0x7fff); a value
// that has these bits all the same is published as another NaN.
constexpr uint32_t kUnwritten = 0xffffu;

__device__ __forceinline__ uint32_t publishable(float v) { return min((uint32_t)__bfloat16_as_ushort(__float2bfloat16(v)), kUnwritten - 1); }
__device__ __forceinline__ void publish_word(bf16* dst, uint32_t w) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(dst), "r"(w) : "memory");
}

// Wait until all values of the warp's blocks [b_begin, b_end) arrived; a[..] then holds them (zeros for rows and blocks that do not exist).
template <typename S, int kBlocks>
__device__ __forceinline__ bool fetch_published(const bf16* __restrict__ A, int n_rows, int K, int b_begin, int b_end, uint4 (&a)[kBlocks][S::MT][2],
                                                int* abort_word, int* status) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  static_assert(kBlocks * S::MT * 2 <= 32, "one bit per vector");
  uint32_t missing = 0u;
#pragma unroll
  for (int i = 0; i < kBlocks; ++i)
#pragma unroll
    for (int m = 0; m < S::MT; ++m)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        a[i][m][q] = make_uint4(0u, 0u, 0u, 0u);
        if (b_begin + i < b_end && m * 16 + q * 8 + g < n_rows) missing |= 1u << ((i * S::MT + m) * 2 + q);
      }
  const bf16* src = A + (size_t)g * K + (b_begin << 5) + 8 * t;
  uint32_t spins = 0;
  while (true) {
#pragma unroll
    for (int i = 0; i < kBlocks; ++i)
#pragma unroll
      for (int m = 0; m < S::MT; ++m)
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (missing >> ((i * S::MT + m) * 2 + q) & 1u) {
            uint4& v = a[i][m][q];
            asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                         : "l"(src + (size_t)(m * 16 + q * 8) * K + (i << 5)) : "memory");
          }
#pragma unroll
    for (int i = 0; i < kBlocks; ++i)
#pragma unroll
      for (int m = 0; m < S::MT; ++m)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4& v = a[i][m][q];
          const uint32_t top = max_u16x2(max_u16x2(v.x, v.y), max_u16x2(v.z, v.w));
          if ((top >> 16) != kUnwritten && (top & 0xffffu) != kUnwritten) missing &= ~(1u << ((i * S::MT + m) * 2 + q));
        }
    if (__all_sync(0xffffffffu, missing == 0u)) return true;
    ++spins;
    if (spins > kSpinLimit || ((spins & 255u) == 0 && *reinterpret_cast<volatile int*>(abort_word))) {
      if (lane == 0) {
        atomicExch(abort_word, 1);
        if (status) atomicCAS(status, 0, (5 << 24) | (int)(blockIdx.x & 0xFFFF));
      }
      return false;
    }
  }
}

// acc += A . Bs^T over the warp's blocks of a published matrix (see step_matmul for the order of k in a block); false: gave up waiting
template <typename S, int NOUT, int kPrefetch>
__device__ __forceinline__ bool published_matmul(const bf16* __restrict__ A, int n_rows, int K, const bf16* __restrict__ Bs, float (&acc)[S::MT][NOUT / 8][4],
                                                 int* abort_word, int* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int pitch = K + kPad;
#pragma unroll
  for (int m = 0; m < S::MT; ++m)
#pragma unroll
    for (int n = 0; n < NOUT / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
  const int m_tiles = (n_rows + 15) / 16;
  const int nblk = K >> 5;
  const int b_begin = warp * nblk / S::W, b_end = (warp + 1) * nblk / S::W;
  for (int bc = b_begin; bc < b_end; bc += kPrefetch) {
    uint4 a[kPrefetch][S::MT][2];
    if (!fetch_published<S, kPrefetch>(A, n_rows, K, bc, b_end, a, abort_word, status)) return false;
#pragma unroll
    for (int i = 0; i < kPrefetch; ++i) {
      if (bc + i >= b_end) break;
      const int k0 = (bc + i) << 5;
#pragma unroll
      for (int n = 0; n < NOUT / 8; ++n) {
        const uint4 w = *reinterpret_cast<const uint4*>(Bs + (size_t)(n * 8 + g) * pitch + k0 + 8 * t);
#pragma unroll
        for (int m = 0; m < S::MT; ++m) {
          if (m >= m_tiles) continue;
          const uint32_t f0[4] = {a[i][m][0].x, a[i][m][1].x, a[i][m][0].y, a[i][m][1].y};
          mma16816(acc[m][n], f0, w.x, w.y);
          const uint32_t f1[4] = {a[i][m][0].z, a[i][m][1].z, a[i][m][0].w, a[i][m][1].w};
          mma16816(acc[m][n], f1, w.z, w.w);
        }
      }
    }
  }
  return true;
}

template <typename S>
__device__ __forceinline__ void fwd_body_published(const FwdArgs& p, const int cta) {
  constexpr int U = S::U, kThreads = S::Threads, NOUT = 4 * U;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int H = p.H, B = p.B;
  const int pitch = H + kPad;
  bf16* Ws = reinterpret_cast<bf16*>(smem_raw);                      // [4*U][H+kPad]: row q*U+u = W_rec[q*H + j0 + u]
  float* red = reinterpret_cast<float*>(Ws + (size_t)NOUT * pitch);  // [slots][rows][4*U + kRedPad]
  const int j0 = cta * U;
  for (int idx = threadIdx.x; idx < NOUT * (H / 8); idx += kThreads) {
    const int r = idx / (H / 8), v = idx % (H / 8);
    const int q = r / U, u = r % U;
    *reinterpret_cast<uint4*>(Ws + (size_t)r * pitch + v * 8) = *reinterpret_cast<const uint4*>(p.w_rec + ((size_t)q * H + j0 + u) * H + v * 8);
  }
  static_assert(S::PerThread == 1 && U % 2 == 0, "one (row, unit) pair per thread, the units of a word in neighbouring lanes");
  const int b = threadIdx.x / U, u = threadIdx.x % U;
  const bool own = b < B;
  float cst = 0.f, hst = 0.f;
  bf16 zin[4];
  const int len = own && p.lens ? p.lens[b] : p.T;
  auto publish = [&](int t, float h) {  // (all lanes of the warp) h, the state before frame t
    const uint32_t v = publishable(h);
    const uint32_t next = __shfl_down_sync(0xffffffffu, v, 1);
    if (own && (u & 1) == 0) publish_word(p.hprev_all + ((size_t)t * B + b) * H + j0 + u, v | next << 16);
  };
  auto fetch_zin = [&](int t) {
    if (!own) return;
    const bf16* z = p.z_in + ((size_t)t * B + b) * 4 * H + j0 + u;
#pragma unroll
    for (int q = 0; q < 4; ++q) zin[q] = z[(size_t)q * H];
  };
  if (own) {
    hst = __bfloat162float(__float2bfloat16(p.h0[(size_t)b * H + j0 + u]));
    cst = p.c0[(size_t)b * H + j0 + u];
  }
  if (p.T > 0) {
    publish(p.reverse ? p.T - 1 : 0, hst);
    fetch_zin(p.reverse ? p.T - 1 : 0);
  }
  __syncthreads();  // the resident slice is in place
  const int m_tiles = (B + 15) / 16;
  for (int s = 0; s < p.T; ++s) {
    const int t = p.reverse ? p.T - 1 - s : s, t_next = p.reverse ? t - 1 : t + 1;
    float acc[S::MT][NOUT / 8][4];
    const bool ok = published_matmul<S, NOUT, S::PrefetchFwd>(p.hprev_all + (size_t)t * B * H, B, H, Ws, acc, p.abort_word, p.status);
    store_partials<S, NOUT>(acc, m_tiles, red);
    if (!__syncthreads_and(ok ? 1 : 0)) break;
    float gi = 0.f, gf = 0.f, gg = 0.f, go = 0.f;
    if (own && t < len) {
      gi = sigm(red_sum<S, NOUT>(red, b, u) + __bfloat162float(zin[0]));
      gf = sigm(red_sum<S, NOUT>(red, b, U + u) + __bfloat162float(zin[1]));
      gg = tanhf(red_sum<S, NOUT>(red, b, 2 * U + u) + __bfloat162float(zin[2]));
      go = sigm(red_sum<S, NOUT>(red, b, 3 * U + u) + __bfloat162float(zin[3]));
      cst = gf * cst + gi * gg;
      hst = __bfloat162float(__float2bfloat16(go * tanhf(cst)));
    }
    if (s + 1 < p.T) {
      publish(t_next, hst);
      fetch_zin(t_next);
    }
    if (own) {
      const size_t o = ((size_t)t * B + b) * H + j0 + u;
      const size_t zo = ((size_t)t * B + b) * 4 * H + j0 + u;
      p.y[o] = __float2bfloat16(t < len ? hst : 0.f);
      p.c_all[o] = cst;
      p.gates[zo] = __float2bfloat16(gi);
      p.gates[zo + H] = __float2bfloat16(gf);
      p.gates[zo + 2 * (size_t)H] = __float2bfloat16(gg);
      p.gates[zo + 3 * (size_t)H] = __float2bfloat16(go);
    }
    __syncthreads();  // the partial sums have been read
  }
  if (own) {
    p.h_final[(size_t)b * H + j0 + u] = hst;
    p.c_final[(size_t)b * H + j0 + u] = cst;
  }
}

template <typename S>
__device__ __forceinline__ void fwd_body(const FwdArgs& p, const int cta, const int n_cta) {
  constexpr int U = S::U, kThreads = S::Threads, NOUT = 4 * U;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int H = p.H, B = p.B;
  const int pitch = H + kPad;
  bf16* Ws = reinterpret_cast<bf16*>(smem_raw);                           // [4*U][H+kPad]: row q*U+u = W_rec[q*H + j0 + u]
  float* red = reinterpret_cast<float*>(Ws + (size_t)NOUT * pitch);       // [slots][rows][4*U + kRedPad]
  const int j0 = cta * U;
  // resident slice: 4*U rows of H elements, 16-byte copies
  for (int idx = threadIdx.x; idx < NOUT * (H / 8); idx += kThreads) {
    const int r = idx / (H / 8), v = idx % (H / 8);
    const int q = r / U, u = r % U;
    *reinterpret_cast<uint4*>(Ws + (size_t)r * pitch + v * 8) = *reinterpret_cast<const uint4*>(p.w_rec + ((size_t)q * H + j0 + u) * H + v * 8);
  }
  // every thread owns up to PerThread (row, unit) pairs: their state stays in registers, and their input projections z_in[t] are fetched
  // one step ahead (they come from DRAM) so that the cell does not wait for them after the barrier
  constexpr int N = S::PerThread;
  float cst[N], hst[N];
  bf16 zin[N][4];  // as loaded: a conversion next to the load would wait for it
  int len[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    const int b = idx / U, u = idx % U;
    cst[i] = hst[i] = 0.f;
    len[i] = p.T;
    if (idx < B * U) {
      const float h = p.h0[(size_t)b * H + j0 + u];
      const bf16 hb = __float2bfloat16(h);
      cst[i] = p.c0[(size_t)b * H + j0 + u];
      hst[i] = __bfloat162float(hb);
      if (p.lens) len[i] = p.lens[b];
      p.hbuf[(size_t)b * H + j0 + u] = hb;
    }
  }
  auto fetch_zin = [&](int t) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx < B * U) {
        const int b = idx / U, u = idx % U;
        const bf16* z = p.z_in + ((size_t)t * B + b) * 4 * H + j0 + u;
#pragma unroll
        for (int q = 0; q < 4; ++q) zin[i][q] = z[(size_t)q * H];
      }
    }
  };
  uint32_t n_bar = 1;
  barrier_arrive<S>(p.flags, cta, n_cta, n_bar);
  if (p.T > 0) fetch_zin(p.reverse ? p.T - 1 : 0);
  bool ok = barrier_wait<S>(p.flags, n_cta, n_bar, p.abort_word, p.status);
  for (int s = 0; s < p.T && ok; ++s) {
    const int t = p.reverse ? p.T - 1 - s : s;
    const bf16* h_cur = p.hbuf + (size_t)(s & 1) * B * H;
    bf16* h_nxt = p.hbuf + (size_t)((s + 1) & 1) * B * H;
    step_matmul<S, NOUT, S::PrefetchFwd>(h_cur, B, H, Ws, red);
    __syncthreads();
    float gates[N][4], hp[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx >= B * U) continue;
      const int b = idx / U, u = idx % U;
      hp[i] = hst[i];
      gates[i][0] = gates[i][1] = gates[i][2] = gates[i][3] = 0.f;
      if (t < len[i]) {
        const float gi = sigm(red_sum<S, NOUT>(red, b, u) + __bfloat162float(zin[i][0]));
        const float gf = sigm(red_sum<S, NOUT>(red, b, U + u) + __bfloat162float(zin[i][1]));
        const float gg = tanhf(red_sum<S, NOUT>(red, b, 2 * U + u) + __bfloat162float(zin[i][2]));
        const float go = sigm(red_sum<S, NOUT>(red, b, 3 * U + u) + __bfloat162float(zin[i][3]));
        const float c = gf * cst[i] + gi * gg;
        cst[i] = c;
        hst[i] = __bfloat162float(__float2bfloat16(go * tanhf(c)));
        gates[i][0] = gi; gates[i][1] = gf; gates[i][2] = gg; gates[i][3] = go;
      }
      h_nxt[(size_t)b * H + j0 + u] = __float2bfloat16(hst[i]);
    }
    barrier_arrive<S>(p.flags, cta, n_cta, ++n_bar);
    if (s + 1 < p.T) fetch_zin(p.reverse ? p.T - 2 - s : s + 1);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx >= B * U) continue;
      const int b = idx / U, u = idx % U;
      const size_t o = ((size_t)t * B + b) * H + j0 + u;
      const size_t zo = ((size_t)t * B + b) * 4 * H + j0 + u;
      p.hprev_all[o] = __float2bfloat16(hp[i]);
      p.y[o] = __float2bfloat16(t < len[i] ? hst[i] : 0.f);
      p.c_all[o] = cst[i];
#pragma unroll
      for (int q = 0; q < 4; ++q) p.gates[zo + (size_t)q * H] = __float2bfloat16(gates[i][q]);
    }
    ok = barrier_wait<S>(p.flags, n_cta, n_bar, p.abort_word, p.status);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    if (idx >= B * U) continue;
    const size_t o = (size_t)(idx / U) * H + j0 + idx % U;
    p.h_final[o] = hst[i];
    p.c_final[o] = cst[i];
  }
}

__global__ void __launch_bounds__(Narrow::Threads, 1) lstm_persist_fwd_kernel(FwdArgs p) { fwd_body<Narrow>(p, blockIdx.x, gridDim.x); }

// Both directions of a bidirectional layer in one launch: the first half of the grid runs d[0], the second half d[1], each with its own
// flags: two recurrences, each bound by the latency of its barrier and L2 round trips per step, overlap instead of running one after the
// other. Narrow: two CTAs per SM (128 registers per thread); wide: one.
struct FwdPair {
  FwdArgs d[2];
};

template <typename S>
__global__ void __launch_bounds__(S::Threads, S::U == 8 ? 2 : 1) lstm_persist_fwd_pair_kernel(const __grid_constant__ FwdPair pp) {
  const int half = gridDim.x / 2;
  if constexpr (S::U == 16) {
    if ((int)blockIdx.x < half) fwd_body_published<S>(pp.d[0], blockIdx.x);
    else fwd_body_published<S>(pp.d[1], blockIdx.x - half);
  } else {
    if ((int)blockIdx.x < half) fwd_body<S>(pp.d[0], blockIdx.x, half);
    else fwd_body<S>(pp.d[1], blockIdx.x - half, half);
  }
}

struct BwdArgs {
  const bf16* dy;        // [T,B,H] or null
  const float *dh_final, *dc_final;  // [B,H] or null
  const bf16* w_rec;     // [4H,H]
  const int* lens;
  const bf16* gates;     // [T,B,4H]
  const float *c_all, *c0;
  int T, B, H, reverse;
  bf16* dz;              // [T,B,4H]: output and per-step exchange buffer
  float *dh0, *dc0;      // [B,H] outputs
  uint32_t* flags;
  int* abort_word;
  int* status;
};

// the columns of W_rec that a CTA's units feed: Wt[u][n] = W_rec[n][j0 + u], in 16-byte pieces
template <typename S>
__device__ __forceinline__ void load_transposed(const bf16* __restrict__ w_rec, int K, int H, int j0, bf16* __restrict__ Wt) {
  constexpr int U = S::U;
  for (int idx = threadIdx.x; idx < K * (U / 8); idx += S::Threads) {
    const int n = idx / (U / 8), piece = idx % (U / 8);
    const uint4 v = *reinterpret_cast<const uint4*>(w_rec + (size_t)n * H + j0 + piece * 8);
    const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
    for (int i = 0; i < 8; ++i) Wt[(size_t)(piece * 8 + i) * (K + kPad) + n] = e[i];
  }
}

template <typename S>
__device__ __forceinline__ void bwd_body(const BwdArgs& p, const int cta, const int n_cta) {
  constexpr int U = S::U, kThreads = S::Threads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int H = p.H, B = p.B, K = 4 * p.H;
  const int pitch = K + kPad;
  bf16* Wt = reinterpret_cast<bf16*>(smem_raw);                    // [U][4H+kPad]: Wt[u][n] = W_rec[n][j0+u]
  float* red = reinterpret_cast<float*>(Wt + (size_t)U * pitch);   // [slots][rows][U + kRedPad]
  const int j0 = cta * U;
  load_transposed<S>(p.w_rec, K, H, j0, Wt);
  // a thread's (row, unit) pairs: gradients arriving at h_t and c_t, and what the forward pass kept, fetched one step ahead (DRAM)
  constexpr int N = S::PerThread;
  float dhs[N], dcs[N], c_t[N], c_p[N];
  bf16 kept[N][4], dy[N];  // as loaded: a conversion next to the load would wait for it
  int len[N];
  auto fetch = [&](int s) {  // gates, dy and the cell state before step s; (the state after it is that of the step after)
    const int t = p.reverse ? p.T - 1 - s : s;
    const int t_prev = p.reverse ? t + 1 : t - 1;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx >= B * U) continue;
      const int b = idx / U, u = idx % U;
      const bf16* gt = p.gates + ((size_t)t * B + b) * K + j0 + u;
#pragma unroll
      for (int q = 0; q < 4; ++q) kept[i][q] = gt[(size_t)q * H];
      dy[i] = p.dy ? p.dy[((size_t)t * B + b) * H + j0 + u] : __float2bfloat16(0.f);
      c_p[i] = s > 0 ? p.c_all[((size_t)t_prev * B + b) * H + j0 + u] : p.c0[(size_t)b * H + j0 + u];
    }
  };
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    dhs[i] = dcs[i] = c_t[i] = 0.f;
    len[i] = p.T;
    if (idx >= B * U) continue;
    const int b = idx / U, u = idx % U;
    if (p.dh_final) dhs[i] = p.dh_final[(size_t)b * H + j0 + u];
    if (p.dc_final) dcs[i] = p.dc_final[(size_t)b * H + j0 + u];
    if (p.lens) len[i] = p.lens[b];
    if (p.T > 0) c_t[i] = p.c_all[((size_t)(p.reverse ? 0 : p.T - 1) * B + b) * H + j0 + u];
  }
  if (p.T > 0) fetch(p.T - 1);
  __syncthreads();
  uint32_t n_bar = 0;
  bool ok = true;
  for (int s = p.T - 1; s >= 0 && ok; --s) {
    const int t = p.reverse ? p.T - 1 - s : s;
    bf16* dz_t = p.dz + (size_t)t * B * K;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx >= B * U) continue;
      const size_t zo = (size_t)(idx / U) * K + j0 + idx % U;
      if (t >= len[i]) {
        dz_t[zo] = dz_t[zo + H] = dz_t[zo + 2 * H] = dz_t[zo + 3 * H] = __float2bfloat16(0.f);
        continue;  // state was carried: dh and dc pass through
      }
      const float dh = dhs[i] + __bfloat162float(dy[i]);
      const float gi = __bfloat162float(kept[i][0]), gf = __bfloat162float(kept[i][1]), gg = __bfloat162float(kept[i][2]),
                  go = __bfloat162float(kept[i][3]);
      const float tc = tanhf(c_t[i]);
      const float dc = dcs[i] + dh * go * (1.f - tc * tc);
      dz_t[zo] = __float2bfloat16(dc * gg * gi * (1.f - gi));
      dz_t[zo + H] = __float2bfloat16(dc * c_p[i] * gf * (1.f - gf));
      dz_t[zo + 2 * H] = __float2bfloat16(dc * gi * (1.f - gg * gg));
      dz_t[zo + 3 * H] = __float2bfloat16(dh * tc * go * (1.f - go));
      dcs[i] = dc * gf;
      dhs[i] = 0.f;
    }
    barrier_arrive<S>(p.flags, cta, n_cta, ++n_bar);
#pragma unroll
    for (int i = 0; i < N; ++i) c_t[i] = c_p[i];
    if (s > 0) fetch(s - 1);
    ok = barrier_wait<S>(p.flags, n_cta, n_bar, p.abort_word, p.status);  // all slices of dz_t are written
    if (!ok) break;
    step_matmul<S, U, S::PrefetchBwd>(dz_t, B, K, Wt, red);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = threadIdx.x + i * kThreads;
      if (idx < B * U) dhs[i] += red_sum<S, U>(red, idx / U, idx % U);
    }
    // (the slots are written again after the next barrier only)
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int idx = threadIdx.x + i * kThreads;
    if (idx >= B * U) continue;
    const size_t o = (size_t)(idx / U) * H + j0 + idx % U;
    p.dh0[o] = dhs[i];
    p.dc0[o] = dcs[i];
  }
}

__global__ void __launch_bounds__(Narrow::Threads, 1) lstm_persist_bwd_kernel(BwdArgs p) { bwd_body<Narrow>(p, blockIdx.x, gridDim.x); }

// wide form: dz itself is the exchanged matrix, see fetch_published
template <typename S>
__device__ __forceinline__ void bwd_body_published(const BwdArgs& p, const int cta) {
  constexpr int U = S::U, kThreads = S::Threads;
  static_assert(S::PerThread == 1 && U % 2 == 0, "one (row, unit) pair per thread, the units of a word in neighbouring lanes");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int H = p.H, B = p.B, K = 4 * p.H;
  bf16* Wt = reinterpret_cast<bf16*>(smem_raw);                          // [U][4H+kPad]: Wt[u][n] = W_rec[n][j0+u]
  float* red = reinterpret_cast<float*>(Wt + (size_t)U * (K + kPad));    // [slots][rows][U + kRedPad]
  const int j0 = cta * U;
  load_transposed<S>(p.w_rec, K, H, j0, Wt);
  const int b = threadIdx.x / U, u = threadIdx.x % U;
  const bool own = b < B;
  // gradients arriving at h_t and c_t, and what the forward pass kept, fetched one step ahead (DRAM)
  float dhs = 0.f, dcs = 0.f, c_t = 0.f, c_p = 0.f;
  bf16 kept[4], dy = __float2bfloat16(0.f);  // as loaded: a conversion next to the load would wait for it
  const int len = own && p.lens ? p.lens[b] : p.T;
  auto fetch = [&](int s) {  // gates, dy and the cell state before step s; (the state after it is that of the step after)
    if (!own) return;
    const int t = p.reverse ? p.T - 1 - s : s;
    const int t_prev = p.reverse ? t + 1 : t - 1;
    const bf16* gt = p.gates + ((size_t)t * B + b) * K + j0 + u;
#pragma unroll
    for (int q = 0; q < 4; ++q) kept[q] = gt[(size_t)q * H];
    if (p.dy) dy = p.dy[((size_t)t * B + b) * H + j0 + u];
    c_p = s > 0 ? p.c_all[((size_t)t_prev * B + b) * H + j0 + u] : p.c0[(size_t)b * H + j0 + u];
  };
  if (own) {
    if (p.dh_final) dhs = p.dh_final[(size_t)b * H + j0 + u];
    if (p.dc_final) dcs = p.dc_final[(size_t)b * H + j0 + u];
    if (p.T > 0) c_t = p.c_all[((size_t)(p.reverse ? 0 : p.T - 1) * B + b) * H + j0 + u];
  }
  if (p.T > 0) fetch(p.T - 1);
  __syncthreads();  // the resident slice is in place
  const int m_tiles = (B + 15) / 16;
  for (int s = p.T - 1; s >= 0; --s) {
    const int t = p.reverse ? p.T - 1 - s : s;
    bf16* dz_t = p.dz + (size_t)t * B * K;
    uint32_t ifg = 0u, gog = 0u;  // (i, f) and (g, o) of this unit
    if (own && t < len) {  // else the state was carried: dh and dc pass through
      const float dh = dhs + __bfloat162float(dy);
      const float gi = __bfloat162float(kept[0]), gf = __bfloat162float(kept[1]), gg = __bfloat162float(kept[2]), go = __bfloat162float(kept[3]);
      const float tc = tanhf(c_t);
      const float dc = dcs + dh * go * (1.f - tc * tc);
      ifg = publishable(dc * gg * gi * (1.f - gi)) | publishable(dc * c_p * gf * (1.f - gf)) << 16;
      gog = publishable(dc * gi * (1.f - gg * gg)) | publishable(dh * tc * go * (1.f - go)) << 16;
      dcs = dc * gf;
      dhs = 0.f;
    }
    // a word holds two units of one gate: the lane of the even unit stores gates i and f of both, that of the odd one g and o
    const uint32_t other = __shfl_xor_sync(0xffffffffu, (u & 1) ? ifg : gog, 1);
    if (own) {
      bf16* dst = dz_t + (size_t)b * K + j0 + (u & ~1) + ((u & 1) ? 2 * H : 0);
      const uint32_t lo = (u & 1) ? other : ifg, hi = (u & 1) ? gog : other;
      publish_word(dst, __byte_perm(lo, hi, 0x5410));
      publish_word(dst + H, __byte_perm(lo, hi, 0x7632));
    }
    c_t = c_p;
    if (s > 0) fetch(s - 1);
    float acc[S::MT][U / 8][4];
    const bool ok = published_matmul<S, U, S::PrefetchBwd>(dz_t, B, K, Wt, acc, p.abort_word, p.status);
    store_partials<S, U>(acc, m_tiles, red);
    if (!__syncthreads_and(ok ? 1 : 0)) break;
    if (own) dhs += red_sum<S, U>(red, b, u);
    __syncthreads();  // the partial sums have been read
  }
  if (own) {
    p.dh0[(size_t)b * H + j0 + u] = dhs;
    p.dc0[(size_t)b * H + j0 + u] = dcs;
  }
}

struct BwdPair {
  BwdArgs d[2];
};

template <typename S>
__global__ void __launch_bounds__(S::Threads, S::U == 8 ? 2 : 1) lstm_persist_bwd_pair_kernel(const __grid_constant__ BwdPair pp) {
  const int half = gridDim.x / 2;
  if constexpr (S::U == 16) {
    if ((int)blockIdx.x < half) bwd_body_published<S>(pp.d[0], blockIdx.x);
    else bwd_body_published<S>(pp.d[1], blockIdx.x - half);
  } else {
    if ((int)blockIdx.x < half) bwd_body<S>(pp.d[0], blockIdx.x, half);
    else bwd_body<S>(pp.d[1], blockIdx.x - half, half);
  }
}

// barrier words of the calls in flight: 64 slots of (abort word, flags), handed out round robin
constexpr int kSyncSlots = 64;
constexpr int kSyncWords = 32 + kMaxCtas;  // the flags start on a line of their own
static __device__ __align__(128) unsigned int g_lstm_sync[kSyncSlots * kSyncWords];

unsigned int* sync_slot() {
  static unsigned int* base[64] = {nullptr};
  static unsigned next = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (!base[dev]) {
    unsigned int* ptr = nullptr;
    if (cudaGetSymbolAddress((void**)&ptr, g_lstm_sync) != cudaSuccess) return nullptr;
    base[dev] = ptr;
  }
  return base[dev] + kSyncWords * (next++ % kSyncSlots);
}

template <typename S>
size_t fwd_smem(int H) {
  return (size_t)4 * S::U * (H + kPad) * sizeof(bf16) + (size_t)S::Slots * S::Rows * (4 * S::U + kRedPad) * sizeof(float);
}
template <typename S>
size_t bwd_smem(int H) {
  return (size_t)S::U * (4 * H + kPad) * sizeof(bf16) + (size_t)S::Slots * S::Rows * (S::U + kRedPad) * sizeof(float);
}

bool enabled() {
  static const bool on = [] {
    const char* v = getenv("RETURNN_B200_LSTM_PERSIST");
    return !(v && v[0] == '0');
  }();
  return on;
}

}  // namespace

// whether the persistent kernels take this problem (else the per-step executor runs)
bool rb_lstm_persist_supported(int T, int B, int H) {
  if (!enabled() || T <= 0 || B <= 0 || B > kMaxRows || H % 128 || H / Narrow::U > 148) return false;
  return fwd_smem<Narrow>(H) <= 220 * 1024 && bwd_smem<Narrow>(H) <= 220 * 1024;
}

// scratch: hbuf 2*B*H bf16 provided by the caller, contents arbitrary
int rb_lstm_persist_fwd(const void* z_in, const void* w_rec, const int* lens, const float* h0, const float* c0, int T, int B, int H, int reverse,
                        void* y, float* c_all, void* gates, void* hprev_all, float* h_final, float* c_final, void* hbuf, int* status,
                        cudaStream_t stream) {
  unsigned int* sync_words = sync_slot();
  if (!sync_words) {
    rb_set_error("lstm_persist_fwd: no barrier words");
    return RB_ERR_LAUNCH;
  }
  FwdArgs a;
  a.z_in = (const bf16*)z_in; a.w_rec = (const bf16*)w_rec; a.lens = lens; a.h0 = h0; a.c0 = c0;
  a.T = T; a.B = B; a.H = H; a.reverse = reverse;
  a.y = (bf16*)y; a.c_all = c_all; a.gates = (bf16*)gates; a.hprev_all = (bf16*)hprev_all; a.h_final = h_final; a.c_final = c_final;
  a.hbuf = (bf16*)hbuf; a.flags = sync_words + 32; a.abort_word = reinterpret_cast<int*>(sync_words); a.status = status;
  cudaMemsetAsync(sync_words, 0, kSyncWords * sizeof(unsigned int), stream);
  const size_t smem = fwd_smem<Narrow>(H);
  cudaError_t e = cudaFuncSetAttribute(lstm_persist_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  void* args[] = {&a};
  if (e == cudaSuccess) e = cudaLaunchCooperativeKernel((const void*)lstm_persist_fwd_kernel, dim3(H / Narrow::U), dim3(Narrow::Threads), args, smem, stream);
  if (e != cudaSuccess) {
    rb_set_error("lstm_persist_fwd: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return RB_ERR_LAUNCH;
  }
  return RB_OK;
}

int rb_lstm_persist_bwd(const void* dy, const float* dh_final, const float* dc_final, const void* w_rec, const int* lens, const void* gates,
                        const float* c_all, const float* c0, int T, int B, int H, int reverse, void* dz, float* dh0, float* dc0, int* status,
                        cudaStream_t stream) {
  unsigned int* sync_words = sync_slot();
  if (!sync_words) {
    rb_set_error("lstm_persist_bwd: no barrier words");
    return RB_ERR_LAUNCH;
  }
  BwdArgs a;
  a.dy = (const bf16*)dy; a.dh_final = dh_final; a.dc_final = dc_final; a.w_rec = (const bf16*)w_rec; a.lens = lens; a.gates = (const bf16*)gates;
  a.c_all = c_all; a.c0 = c0; a.T = T; a.B = B; a.H = H; a.reverse = reverse; a.dz = (bf16*)dz; a.dh0 = dh0; a.dc0 = dc0;
  a.flags = sync_words + 32; a.abort_word = reinterpret_cast<int*>(sync_words); a.status = status;
  cudaMemsetAsync(sync_words, 0, kSyncWords * sizeof(unsigned int), stream);
  const size_t smem = bwd_smem<Narrow>(H);
  cudaError_t e = cudaFuncSetAttribute(lstm_persist_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  void* args[] = {&a};
  if (e == cudaSuccess) e = cudaLaunchCooperativeKernel((const void*)lstm_persist_bwd_kernel, dim3(H / Narrow::U), dim3(Narrow::Threads), args, smem, stream);
  if (e != cudaSuccess) {
    rb_set_error("lstm_persist_bwd: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return RB_ERR_LAUNCH;
  }
  return RB_OK;
}

// ---- both directions of a bidirectional layer in one cooperative launch -------------------------------------------------

namespace {

// whether both grids of a pair of kernels of this shape are co-resident on the current device; raises their shared-memory limits
template <typename S>
bool pair_fits(int H) {
  static thread_local int last_dev = -1, last_h = 0;
  static thread_local bool last_ok = false;
  const size_t sf = fwd_smem<S>(H), sb = bwd_smem<S>(H);
  constexpr int kLimit = 220 * 1024;
  int dev = 0, sm_count = 0, of = 0, ob = 0;
  if (sf > kLimit || sb > kLimit || H % S::U || H / S::U > kMaxCtas || cudaGetDevice(&dev) != cudaSuccess) return false;
  if (dev == last_dev && H == last_h) return last_ok;
  bool ok = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
            cudaFuncSetAttribute(lstm_persist_fwd_pair_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLimit) == cudaSuccess &&
            cudaFuncSetAttribute(lstm_persist_bwd_pair_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLimit) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&of, lstm_persist_fwd_pair_kernel<S>, S::Threads, sf) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ob, lstm_persist_bwd_pair_kernel<S>, S::Threads, sb) == cudaSuccess;
  if (!ok) cudaGetLastError();
  ok = ok && of * sm_count >= 2 * (H / S::U) && ob * sm_count >= 2 * (H / S::U);
  last_dev = dev;
  last_h = H;
  last_ok = ok;
  return ok;
}

enum { kNoPair = 0, kNarrow = 1, kWide1 = 2, kWide2 = 3 };

// The shape that runs a bidirectional layer. Training, T = 100, wide / narrow, us (at H = 1024 the narrow form is timed with the counter of 33
// rows): H = 1024: 1 row 1130 / 2150, 16: 1360 / 2410, 17: 1800 / 2490, 32: 2110 / 2705; H = 512: 850 / 1114, 930 / 1250, 1170 / 1293,
// 1355 / 1420. At H <= 256 the forms are within 7 % of each other with 17 to 32 rows (256, 32 rows: 1155 / 1100), and the wide one is ahead below.
int pair_shape(int T, int B, int H) {
  if (!rb_lstm_persist_supported(T, B, H)) return kNoPair;
  if (B <= 16 && pair_fits<Wide1>(H)) return kWide1;
  if (B <= 32 && pair_fits<Wide2>(H)) return kWide2;
  return pair_fits<NarrowPair>(H) ? kNarrow : kNoPair;
}

template <typename S>
cudaError_t launch_fwd_pair(FwdPair& pp, int H, cudaStream_t stream) {
  void* args[] = {&pp};
  return cudaLaunchCooperativeKernel((const void*)lstm_persist_fwd_pair_kernel<S>, dim3(2 * (H / S::U)), dim3(S::Threads), args, fwd_smem<S>(H), stream);
}
template <typename S>
cudaError_t launch_bwd_pair(BwdPair& pp, int H, cudaStream_t stream) {
  void* args[] = {&pp};
  return cudaLaunchCooperativeKernel((const void*)lstm_persist_bwd_pair_kernel<S>, dim3(2 * (H / S::U)), dim3(S::Threads), args, bwd_smem<S>(H), stream);
}

}  // namespace

// whether the two-direction kernels take this problem: the single-direction conditions, and both grids co-resident
// 0: not supported; 1: the narrow form, which takes an exchange buffer; more: a wide form, which takes none
RB_EXPORT int rb200_blstm_supported(int T, int B, int H) { return pair_shape(T, B, H); }

// ptrs[d * 11 + i] for direction d (0: forward in time, 1: reversed):
//   0 z_in [T,B,4H] bf16, 1 w_rec [4H,H] bf16, 2 h0, 3 c0 [B,H] fp32, 4 y [T,B,H] bf16, 5 c_all [T,B,H] fp32, 6 gates [T,B,4H] bf16,
//   7 hprev_all [T,B,H] bf16, 8 h_final, 9 c_final [B,H] fp32, 10 exchange buffer (narrow form: scratch, 2*B*H bf16)
RB_EXPORT int rb200_blstm_fwd(void* const* ptrs, const int* lens, int T, int B, int H, int* status, cudaStream_t stream) {
  if (T <= 0 || B <= 0) return RB_OK;
  const int shape = pair_shape(T, B, H);
  if (shape == kNoPair) {
    rb_set_error("blstm_fwd: shape T=%d B=%d H=%d is not supported by the two-direction kernel", T, B, H);
    return RB_ERR_UNSUPPORTED;
  }
  FwdPair pp;
  for (int d = 0; d < 2; ++d) {
    unsigned int* sync_words = sync_slot();
    if (!sync_words) {
      rb_set_error("blstm_fwd: no barrier words");
      return RB_ERR_LAUNCH;
    }
    void* const* q = ptrs + d * 11;
    FwdArgs& a = pp.d[d];
    a.z_in = (const bf16*)q[0]; a.w_rec = (const bf16*)q[1]; a.lens = lens; a.h0 = (const float*)q[2]; a.c0 = (const float*)q[3];
    a.T = T; a.B = B; a.H = H; a.reverse = d;
    a.y = (bf16*)q[4]; a.c_all = (float*)q[5]; a.gates = (bf16*)q[6]; a.hprev_all = (bf16*)q[7]; a.h_final = (float*)q[8]; a.c_final = (float*)q[9];
    a.hbuf = (bf16*)q[10];
    if (shape != kNarrow) cudaMemsetAsync(a.hprev_all, 0xff, (size_t)T * B * H * sizeof(bf16), stream);  // kUnwritten
    a.flags = sync_words + 32; a.abort_word = reinterpret_cast<int*>(sync_words); a.status = status;
    cudaMemsetAsync(sync_words, 0, kSyncWords * sizeof(unsigned int), stream);
  }
  const cudaError_t e = shape == kWide1   ? launch_fwd_pair<Wide1>(pp, H, stream)
                        : shape == kWide2 ? launch_fwd_pair<Wide2>(pp, H, stream)
                                          : launch_fwd_pair<NarrowPair>(pp, H, stream);
  if (e != cudaSuccess) {
    rb_set_error("blstm_fwd: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return RB_ERR_LAUNCH;
  }
  return RB_OK;
}

// ptrs[d * 12 + i]: 0 dy [T,B,H] bf16 or null, 1 dh_final, 2 dc_final [B,H] fp32 or null, 3 w_rec bf16, 4 gates, 5 c_all, 6 c0, 7 hprev_all,
//   8 dz [T,B,4H] bf16 (out), 9 dw_rec [4H,H] fp32 (accumulated into; may be null), 10 dh0, 11 dc0 [B,H] fp32 (out)
RB_EXPORT int rb200_blstm_bwd(void* const* ptrs, const int* lens, int T, int B, int H, int* status, int* n_launch, cudaStream_t stream) {
  if (T <= 0 || B <= 0) return RB_OK;
  const int shape = pair_shape(T, B, H);
  if (shape == kNoPair) {
    rb_set_error("blstm_bwd: shape T=%d B=%d H=%d is not supported by the two-direction kernel", T, B, H);
    return RB_ERR_UNSUPPORTED;
  }
  BwdPair pp;
  for (int d = 0; d < 2; ++d) {
    unsigned int* sync_words = sync_slot();
    if (!sync_words) {
      rb_set_error("blstm_bwd: no barrier words");
      return RB_ERR_LAUNCH;
    }
    void* const* q = ptrs + d * 12;
    BwdArgs& a = pp.d[d];
    a.dy = (const bf16*)q[0]; a.dh_final = (const float*)q[1]; a.dc_final = (const float*)q[2]; a.w_rec = (const bf16*)q[3]; a.lens = lens;
    a.gates = (const bf16*)q[4]; a.c_all = (const float*)q[5]; a.c0 = (const float*)q[6]; a.T = T; a.B = B; a.H = H; a.reverse = d;
    a.dz = (bf16*)q[8]; a.dh0 = (float*)q[10]; a.dc0 = (float*)q[11];
    if (shape != kNarrow) cudaMemsetAsync(a.dz, 0xff, (size_t)T * B * 4 * H * sizeof(bf16), stream);  // kUnwritten
    a.flags = sync_words + 32; a.abort_word = reinterpret_cast<int*>(sync_words); a.status = status;
    cudaMemsetAsync(sync_words, 0, kSyncWords * sizeof(unsigned int), stream);
  }
  const cudaError_t e = shape == kWide1   ? launch_bwd_pair<Wide1>(pp, H, stream)
                        : shape == kWide2 ? launch_bwd_pair<Wide2>(pp, H, stream)
                                          : launch_bwd_pair<NarrowPair>(pp, H, stream);
  if (e != cudaSuccess) {
    rb_set_error("blstm_bwd: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return RB_ERR_LAUNCH;
  }
  int launches = 3;
  for (int d = 0; d < 2; ++d) {
    void* const* q = ptrs + d * 12;
    if (!q[9]) continue;
    // dW_rec[4H,H] += dz^T [4H, T*B] . h_prev [T*B, H]
    RbGemm g;
    g.a = q[8]; g.b = q[7]; g.c = q[9]; g.m = 4 * H; g.n = H; g.k = T * B; g.lda = 4 * H; g.ldb = H; g.ldc = H;
    g.a_mn_major = 1; g.b_mn_major = 1; g.out_fp32 = 1; g.accumulate = 2; g.status = status;
    int st = rb_gemm(g, stream);
    if (st) return st;
    ++launches;
  }
  if (n_launch) *n_launch = launches;
  return rb_check_launch("blstm_bwd");
}

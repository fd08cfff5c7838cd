// Persistent bf16 GEMM on the 5th-generation tensor cores (sm_100a) with a fused epilogue.
//
//   D[M,N] = epilogue(alpha * op(A)·op(B)),   fp32 accumulation in tensor memory
//
// One CTA per SM (two for batches of small problems, see Layout) walks a list of work units (128 x BN output tile, BN = 256, 128 or 64, optionally one
// slice of K):
//   warp 0   TMA producer: cp.async.bulk.tensor (128-byte swizzle, no cluster multicast) into a shared-memory ring that keeps
//            running across units, so the loads of the next tile are in flight while the current one is still multiplied
//   warp 1   MMA issuer: one lane issues tcgen05.mma (cta_group::1, kind::f16, 128 x BN x 16); tcgen05.commit frees the ring
//            stage and, after the last K block, publishes the accumulator. In both warps the whole warp walks and waits, and an elected lane of it
//            issues, so that addresses, descriptors and coordinates stay in uniform registers: the batched products of attention, with one to
//            eight K blocks a tile, are bound by this walk (dV of 36 x 333 frames, 8 heads: 20.1 -> 16.8 us, position gradient 29.4 -> 24.7,
//            20 x 500 frames 21.6 -> 17.8 and 29.5 -> 24.9)
//   the rest epilogue, 16 warps (8 where two CTAs share an SM), a warp for 32 rows and a quarter (half) of the columns: tcgen05.ld (32x32b) -> registers
//            -> per-warp shared staging (swizzled fp32) -> every lane then owns 8 consecutive columns of one row, so that bias, activation, activation
//            gradient, dropout (counter-based), residual add and the store are all 16-byte coalesced accesses
// The accumulator is double-buffered in tensor memory (2 x BN columns): the epilogue of unit i overlaps the MMAs of unit i+1.
//
// Split-K: with accumulate == 2 the launcher may cut K into slices; every slice adds its partial tile to the fp32 output
// with vector atomics. This is what the weight gradient dW += X^T·dY uses (few output tiles, long contraction).
//
// Every mbarrier wait is bounded. A wait that gives up raises the CTA's abort flag and writes a status word; all roles
// leave their loops, the CTA waits for its TMA copies in flight, frees its tensor memory and returns.
#include "gemm_epilogue.cuh"
#include <algorithm>
#include <cstring>
#include <cstdlib>

using namespace rbt;
using namespace rbg;

namespace {

constexpr int BM = 128;
constexpr int kBarrierBytes = 256;
constexpr int kMaxStages = 8;

// What a CTA of the kernel has: one per SM with a long ring and 16 epilogue warps, or two per SM with 8 for batched problems of few K blocks, where a unit
// is a chain of first load, few products and epilogue that one CTA's two accumulators do not hide. 36 x 333 frames, 8 heads (lengths from half on):
// dV 16.8 -> 14.7 us, position gradient 24.7 -> 18.0; 20 x 500 frames 17.8 -> 17.4 and 24.9 -> 19.8. Three CTAs with two stages each: 15.2 and 21.3;
// a CTA per unit, handed out by the hardware: 20.9 and 17.9. Products of whole rows (attention scores and band, one K block) within a pass of 6912
// rows: 23 and 34 -> 16.7 us each, most of it by boxes of 128-byte rows that are written while the unit after them is multiplied.
template <int BN, int CTAS>
struct Layout {
  static constexpr bool kBoxes = CTAS > 1 && BN == 128;  // (whole rows of the output: bulk stores of 32 rows x 64 columns)
  static constexpr bool kNext = CTAS > 1 && BN == 64;    // (two sets of problems in one launch, see gemm.h)
  static constexpr int kWarps = CTAS > 1 ? 8 : kEpilogueWarps;
  static constexpr int kThreads = 64 + kWarps * 32;
  static constexpr int kStageBytes = (BM + BN) * BK * 2;
  static constexpr int kStages = CTAS == 1 ? 196608 / kStageBytes : BN == 128 ? 2 : 3;
  static constexpr int kRingBytes = kStages * kStageBytes;
  static constexpr int kStaging = kBoxes ? kStoreBoxBytesPerWarp : kStagingBytesPerWarp;  // per warp
  static constexpr int kSmemBytes = kRingBytes + kWarps * kStaging + kBarrierBytes + 1024;
  static_assert(kStages <= kMaxStages && kStages >= 2 && CTAS * (kSmemBytes + 1024) <= 228 * 1024 && CTAS * 2 * BN <= 512, "layout");
};

template <int BN, bool FULL, int CTAS>
__global__ void __launch_bounds__(Layout<BN, CTAS>::kThreads, CTAS)
gemm_persist_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_c,
                    const __grid_constant__ CUtensorMap tm_a2, const __grid_constant__ CUtensorMap tm_b2, const Params p) {
  constexpr int kTileBytesA = BM * BK * 2;
  using L = Layout<BN, CTAS>;
  constexpr int kStageBytes = L::kStageBytes, kStages = L::kStages;
  constexpr uint32_t kTmemCols = 2 * BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* staging = reinterpret_cast<float*>(smem + L::kRingBytes);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kRingBytes + L::kWarps * L::kStaging);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* acc_full = empty_bar + kMaxStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const RbGemm& g = p.g;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], L::kWarps);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    prefetch_map(&tm_a);
    prefetch_map(&tm_b);
    if (L::kBoxes) prefetch_map(&tm_c);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // several CTAs per SM: no tensor memory is taken before the kernel in front has given its own back, and none of the next kernel's before this one
  // has (a CTA of either that waits for tensor memory while it is waited for itself would never get it)
  if (CTAS > 1) rb_pdl_wait();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // everything above touched no global memory: it may overlap the tail of the preceding kernel
  if (CTAS == 1) rb_pdl_wait();
  rb_pdl_launch();
  if (warp == 0) {
    // ---------------- TMA producer: the warp walks, one lane of it issues ----------------
    uint32_t it = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
      const Unit w = decode_unit<BM, BN>(p, u);
      if (!w.valid) continue;
      const int m0 = w.m0, n0 = w.n0;
      const CUtensorMap *map_a = L::kNext && w.next ? &tm_a2 : &tm_a, *map_b = L::kNext && w.next ? &tm_b2 : &tm_b;
      BandWalk walk(g, w, BM);
      for (int kb = w.kb0; kb < w.kb1; ++kb) {
        if (walk.skip(kb == w.kb0)) continue;
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        ++it;
        if (!warp_wait(&empty_bar[s], ph ^ 1u, abort_flag)) {
          *abort_flag = 1;
          if (g.status && lane == 0) atomicCAS(g.status, 0, (1 << 24) | (kb & 0xFFFFFF));
          ok = false;
          break;
        }
        uint8_t* sa = smem + s * kStageBytes;
        uint8_t* sb = sa + kTileBytesA;
        const int k0 = kb * BK;
        // (rows past the end of the matrix are read as zeros)
        const int a_row = walk.zeros ? (int)g.a_rows : w.a_r0 + k0, b_row = walk.zeros ? (int)g.b_rows : w.b_r0 + k0;
        if (elect_one()) {
          mbar_expect_tx(&full_bar[s], kStageBytes);
          if (!g.a_mn_major) {
            tma_load_2d(sa, map_a, w.a_c0 + k0, w.a_r0 + m0, &full_bar[s]);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * 8192, map_a, w.a_c0 + m0 + 64 * j, a_row, &full_bar[s]);
          }
          if (!g.b_mn_major) {
            tma_load_2d(sb, map_b, w.b_c0 + k0, w.b_r0 + n0, &full_bar[s]);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, map_b, w.b_c0 + n0 + 64 * j, b_row, &full_bar[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the warp walks, one lane of it issues ----------------
    const uint32_t ab_fmt = g.ab_fp16 ? 0u : 1u;  // operand format field: 0 = fp16, 1 = bf16 (accumulator fp32 either way)
    const uint32_t idesc = (1u << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((uint32_t)(g.a_mn_major ? 1 : 0) << 15) |
                           ((uint32_t)(g.b_mn_major ? 1 : 0) << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    const uint32_t a_lo = desc_lo(smem_u32(smem), g.a_mn_major ? 8192 : 16), b_lo = desc_lo(smem_u32(smem) + kTileBytesA, g.b_mn_major ? 8192 : 16);
    // K-major: 16 elements = 32 bytes along the swizzled row; MN-major: 16 K-rows of 128 bytes = 2 swizzle atoms, 64-wide MN groups 8192 bytes apart
    const uint32_t a_step = g.a_mn_major ? 128 : 2, b_step = g.b_mn_major ? 128 : 2;
    uint32_t it = 0, t_local = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
      const Unit w = decode_unit<BM, BN>(p, u);
      if (!w.valid) continue;
      const int kb0 = w.kb0, kb1 = w.kb1;
      const uint32_t buf = t_local & 1u;
      if (!warp_wait(&acc_empty[buf], ((t_local >> 1) & 1u) ^ 1u, abort_flag)) {
        *abort_flag = 1;
        if (g.status && lane == 0) atomicCAS(g.status, 0, (4 << 24) | (u & 0xFFFFFF));
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d_tmem = tmem_base + buf * BN;
      BandWalk walk(g, w, BM);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (walk.skip(kb == kb0)) continue;
        const int s = it % kStages;
        const uint32_t ph = (it / kStages) & 1u;
        ++it;
        if (!warp_wait(&full_bar[s], ph, abort_flag)) {
          *abort_flag = 1;
          if (g.status && lane == 0) atomicCAS(g.status, 0, (2 << 24) | (kb & 0xFFFFFF));
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = a_lo + s * (kStageBytes >> 4), b = b_lo + s * (kStageBytes >> 4);
        umma_f16_warp(d_tmem, a, b, idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
        for (int kk = 1; kk < BK / 16; ++kk) umma_f16_warp(d_tmem, a + kk * a_step, b + kk * b_step, idesc, 1u);
        umma_commit_warp(&empty_bar[s]);
      }
      if (ok) umma_commit_warp(&acc_full[buf]);
      ++t_local;
    }
  } else {
    // ---------------- epilogue: TMEM lane quarter = warp % 4 ----------------
    const int q = warp & 3;
    float* stg = staging + (warp - 2) * (L::kStaging / 4);
    uint32_t t_local = 0;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
      const Unit w = decode_unit<BM, BN>(p, u);
      if (!w.valid) continue;
      const int m0 = w.m0, n0 = w.n0;
      const uint32_t buf = t_local & 1u;
      bool ok = mbar_wait(&acc_full[buf], (t_local >> 1) & 1u, abort_flag);
      if (!ok && lane == 0) {
        *abort_flag = 1;
        if (g.status) atomicCAS(g.status, 0, (3 << 24) | (u & 0xFFFFFF));
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t_addr = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      const int part = (warp - 2) >> 2;  // four (two) warps per lane quarter, each with a quarter (half) of the columns
      constexpr int kCols = BN / (L::kWarps / 4);
      if (L::kBoxes)
        epilogue_boxes(p, w, (int)(w.c_off / g.ldc), t_addr, part * 64, reinterpret_cast<uint8_t*>(stg), &tm_c, lane, q, [&]() { mbar_arrive(&acc_empty[buf]); });
      else
        epilogue_columns<FULL, L::kNext>(p, w, m0, n0, t_addr, part * kCols, (part + 1) * kCols, stg, lane, q, [&]() { mbar_arrive(&acc_empty[buf]); });
      ++t_local;
    }
    if (L::kBoxes && lane == 0) tma_store_wait_read();  // before the shared memory is handed on
  }

  // ---------------- teardown ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // let copies that are still in flight land before the shared memory goes away (bounded: about 1 ms)
    for (uint32_t i = 0; i < (1u << 12); ++i) __nanosleep(256);
  }
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

bool epilogue_full(const RbGemm& g) { return g.dact_z != nullptr || g.drop_p > 0.f || g.resid != nullptr; }

bool aligned16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }  // (also: not there)

// whether the problems of a batch own whole rows of an output that bulk stores can write (see gemm.h)
bool boxes_ok(const RbGemm& g) {
  return !epilogue_full(g) && g.batch > 0 && g.c_rows > 0 && !g.out_fp32 && !g.c2 && !g.bias && !g.act && g.ldc % 8 == 0 && aligned16(g.c) &&
         g.c_sb % g.ldc == 0 && g.c_sh % g.ldc == 0;
}

template <int BN, int CTAS>
int launch(const RbGemm& g, cudaStream_t stream) {
  using L = Layout<BN, CTAS>;
  constexpr bool kFull = CTAS == 1;  // several CTAs per SM: the plain epilogue only
  static RbPerDevice attr_set;
  if (attr_set.needed()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_persist_kernel<BN, false, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemBytes);
    if (kFull && e == cudaSuccess) e = cudaFuncSetAttribute(gemm_persist_kernel<BN, kFull, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmemBytes);
    if (e != cudaSuccess) {
      rb_set_error("gemm: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return RB_ERR_LAUNCH;
    }
    attr_set.done();
  }
  Params p;
  p.g = g;
  p.tiles_m = (g.m + BM - 1) / BM;
  p.tiles_n = (g.n + BN - 1) / BN;
  p.num_kb = (g.k + BK - 1) / BK;
  const int tiles = p.tiles_m * p.tiles_n;
  const int sms = num_sms();
  int split = 1;
  if (g.accumulate == 2) {
    split = g.split_k > 0 ? g.split_k : (tiles >= sms ? 1 : sms / tiles);
    const int max_split = p.num_kb >= 4 ? p.num_kb / 4 : 1;  // at least 4 K blocks per slice
    if (split > max_split) split = max_split;
    if (split < 1) split = 1;
  }
  p.kb_per_split = (p.num_kb + split - 1) / split;
  p.split = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;  // no empty slices
  p.units = tiles * p.split;
  if (g.batch > 0) {
    p.split = 1;
    p.units = tiles * g.batch * (g.a_next ? 2 : 1);
  }
  p.c_next = 0;
  p.alpha_first = g.alpha;
  if (g.a_next) {
    p.c_next = (static_cast<const char*>(g.c_next) - static_cast<const char*>(g.c)) / (g.out_fp32 ? 4 : 2);
    p.g.alpha = 1.f;
  }
  p.vec_ok = (g.ldc % 8 == 0) && aligned16(g.c) && aligned16(g.c2) && aligned16(g.resid) && aligned16(g.dact_z);
  p.bias_vec = g.bias != nullptr && !g.bias_bf16 && aligned16(g.bias);
  CUtensorMap tm_a, tm_b, tm_c, tm_a2, tm_b2;
  memset(&tm_c, 0, sizeof(tm_c));
  int st;
  p.tma_store = L::kBoxes;
  if (L::kBoxes) {
    st = make_map(&tm_c, g.c, g.ldc, g.c_rows, g.ldc, 64, 32);
    if (st) return st;
  }
  long long a_rows = g.a_mn_major ? g.k : g.m, a_cols = g.a_mn_major ? g.m : g.k;
  long long b_rows = g.b_mn_major ? g.k : g.n, b_cols = g.b_mn_major ? g.n : g.k;
  if (g.batch > 0) {
    a_rows = g.a_rows; a_cols = g.a_cols; b_rows = g.b_rows; b_cols = g.b_cols;
  }
  auto operand_a = [&](CUtensorMap* map, const void* at) {
    return g.a_mn_major ? make_map(map, at, a_cols, a_rows, g.lda, 64, BK) : make_map(map, at, a_cols, a_rows, g.lda, BK, BM);
  };
  auto operand_b = [&](CUtensorMap* map, const void* at) {
    return g.b_mn_major ? make_map(map, at, b_cols, b_rows, g.ldb, 64, BK) : make_map(map, at, b_cols, b_rows, g.ldb, BK, BN);
  };
  st = operand_a(&tm_a, g.a);
  if (!st) st = operand_b(&tm_b, g.b);
  tm_a2 = tm_a;
  tm_b2 = tm_b;
  if (!st && g.a_next) st = operand_a(&tm_a2, g.a_next);
  if (!st && g.a_next) st = operand_b(&tm_b2, g.b_next);
  if (st) return st;
  int grid = p.units < CTAS * sms ? p.units : CTAS * sms;
  {
    // tuning knob: cap the number of CTAs (for bandwidth / latency experiments)
    static int cap = -1;
    if (cap < 0) {
      const char* e = getenv("RETURNN_B200_GEMM_MAX_CTAS");
      cap = e ? atoi(e) : 0;
    }
    if (cap > 0 && grid > cap) grid = cap;
  }
  if (kFull && epilogue_full(g)) rb_launch_pdl(gemm_persist_kernel<BN, kFull, CTAS>, dim3(grid), dim3(L::kThreads), L::kSmemBytes, stream, tm_a, tm_b, tm_c, tm_a2, tm_b2, p);
  else rb_launch_pdl(gemm_persist_kernel<BN, false, CTAS>, dim3(grid), dim3(L::kThreads), L::kSmemBytes, stream, tm_a, tm_b, tm_c, tm_a2, tm_b2, p);
  return rb_check_launch("gemm_persist");
}

}  // namespace

int rb_gemm(const RbGemm& g, cudaStream_t stream) {
  if (g.m <= 0 || g.n <= 0) return RB_OK;
  if (g.k <= 0 && !(g.batch > 0 && g.k_from_lens)) {
    rb_set_error("gemm: k=%d", g.k);
    return RB_ERR_ARG;
  }
  if (g.batch > 0 && (g.accumulate == 2 || g.split_k > 1 || g.a_rows <= 0 || g.a_cols <= 0 || g.b_rows <= 0 || g.b_cols <= 0)) {
    rb_set_error("gemm: the batched form needs the stored extents and supports no split-K");
    return RB_ERR_ARG;
  }
  if ((g.lda % 8) || (g.ldb % 8) || (reinterpret_cast<uintptr_t>(g.a) & 15) || (reinterpret_cast<uintptr_t>(g.b) & 15)) {
    rb_set_error("gemm: operands need 16-byte aligned bases and pitches that are multiples of 8 elements (lda %d ldb %d)", g.lda, g.ldb);
    return RB_ERR_ARG;
  }
  if (g.accumulate && !g.out_fp32) {
    rb_set_error("gemm: accumulate needs fp32 output");
    return RB_ERR_ARG;
  }
  if (g.out_fp32 && (g.c2 || g.resid)) {
    rb_set_error("gemm: second output / residual need bf16 output");
    return RB_ERR_ARG;
  }
  if (g.drop_p > 0.f && (!g.seed || !g.offset || (g.ldc % 8) || !(g.drop_p < 1.f))) {
    rb_set_error("gemm: dropout epilogue needs seed/offset pointers, ldc %% 8 == 0 and p < 1 (ldc %d, p %f)", g.ldc, g.drop_p);
    return RB_ERR_ARG;
  }
  if (g.a_next && (g.batch <= 0 || g.n > 64 || epilogue_full(g) || g.bias || g.act || g.c2 || g.win || !g.b_next || !g.c_next || !aligned16(g.a_next) ||
                   !aligned16(g.b_next) || !aligned16(g.c_next))) {
    rb_set_error("gemm: a second set of problems needs the batched form, at most 64 columns and a plain epilogue");
    return RB_ERR_ARG;
  }
  if (g.win && (g.batch <= 0 || g.heads <= 0 || (g.win == 1 ? !g.lens || !g.m_from_lens
                                                            : !g.a_mn_major || !g.win_lens || g.win_lp <= 0 || g.win_lp % BK || g.k % BK || g.k_from_lens))) {
    rb_set_error("gemm: windows need the batched form, lengths and blocks of whole sequences");
    return RB_ERR_ARG;
  }
  if (g.split_k > 1 && g.accumulate != 2) {
    rb_set_error("gemm: split_k needs accumulate == 2");
    return RB_ERR_ARG;
  }
  if (g.seg_a > 0 && (!rb_gemm_pair_wanted(g) || g.a_mn_major || !g.b_mn_major || g.accumulate == 2)) {
    rb_set_error("gemm: split operands need the CTA-pair kernel, A stored [m][k] and B stored [k][n]");
    return RB_ERR_UNSUPPORTED;
  }
  if (rb_gemm_pair_wanted(g)) return rb_gemm_pair(g, stream);
  // Narrow tiles where wider ones would load and multiply columns that are not wanted: one head of 64 columns, the windows of a band
  if (g.n > 64 && boxes_ok(g)) return launch<128, 2>(g, stream);
  if (g.n > 128 && g.win != 1) return launch<256, 1>(g, stream);
  if (g.n > 64) return launch<128, 1>(g, stream);
  // (with a unit per SM or less there is nothing to overlap, and tensor memory is to be had before the kernel in front has ended: 4 x 50 frames
  // 4.0 us, with two CTAs per SM 4.5)
  if (g.a_next) return launch<64, 2>(g, stream);
  if (g.batch > 0 && !epilogue_full(g) && (long long)((g.m + BM - 1) / BM) * g.batch > num_sms()) return launch<64, 2>(g, stream);
  return launch<64, 1>(g, stream);
}

// C entry points with the full epilogue (see gemm.h for the meaning of the arguments); the second reads A and B as fp16
static int gemm_ex(const void* a, const void* b, void* c, void* c2, const void* bias, int m, int n, int k, int lda, int ldb, int ldc, int a_mn_major,
                   int b_mn_major, int bias_bf16, int act, int out_fp32, int accumulate, float alpha, const void* dact_z, float drop_p,
                   const long long* seed, const long long* offset, unsigned long long drop_site, const void* resid, float res_scale, int split_k,
                   int* status, int ab_fp16, cudaStream_t stream) {
  RbGemm g;
  g.a = a; g.b = b; g.c = c; g.c2 = c2; g.bias = bias; g.bias_bf16 = bias_bf16;
  g.m = m; g.n = n; g.k = k; g.lda = lda; g.ldb = ldb; g.ldc = ldc;
  g.a_mn_major = a_mn_major; g.b_mn_major = b_mn_major; g.ab_fp16 = ab_fp16;
  g.act = act; g.out_fp32 = out_fp32; g.accumulate = accumulate; g.alpha = alpha;
  g.dact_z = dact_z; g.drop_p = drop_p; g.seed = seed; g.offset = offset; g.drop_site = drop_site;
  g.resid = resid; g.res_scale = res_scale; g.split_k = split_k; g.status = status;
  return rb_gemm(g, stream);
}

RB_EXPORT int rb200_gemm_bf16_ex(const void* a, const void* b, void* c, void* c2, const void* bias, int m, int n, int k, int lda, int ldb,
                                 int ldc, int a_mn_major, int b_mn_major, int bias_bf16, int act, int out_fp32, int accumulate, float alpha,
                                 const void* dact_z, float drop_p, const long long* seed, const long long* offset,
                                 unsigned long long drop_site, const void* resid, float res_scale, int split_k, int* status,
                                 cudaStream_t stream) {
  return gemm_ex(a, b, c, c2, bias, m, n, k, lda, ldb, ldc, a_mn_major, b_mn_major, bias_bf16, act, out_fp32, accumulate, alpha, dact_z, drop_p, seed,
                 offset, drop_site, resid, res_scale, split_k, status, 0, stream);
}

RB_EXPORT int rb200_gemm_fp16_ex(const void* a, const void* b, void* c, void* c2, const void* bias, int m, int n, int k, int lda, int ldb,
                                 int ldc, int a_mn_major, int b_mn_major, int bias_bf16, int act, int out_fp32, int accumulate, float alpha,
                                 const void* dact_z, float drop_p, const long long* seed, const long long* offset,
                                 unsigned long long drop_site, const void* resid, float res_scale, int split_k, int* status,
                                 cudaStream_t stream) {
  return gemm_ex(a, b, c, c2, bias, m, n, k, lda, ldb, ldc, a_mn_major, b_mn_major, bias_bf16, act, out_fp32, accumulate, alpha, dact_z, drop_p, seed,
                 offset, drop_site, resid, res_scale, split_k, status, 1, stream);
}

// Gradients of keys and values of attention with heads of 64 columns over padded sequences, both products in one launch (36 x 333 frames, 8 heads: two
// launches 33.2 us, one 28.1; 20 x 500: 37.8 and 30.8; 4 x 50: 7.8 and 4.7): dv = p^T d_o, dk = scale * ds^T q; p, ds [B*H, lp, lp], the rest [B, lp, heads * 64]
RB_EXPORT int rb200_att_dkv(const void* p, const void* d_o, const void* ds, const void* q, void* dv, void* dk, const int* lens, int batch, int heads, int lp,
                            float scale, int* status, cudaStream_t stream) {
  if (batch <= 0 || heads <= 0 || lp <= 0) return RB_OK;
  const int hd = heads * 64;
  RbGemm g;
  g.a = p; g.b = d_o; g.c = dv;
  g.a_next = ds; g.b_next = q; g.c_next = dk; g.alpha_next = scale;
  g.m = lp; g.n = 64; g.k = lp; g.lda = lp; g.ldb = hd; g.ldc = hd;
  g.a_mn_major = g.b_mn_major = 1; g.status = status;
  g.batch = batch * heads; g.heads = heads;
  g.a_rb = (long long)heads * lp; g.a_rh = lp; g.b_rb = lp; g.b_ch = 64; g.c_sb = (long long)lp * hd; g.c_sh = 64;
  g.a_rows = (long long)batch * heads * lp; g.a_cols = lp; g.b_rows = (long long)batch * lp; g.b_cols = hd;
  g.lens = lens; g.m_from_lens = g.k_from_lens = 1;
  return rb_gemm(g, stream);
}

// whether rb200_gemm_fp16_split takes a product of this size (the CTA-pair kernel can be switched off by the environment)
RB_EXPORT int rb200_gemm_fp16_split_supported(int m, int n) {
  RbGemm g;
  g.m = m; g.n = n;
  return rb_gemm_pair_wanted(g) ? 1 : 0;
}

// c[m,n] (fp32) = A·B with fp16 operands split in two: A = hi + lo, hi stored [m][k] at `a` and lo a_lo_rows rows further on, B likewise
// stored [k][n]; the product of the two lo parts (2^-22 of the result) is left out. RB_ERR_UNSUPPORTED: not a shape of the CTA-pair kernel.
RB_EXPORT int rb200_gemm_fp16_split(const void* a, const void* b, void* c, int m, int n, int k, int lda, int ldb, int ldc, int a_lo_rows, int b_lo_rows,
                                    int* status, cudaStream_t stream) {
  RbGemm g;
  g.a = a; g.b = b; g.c = c; g.m = m; g.n = n; g.k = k; g.lda = lda; g.ldb = ldb; g.ldc = ldc;
  g.b_mn_major = 1; g.ab_fp16 = 1; g.out_fp32 = 1; g.status = status;
  g.seg_a = a_lo_rows; g.seg_b = b_lo_rows;
  if (a_lo_rows < m || b_lo_rows < k) {
    rb_set_error("gemm_fp16_split: the lo rows overlap the hi rows");
    return RB_ERR_ARG;
  }
  return rb_gemm(g, stream);
}

RB_EXPORT int rb200_sum_slices_f32(const float* x, float* y, int slices, long long n, cudaStream_t stream);

// Rows of x and dy per slice of a weight gradient x^T dy that is the same in every run (rb200_weight_grad_sliced); 0: one product. Where the result
// has few tiles and the contraction is long, it is cut into slices whose products are added in their order.
// One CTA per tile of 128 x 256 and slice, all of them at once; at least 256 rows per slice (shorter ones gain less than the sum of the
// slices costs); no more than 12, from where the slices that are written and read again cost more than shorter products save.
// 6656 x 512 x 512: 12 slices 16 us, one 42; 25000 x 512 x 512: 26 and 138; 6656 x 512 x 2048: 4 slices 24 us, one 43 (slices that add
// onto one result by atomics, in any order: 13, 19 and 21 us); 600 x 512 x 512: 2 slices 12.5, one 11.2
RB_EXPORT int rb200_weight_grad_slices(int m, int k, int n) {
  const long long tiles = (long long)((k + 127) / 128) * ((n + 255) / 256);
  if (m <= 0 || tiles <= 0) return 0;
  const int slices = (int)std::min<long long>({148 / tiles, 12, m / 256});
  return slices <= 1 ? 0 : ((m + slices - 1) / slices + 63) / 64 * 64;  // (rows past the last one are read as zeros)
}

// dw [k][n] (fp32) = x^T dy, x [m][k], dy [m][n] bf16: one product per slice of `rows` rows into part [ceil(m / rows)][k][n], then their sum in
// the order of the slices
RB_EXPORT int rb200_weight_grad_sliced(const void* x, const void* dy, float* part, float* dw, int m, int k, int n, int rows, int* status,
                                       cudaStream_t stream) {
  if (m <= 0 || rows <= 0) {
    rb_set_error("weight_grad_sliced: m=%d rows=%d", m, rows);
    return RB_ERR_ARG;
  }
  RbGemm g;
  g.a = x; g.b = dy; g.c = part; g.m = k; g.n = n; g.k = rows; g.lda = k; g.ldb = n; g.ldc = n;
  g.a_mn_major = 1; g.b_mn_major = 1; g.out_fp32 = 1; g.status = status;
  const int slices = (m + rows - 1) / rows;
  RbGemm pair = g;
  pair.k = m;
  pair.slice_k = rows;
  if (rb_gemm_slices(pair)) {  // the same slices with tiles of 256 x 256 by CTA pairs (6656 x 512 x 2048, four slices: 23 -> 20 us in a profile)
    const int st = rb_gemm(pair, stream);
    return st ? st : rb200_sum_slices_f32(part, dw, slices, (long long)k * n, stream);
  }
  g.batch = slices; g.heads = 1;
  g.a_rb = rows; g.b_rb = rows; g.c_sb = (long long)k * n;
  g.a_rows = m; g.a_cols = k; g.b_rows = m; g.b_cols = n;
  const int st = rb_gemm(g, stream);
  return st ? st : rb200_sum_slices_f32(part, dw, slices, (long long)k * n, stream);
}

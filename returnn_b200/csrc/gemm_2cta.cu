// CTA-pair variant of the persistent bf16 GEMM: two CTAs of a cluster (two SMs) compute one 256 x 256 output tile with
// tcgen05.mma.cta_group::2. Each CTA loads its own 128 rows of A and half of the B tile, so a pair moves 64 KB per K block for
// 256 x 256 x 64 multiply-adds: two thirds of the operand traffic per flop of the one-CTA kernel (128 x 256 tiles, 48 KB per
// CTA and K block). The traffic does not bound it: 148 SMs fetch 19 TB/s by TMA from the L2 (69 bytes per cycle and SM), a pair needs 64 KB per
// 512 cycles. What does is, beside the multiplication (512 cycles per K block; 612 while one lane on its own issued it), the fixed time of a
// product (first load 1.3 us, last epilogue 2.9, teardown 1.2, of 7.5 us at 6912 x 512 x 512) and waves of few tiles (54 on 74 pairs for n = 512).
//
// Roles per CTA: warp 0 = TMA producer (loads with .cta_group::2 and no multicast; they complete on the *leader's* full barrier,
// which is armed for the bytes of both CTAs), warp 1 = TMEM allocation, and in the leader CTA (cluster rank 0) the MMA issuer,
// warps 2-17 = epilogue of the CTA's own 128 accumulator rows (tensor memory is per SM): every lane owns one row, reads 64 columns of
// it from tensor memory, and the results leave through a swizzled box in shared memory and one bulk tensor store per warp (bulk
// reduce-add for the accumulating fp32 outputs of the weight gradients); see epilogue_rows_tma. Outputs that a tensor map cannot
// describe (unaligned pitch or base) take the per-lane st.global path. tcgen05.commit with a cluster
// multicast mask releases a ring stage / publishes an accumulator in both CTAs at once; the epilogue warps of both CTAs arrive on
// the leader's "accumulator free" barrier. All waits are bounded; a CTA never exits before its peer (cluster barrier at the end),
// because the leader's MMAs read the peer's shared memory.
#include "gemm_epilogue.cuh"
#include <cstdlib>
#include <cstring>

using namespace rbt;
using namespace rbg;

namespace {

constexpr int BM = 256;              // per pair; 128 per CTA
constexpr int BN = 256;
constexpr int kThreads = kGemmThreads;
constexpr int kTileBytesA = 128 * BK * 2;        // 16 KB: this CTA's rows of A
constexpr int kTileBytesB = (BN / 2) * BK * 2;   // 16 KB: this CTA's half of B
constexpr int kStageBytes = kTileBytesA + kTileBytesB;
constexpr int kStages = 5;
constexpr int kRingBytes = kStages * kStageBytes;  // 160 KB
constexpr int kStagingBytes = kEpilogueWarps * kStoreBoxBytesPerWarp;  // 64 KB: one 4 KB store box per epilogue warp (1024-byte aligned)
static_assert(kStoreBoxBytesPerWarp >= kStagingBytesPerWarp, "the st.global path stages in the same area");
constexpr int kSmemBytes = kRingBytes + kStagingBytes + 256 + 1024;
constexpr uint32_t kTmemCols = 2 * BN;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Orders execution only: what the CTAs share goes through mbarriers (their initialisation through fence.mbarrier_init). With .release the arrival
// waits for all stores before it, 0.7 us at the end of every product.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// Relaxed: what is handed over is tensor memory, which tcgen05.wait::ld and tcgen05.fence order; .release took 1100 cycles per tile and warp.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
// (one lane of a converged warp, see umma_f16_warp)
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "n"(kDescHi)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs once the pair's MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(smem_u32(bar)), "h"(mask)
               : "memory");
}

// The units of a pair, one after another: (slice of the contraction, row of tiles, column of tiles), with one division at the start. Divisions per
// unit left the producer 500 cycles late at every tile.
struct Walk {
  const Params& p;
  int u, sp, mi, ni;
  __device__ __forceinline__ Walk(const Params& p_, int first) : p(p_), u(first) {
    const int tiles = p.tiles_m * p.tiles_n;
    sp = p.split > 1 ? u / tiles : 0;
    const int t = u - sp * tiles;
    mi = t / p.tiles_n;
    ni = t - mi * p.tiles_n;
  }
  __device__ __forceinline__ bool more() const { return u < p.units; }
  __device__ __forceinline__ void next() {
    u += p.step;
    sp += p.step_sp;
    mi += p.step_m;
    ni += p.step_n;
    if (ni >= p.tiles_n) {
      ni -= p.tiles_n;
      ++mi;
    }
    if (mi >= p.tiles_m) {
      mi -= p.tiles_m;
      ++sp;
    }
  }
  __device__ __forceinline__ int kb0() const { return sp * p.kb_per_split; }
  __device__ __forceinline__ int kb1() const { return min(p.num_kb, (sp + 1) * p.kb_per_split); }
};

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const __grid_constant__ CUtensorMap tm_c,
                 const __grid_constant__ CUtensorMap tm_c2, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* staging = reinterpret_cast<float*>(smem + kRingBytes);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kRingBytes + kStagingBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_full = empty_bar + kStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const RbGemm& g = p.g;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);   // leader: one expect_tx arrival per use, both CTAs' bytes
      mbar_init(&empty_bar[s], 1);  // one multicast commit per use
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 2 * kEpilogueWarps);  // leader: the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    prefetch_map(&tm_a);
    prefetch_map(&tm_b);
    if (p.tma_store) prefetch_map(&tm_c);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // barriers of both CTAs are initialised before anyone signals across
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // everything above touched no global memory: it may overlap the tail of the preceding kernel. The roles wait for that one themselves, with their
  // first unit at hand.
  rb_pdl_launch();

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs): the warp walks, one lane of it issues ----------------
    const uint32_t full0 = map_to_cta(smem_u32(full_bar), 0);  // the leader's barriers collect both CTAs' bytes
    uint32_t s = 0, ph = 0;
    bool ok = true;
    Walk w(p, pair);
    rb_pdl_wait();
    for (; w.more() && ok; w.next()) {
      const int m0 = w.mi * BM + (int)rank * 128;
      const int n0 = w.ni * BN + (int)rank * (BN / 2);
      const int kb1 = w.kb1();
      for (int kb = w.kb0(); kb < kb1; ++kb) {
        if (!warp_wait(&empty_bar[s], ph ^ 1u, abort_flag)) {
          *abort_flag = 1;
          if (g.status && lane == 0) atomicCAS(g.status, 0, (1 << 24) | (kb & 0xFFFFFF));
          ok = false;
          break;
        }
        uint8_t* sa = smem + s * kStageBytes;
        uint8_t* sb = sa + kTileBytesA;
        const uint32_t bar = full0 + s * 8;
        const bool issuer = elect_one();
        if (issuer && leader) mbar_expect_tx(&full_bar[s], 2 * kStageBytes);
        // split operands: block kb belongs to hi*lo, lo*hi or hi*hi (columns of A past k read zeros, so the rows of B there do not
        // count). The small products come first: additions to a large accumulator are what the tensor core rounds
        const int seg = p.seg_kb ? kb / p.seg_kb : 0;
        const int k0 = (kb - seg * p.seg_kb) * BK;
        const int a_row = p.seg_kb && seg == 1 ? g.seg_a : 0, b_row = p.seg_kb && seg == 0 ? g.seg_b : 0;
        if (issuer) {
          if (!g.a_mn_major) {
            tma_load_2d_pair(sa, &tm_a, k0, a_row + m0, bar);
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) tma_load_2d_pair(sa + j * 8192, &tm_a, m0 + 64 * j, k0, bar);
          }
          if (!g.b_mn_major) {
            tma_load_2d_pair(sb, &tm_b, k0, n0, bar);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_pair(sb + j * 8192, &tm_b, n0 + 64 * j, b_row + k0, bar);
          }
        }
        if (++s == kStages) {
          s = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    if (leader) {
      // ---------------- MMA issuer (leader CTA only): the warp walks, one lane of it issues ----------------
      const uint32_t ab_fmt = g.ab_fp16 ? 0u : 1u;  // operand format field: 0 = fp16, 1 = bf16 (accumulator fp32 either way)
      const uint32_t idesc = (1u << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((uint32_t)(g.a_mn_major ? 1 : 0) << 15) |
                             ((uint32_t)(g.b_mn_major ? 1 : 0) << 16) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint32_t a_lo = desc_lo(smem_u32(smem), g.a_mn_major ? 8192 : 16), b_lo = desc_lo(smem_u32(smem) + kTileBytesA, g.b_mn_major ? 8192 : 16);
      const uint32_t a_step = g.a_mn_major ? 128 : 2, b_step = g.b_mn_major ? 128 : 2;  // 16 of the contraction, in units of 16 bytes
      uint32_t s = 0, ph = 0, t_local = 0;
      bool ok = true;
      for (Walk w(p, pair); w.more() && ok; w.next()) {
        const uint32_t buf = t_local & 1u;
        if (!warp_wait(&acc_empty[buf], ((t_local >> 1) & 1u) ^ 1u, abort_flag)) {
          *abort_flag = 1;
          if (g.status && lane == 0) atomicCAS(g.status, 0, (4 << 24) | (w.u & 0xFFFFFF));
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_tmem = tmem_base + buf * BN;
        const int kb0 = w.kb0(), kb1 = w.kb1();
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!warp_wait(&full_bar[s], ph, abort_flag)) {
            *abort_flag = 1;
            if (g.status && lane == 0) atomicCAS(g.status, 0, (2 << 24) | (kb & 0xFFFFFF));
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = a_lo + s * (kStageBytes >> 4), b = b_lo + s * (kStageBytes >> 4);
          umma_f16_pair(d_tmem, a, b, idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
          for (int kk = 1; kk < BK / 16; ++kk) umma_f16_pair(d_tmem, a + kk * a_step, b + kk * b_step, idesc, 1u);
          umma_commit_pair(&empty_bar[s]);
          if (++s == kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        if (ok) umma_commit_pair(&acc_full[buf]);
        ++t_local;
      }
    }
  } else {
    // ---------------- epilogue: this CTA's 128 rows ----------------
    const int q = warp & 3;
    uint8_t* box = reinterpret_cast<uint8_t*>(staging) + (warp - 2) * kStoreBoxBytesPerWarp;
    uint32_t t_local = 0;
    Walk walk(p, pair);
    Unit w = {};
    w.M = g.m;
    w.N = g.n;
    rb_pdl_wait();
    const EpiRng rng = EpiRng::load<KIND>(g);
    for (; walk.more(); walk.next()) {
      w.m0 = walk.mi * BM;
      w.n0 = walk.ni * BN;
      if (KIND == kEpiF32 && g.slice_k) w.c_r0 = walk.sp * g.m;
      const int m0 = w.m0 + (int)rank * 128, n0 = w.n0;
      const uint32_t buf = t_local & 1u;
      const int part = (warp - 2) >> 2;  // four warps per lane quarter, each with a quarter of the columns
      // the epilogue's global input of this lane's row (first 16 columns) is requested before the wait: it arrives while the tile is
      // still multiplied
      uint4 in_a = make_uint4(0u, 0u, 0u, 0u), in_b = in_a;
      const bool prefetched = epi_has_input(KIND) || (KIND == kEpiAny && p.tma_store && (g.dact_z != nullptr || g.resid != nullptr));
      if (prefetched) epilogue_prefetch16(p, w.M, w.N, m0 + q * 32 + lane, n0 + part * (BN / 4), in_a, in_b);
      bool ok = mbar_wait(&acc_full[buf], (t_local >> 1) & 1u, abort_flag);
      if (!ok && lane == 0) {
        *abort_flag = 1;
        if (g.status) atomicCAS(g.status, 0, (3 << 24) | (walk.u & 0xFFFFFF));
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t_addr = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      // (nobody waits for the buffers of the last two units: no arrival is on its way to the leader when the CTAs end)
      const bool reused = walk.u + 2 * p.step < p.units;
      auto release = [&]() {
        if (reused) mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty[buf]), 0));
      };
      if constexpr (!epi_generic(KIND))
        epilogue_kind_tma<KIND>(p, w, m0, n0, t_addr, part * (BN / 4), box, &tm_c, &tm_c2, lane, q, release, in_a, in_b, rng);
      else if (p.tma_store)
        epilogue_rows_tma<KIND == kEpiAny>(p, w, m0, n0, t_addr, part * (BN / 4), box, &tm_c, &tm_c2, lane, q, release, in_a, in_b, prefetched);
      else
        epilogue_columns<KIND == kEpiAny>(p, w, m0, n0, t_addr, part * (BN / 4), (part + 1) * (BN / 4), reinterpret_cast<float*>(box), lane, q, release);
      ++t_local;
    }
    // the bulk stores read this CTA's shared memory: the reads must have finished before the CTA exits and its shared memory is
    // handed to another CTA (the writes themselves complete like any other store of the grid)
    if (p.tma_store && lane == 0) tma_store_wait_read();
  }

  // ---------------- teardown ----------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (uint32_t i = 0; i < (1u << 12); ++i) __nanosleep(256);
  }
  __syncthreads();
  cluster_sync();  // the peer's MMAs and barrier signals may still touch this CTA's shared memory until here
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

}  // namespace

// whether rb_gemm should route this problem to the CTA-pair kernel
bool rb_gemm_pair_wanted(const RbGemm& g) {
  static int enabled = -1;
  if (enabled < 0) {
    const char* e = getenv("RETURNN_B200_GEMM_2CTA");
    enabled = (e && e[0] == '0') ? 0 : 1;
  }
  return enabled && g.batch == 0 && g.m > 128 && g.n > 128;
}

static bool tma_store_on() {
  static int enabled = -1;
  if (enabled < 0) {
    const char* e = getenv("RETURNN_B200_GEMM_TMA_STORE");
    enabled = (e && e[0] == '0') ? 0 : 1;
  }
  return enabled != 0;
}

static bool full_epilogue(const RbGemm& g) { return g.dact_z != nullptr || g.drop_p > 0.f || g.resid != nullptr; }

static bool aligned_outputs(const RbGemm& g) {
  auto al16 = [](const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return (g.ldc % 8 == 0) && al16(g.c) && al16(g.c2) && al16(g.resid) && al16(g.dact_z);
}

bool rb_gemm_column_sums(const RbGemm& g) {
  return rb_gemm_pair_wanted(g) && tma_store_on() && full_epilogue(g) && aligned_outputs(g) && g.c != nullptr && g.c2 == nullptr && !g.out_fp32;
}

bool rb_gemm_slices(const RbGemm& g) {
  return rb_gemm_pair_wanted(g) && tma_store_on() && aligned_outputs(g) && g.c != nullptr && g.out_fp32 && !g.accumulate && !full_epilogue(g) && !g.bias && !g.act &&
         !g.c2 && !g.seg_a && g.m % 32 == 0 && g.n % 8 == 0 && g.slice_k > 0 && g.slice_k % BK == 0;
}

int rb_gemm_pair(const RbGemm& g, cudaStream_t stream) {
  if (g.slice_k && !rb_gemm_slices(g)) {
    rb_set_error("gemm (pair): m=%d n=%d slice_k=%d is not a product in slices", g.m, g.n, g.slice_k);
    return RB_ERR_ARG;
  }
  if (g.colsum && !rb_gemm_column_sums(g)) {
    rb_set_error("gemm (pair): this problem's epilogue leaves no column sums");
    return RB_ERR_ARG;
  }
  using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const Params);
  static const Kernel kernels[] = {gemm_pair_kernel<kEpiSome>,  gemm_pair_kernel<kEpiAny>,       gemm_pair_kernel<kEpiPlain>, gemm_pair_kernel<kEpiF32>,
                                   gemm_pair_kernel<kEpiTwo>,   gemm_pair_kernel<kEpiTwoDrop>,   gemm_pair_kernel<kEpiResid>, gemm_pair_kernel<kEpiResidDrop>,
                                   gemm_pair_kernel<kEpiDact>,  gemm_pair_kernel<kEpiDactDrop>};
  static RbPerDevice attr_set;
  if (attr_set.needed()) {
    for (const Kernel k : kernels) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
      if (e != cudaSuccess) {
        rb_set_error("gemm (pair): cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        return RB_ERR_LAUNCH;
      }
    }
    attr_set.done();
  }
  Params p;
  p.g = g;
  p.tiles_m = (g.m + BM - 1) / BM;
  p.tiles_n = (g.n + BN - 1) / BN;
  p.num_kb = (g.k + BK - 1) / BK;
  p.seg_kb = g.seg_a > 0 ? p.num_kb : 0;
  if (p.seg_kb) p.num_kb *= 3;
  const int tiles = p.tiles_m * p.tiles_n;
  const int pairs_max = num_sms() / 2;
  int split = 1;
  if (g.accumulate == 2) {
    split = g.split_k > 0 ? g.split_k : (tiles >= pairs_max ? 1 : pairs_max / tiles);
    const int max_split = p.num_kb >= 4 ? p.num_kb / 4 : 1;
    if (split > max_split) split = max_split;
    if (split < 1) split = 1;
  }
  p.kb_per_split = g.slice_k ? g.slice_k / BK : (p.num_kb + split - 1) / split;
  p.split = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;
  p.units = tiles * p.split;
  p.vec_ok = aligned_outputs(g);
  p.bias_vec = g.bias != nullptr && !g.bias_bf16 && (reinterpret_cast<uintptr_t>(g.bias) & 15) == 0;
  // bulk tensor stores need what a tensor map needs: 16-byte aligned base, row pitch a multiple of 16 bytes
  p.tma_store = tma_store_on() && p.vec_ok && g.c != nullptr && (g.out_fp32 ? true : (g.ldc % 8 == 0));
  const int kind = epilogue_kind(p);
  CUtensorMap tm_a, tm_b, tm_c, tm_c2;
  memset(&tm_c, 0, sizeof(tm_c));
  memset(&tm_c2, 0, sizeof(tm_c2));
  int st;
  if (p.tma_store) {
    // boxes of 32 rows x 128 bytes: 64 bf16 or 32 fp32 columns; with a second output, and in the fp32 form, 32 rows x 64 bytes each
    if (g.c2) {
      st = make_map(&tm_c, g.c, g.n, g.m, g.ldc, 32, 32, false, true);
      if (st) return st;
      st = make_map(&tm_c2, g.c2, g.n, g.m, g.ldc, 32, 32, false, true);
    } else if (kind == kEpiF32) {
      st = make_map(&tm_c, g.c, g.n, (long long)g.m * (g.slice_k ? p.split : 1), g.ldc, 16, 32, true, true);
    } else {
      st = make_map(&tm_c, g.c, g.n, g.m, g.ldc, g.out_fp32 ? 32 : 64, 32, g.out_fp32 != 0);
    }
    if (st) return st;
  }
  const long long a_rows = (g.a_mn_major ? g.k : g.m) + (long long)g.seg_a, a_cols = g.a_mn_major ? g.m : g.k;
  const long long b_rows = (g.b_mn_major ? g.k : g.n) + (long long)g.seg_b, b_cols = g.b_mn_major ? g.n : g.k;
  st = g.a_mn_major ? make_map(&tm_a, g.a, a_cols, a_rows, g.lda, 64, BK) : make_map(&tm_a, g.a, a_cols, a_rows, g.lda, BK, 128);
  if (st) return st;
  st = g.b_mn_major ? make_map(&tm_b, g.b, b_cols, b_rows, g.ldb, 64, BK) : make_map(&tm_b, g.b, b_cols, b_rows, g.ldb, BK, BN / 2);
  if (st) return st;
  const int pairs = p.units < pairs_max ? p.units : pairs_max;
  p.step = pairs;
  p.step_sp = pairs / tiles;
  p.step_m = pairs % tiles / p.tiles_n;
  p.step_n = pairs % tiles % p.tiles_n;
  rb_launch_pdl(kernels[kind], dim3(2 * pairs), dim3(kThreads), kSmemBytes, stream, tm_a, tm_b, tm_c, tm_c2, p);
  return rb_check_launch("gemm_pair");
}

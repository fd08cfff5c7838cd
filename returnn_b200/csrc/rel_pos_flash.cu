// Relative-position self-attention for head dim 64, fused: scores, shifted position scores, mask, softmax, dropout and the product with the
// values in one kernel; in the backward pass the recomputed scores, dP, dS and the query gradients in another.
//
// Operands are the zero-padded [B, Lp, H*64] matrices of att_prepare (queries with either bias, keys, values) and the projected positions
// [R, H*64]: score(i, j) = scale * (qu_i . k_j + qv_i . p_{center + j - i}). For a tile of 128 queries from i0 and W keys from j0 the second
// term needs the W + 127 position rows from center + j0 - i0 - 127 on: one product [128, W + 128] against a window of the position matrix
// that TMA reads in place (rows outside it are zero). Row i of the result is needed from column 127 - i on: a thread owns a row, the 32 rows
// of a warp read a common window of tensor memory, and each lane shifts its registers by 31 - lane places in five conditional steps.
//
//   rel_fwd  one CTA per (batch entry, head, 128 queries), W = 128: two groups of 128 threads with 64 keys each, each with its own running
//            maximum, sum and accumulator, merged at the end (tensor memory: 128 scores + 256 positions + 2 x 64 outputs = all 512 columns)
//   rel_bwd  the same split, W = 64, two groups with 32 keys each: P and dS go to memory for the two products over queries (dV, dK), dQu
//            and dQv accumulate in tensor memory. dS shifted back fills the band that the position gradient is a product of: the 64 columns
//            of a row that a tile of keys fills are followed by those of the next tile, so a window of three blocks of 64 columns walks over
//            the band in a ring of shared memory, and with every tile its first block is complete. A complete block is stored once and
//            multiplied once (dQv). Adding all three blocks of every tile to a zeroed band, and multiplying them, took three times the bulk
//            traffic and twelve small products instead of four, and 58 us of fills (a pass at 36 x 333 frames, 8 heads: 403 -> 343 us). The margins of the band, and
//            the rows of tiles without a valid query, are zeros that this kernel writes while its first loads are under way.
// What went through memory before: scores and position band written and read in both passes, probabilities, dP.
//
// Both are bound by the row work (window reads, shifts, exponentials: issue slots of the eight row warps). Loads, products and bulk stores are issued by
// a ninth warp, which meets the rows at mbarriers only: with one of the row threads issuing, all 256 waited for it at block barriers, four times a
// tile. The outputs stay in tensor memory, where they are rescaled with the maximum of a row (see tmem_scale64). Tile t + 2 is loaded
// while the rows are at tile t: the windows of consecutive tiles share all but one block of 64 (forward: 128) positions, so that only that block is
// loaded anew, and a ring of five (three) blocks leaves the room for a third tile of what both products read (rel_bwd at 36 x 333 frames 104 -> 102 us,
// 20 x 500 frames with gradients 258 -> 252). Kernels within the
// backward pass of 6912 rows: rel_bwd 98.3 -> 87.3 us; passes alone, forward 36 x 333 frames, 8 heads 92.0 -> 85.9 us, with gradients 323 -> 307
// (products of dV, dK and positions included), 20 x 500 frames 305 -> 276, 300 x 40 frames 445 -> 407.
#include "flash.cuh"
#include "gemm.h"

using namespace rbf;

namespace {

constexpr int kThreads = 256;        // rows: two groups of 128
constexpr int kCta = kThreads + 32;  // and the warp that issues (see Pipe)

struct Rel {
  const int* lens;
  float* lse;      // [B*H, lp] log2 of the softmax denominator, maximum included
  uint32_t* keep;  // [B*H, lp, words] dropout: bit j of word w = key 32 w + j is kept
  const __nv_bfloat16* w;  // [B*H, lp, lp] (backward, saved form) probabilities
  __nv_bfloat16* p;        // [B*H, lp, lp] (backward) dropped probabilities (saved form: read)
  __nv_bfloat16 *dqu, *dqv, *band;  // (backward) where the zeros of the padding go
  __nv_bfloat16* out;               // (forward) packed rows, the sequences back to back
  const long long* seed;
  const long long* offset;
  int* status;
  int batch, heads, lp, tiles, words, center, band_off, band_w;
  int sparse;  // (backward) the padding is written only where the position gradient's product reads it
  float scale, p_drop;
};

template <uint32_t N>
__device__ __forceinline__ void mma_n(uint32_t d, const uint8_t* a, const uint8_t* b) {  // D[128, N] = A[128, 64] B[N, 64]^T, both K-major
  constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  const uint32_t da = desc_lo(smem_u32(a), 16), db = desc_lo(smem_u32(b), 16);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) umma_f16_warp(d, da + 2 * kk, db + 2 * kk, idesc, kk > 0 ? 1u : 0u);
}

// g[j] <- g[j + shift] for j < N, shift in [0, 31]; g holds N + 31 values
template <int N, int B>
__device__ __forceinline__ void shift_step(float* g, int shift) {
  const bool on = shift & B;
#pragma unroll
  for (int j = 0; j < N + B - 1; ++j) g[j] = on ? g[j + B] : g[j];
}
template <int N>
__device__ __forceinline__ void shift_down(float* g, int shift) {
  shift_step<N, 16>(g, shift);
  shift_step<N, 8>(g, shift);
  shift_step<N, 4>(g, shift);
  shift_step<N, 2>(g, shift);
  shift_step<N, 1>(g, shift);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

template <bool DROP>
__global__ void __launch_bounds__(kCta, 1)
rel_fwd_kernel(const __grid_constant__ CUtensorMap tm_qu, const __grid_constant__ CUtensorMap tm_qv, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_pos, const __grid_constant__ CUtensorMap tm_o,
               const Rel p) {
  rb_pdl_wait();
  rb_pdl_launch();
  const int z = blockIdx.x / p.tiles;
  const int q0 = (int)(blockIdx.x % p.tiles) * kRows;
  const int b = z / p.heads, h = z - b * p.heads;
  const int len = p.lens[b];
  if (q0 >= len) return;  // nobody reads the padding rows of the output
  extern __shared__ uint8_t smem_raw[];
  uint8_t* squ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sqv = squ + kBig;
  uint8_t* sk = sqv + kBig;        // [2][128 keys]
  uint8_t* sv = sk + 2 * kBig;     // [3][128 keys]
  uint8_t* spos = sv + 3 * kBig;   // [3][128 positions]: blocks of the windows, tile t's are t and t + 1
  uint8_t* sp = spos + 3 * kBig;   // [2 groups][128 queries][64 keys]
  const Pipe w = pipe_begin<512, 8>(sp + 2 * kBig);
  const Cta& c = w.c;
  const int tid = threadIdx.x, wg = tid >> 7, r = tid & 127, lane = tid & 31;
  const int n_tiles = (len + 127) / 128;
  const uint32_t t_s = c.tmem, t_g = c.tmem + 128, t_o = c.tmem + 384;
  if (tid >= kThreads) {
    auto load = [&](int t) {
      if (!elect_one()) return;
      const int s = t & 1;
      const int p0 = p.center - q0 - 127;  // first position of block 0
      mbar_expect_tx(&c.full[s], (t == 0 ? 6 : 3) * kBig);
      if (t == 0) {
        tma_load_3d(squ, &tm_qu, h * 64, q0, b, &c.full[0]);
        tma_load_3d(sqv, &tm_qv, h * 64, q0, b, &c.full[0]);
        tma_load_2d(spos, &tm_pos, h * 64, p0, &c.full[0]);
      }
      tma_load_3d(sk + s * kBig, &tm_k, h * 64, t * 128, b, &c.full[s]);
      tma_load_3d(sv + t % 3 * kBig, &tm_v, h * 64, t * 128, b, &c.full[s]);
      tma_load_2d(spos + (t + 1) % 3 * kBig, &tm_pos, h * 64, p0 + (t + 1) * 128, &c.full[s]);
    };
    load(0);
    if (n_tiles > 1) load(1);
    pipe_issue_ahead(w, n_tiles, p.status, load,
                     [&](int t) {
                       mma_n<128>(t_s, squ, sk + (t & 1) * kBig);
                       mma_n<128>(t_g, sqv, spos + t % 3 * kBig);
                       mma_n<128>(t_g + 128, sqv, spos + (t + 1) % 3 * kBig);
                     },
                     [&](int t) {
                       const uint8_t* v = sv + t % 3 * kBig;
                       mma64_warp<true>(t_o, sp, v, t > 0);
                       mma64_warp<true>(t_o + 64, sp + kBig, v + kSmall, t > 0);
                     },
                     [](int) {});
  } else {
    const int row = q0 + r;
    const uint32_t t_lane = (uint32_t)(r & ~31) << 16;
    const float cs = p.scale * kLog2e;
    const uint64_t sd = DROP ? (uint64_t)p.seed[0] : 0, off = DROP ? (uint64_t)p.offset[0] : 0;
    const uint32_t thresh = DROP ? (uint32_t)(p.p_drop * 4294967296.0) : 0u;
    const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      uint32_t bits[2] = {0u, 0u};
      if constexpr (DROP) {  // while the scores are multiplied (after the exponentials: 36 x 333 frames, 8 heads 110 us for 101, 300 x 40 186 for 162)
        const uint64_t base = off + ((uint64_t)z * p.lp + row) * p.lp + it * 128 + wg * 64;
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
          const uint64_t ctr = base + j;
          const uint4 x = philox4x32(make_uint2((uint32_t)sd, (uint32_t)(sd >> 32)), make_uint4((uint32_t)ctr, (uint32_t)(ctr >> 32), 0x52u, 0u));
          const uint32_t r4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (r4[e] >= thresh) bits[(j + e) >> 5] |= 1u << ((j + e) & 31);
        }
        if (row < len) *reinterpret_cast<uint2*>(p.keep + ((long long)z * p.lp + row) * p.words + it * 4 + wg * 2) = make_uint2(bits[0], bits[1]);
      }
      ok = pipe_wait(w, w.scores, it, p.status, 22);
      if (!ok) break;
      float s[96];
      uint32_t* raw = reinterpret_cast<uint32_t*>(s);
      // the position scores of this warp's rows: 95 columns from 127 - (its last row) + 64 * group on
      const uint32_t g0 = t_g + t_lane + (uint32_t)(96 - (r & ~31) + wg * 64);
      tmem_ld32(g0, raw);
      tmem_ld32(g0 + 32, raw + 32);
      tmem_ld32(g0 + 64, raw + 64);
      tmem_wait_ld();
      shift_down<64>(s, 31 - lane);
      const int left = len - (it * 128 + wg * 64);  // keys of this group's half that exist
      float mx = -INFINITY;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float a[32];
        tmem_ld32(t_s + t_lane + wg * 64 + half * 32, reinterpret_cast<uint32_t*>(a));
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int jj = half * 32 + j;
          s[jj] = jj < left ? (a[j] + s[jj]) * cs : -INFINITY;
          mx = fmaxf(mx, s[jj]);
        }
      }
      pipe_arrive(w.taken);
      const bool grow = mx > m;  // (also from -inf to anything)
      const float corr = grow ? ex2(m - mx) : 1.f;
      if (grow) m = mx;
      l *= corr;
      const float mu = m == -INFINITY ? 0.f : m;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        s[j] = ex2(s[j] - mu);
        sum += s[j];
      }
      l += sum;
      if constexpr (DROP) {
#pragma unroll
        for (int j = 0; j < 64; ++j) s[j] = bits[j >> 5] >> (j & 31) & 1u ? s[j] * keep_scale : 0.f;
      }
      if (it > 0) {
        ok = pipe_wait(w, w.out, it - 1, p.status, 24);  // P of the tile before has been read, its product is in the output
        if (!ok) break;
        if (__any_sync(0xffffffffu, grow)) tmem_scale64(t_o + t_lane + wg * 64, corr);
      }
      store_row64(sp + wg * kBig, r, s);
      fence_proxy_async_smem();
      pipe_arrive(w.put);
    }
    ok = ok && pipe_wait(w, w.out, n_tiles - 1, p.status, 29);
    rows_sync<kThreads>();
    if (ok && !*c.abort_flag) {
      int start = 0;  // first packed row of the sequence
      for (int i = lane; i < b; i += 32) start += p.lens[i];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) start += __shfl_xor_sync(0xffffffffu, start, o);
      float acc[64];
      tmem_ld64(t_o + t_lane + wg * 64, acc);
      // merge the two groups through shared memory (the position tiles are not needed any more)
      float* ex = reinterpret_cast<float*>(spos) + r * 67;
      if (wg == 1) {
#pragma unroll
        for (int j = 0; j < 64; ++j) ex[j] = acc[j];
        ex[64] = m;
        ex[65] = l;
      }
      rows_sync<kThreads>();
      if (wg == 0) {
        const float m1 = ex[64], mm = fmaxf(m, m1);  // (the first key is always there: m is finite for valid rows)
        const float e0 = ex2(m - mm), e1 = ex2(m1 - mm);
        l = l * e0 + ex[65] * e1;
        const float inv = 1.f / l;
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = row < len ? (acc[j] * e0 + ex[j] * e1) * inv : 0.f;
        store_row64_f32(squ, r, acc);  // (over both query tiles)
        if (row < len) {
          p.lse[(long long)z * p.lp + row] = mm + __log2f(l);
          __nv_bfloat16* out = p.out + ((long long)start + row) * (p.heads * 64) + h * 64;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            F8 x;
#pragma unroll
            for (int i = 0; i < 8; ++i) x.v[i] = acc[8 * j + i];
            store8(out, 8 * j, x, 1);
          }
        }
      }
      fence_proxy_async_smem();
      rows_sync<kThreads>();
      if (tid == 0) {
        tma_store_3d(&tm_o, h * 64, q0, b, squ);
        tma_store_3d(&tm_o, h * 64 + 32, q0, b, squ + kBig);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }
  cta_end<512>(c);
}

// SAVED: the probabilities (and, dropped, those of the value product) come from memory, as the forward pass of the encoder executor left them;
// else they are recomputed and the dropped ones written
template <bool DROP, bool SAVED>
__global__ void __launch_bounds__(kCta, 1)
rel_bwd_kernel(const __grid_constant__ CUtensorMap tm_qu, const __grid_constant__ CUtensorMap tm_qv, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_pos, const __grid_constant__ CUtensorMap tm_o,
               const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_dqu, const __grid_constant__ CUtensorMap tm_dqv,
               const __grid_constant__ CUtensorMap tm_band, const __grid_constant__ CUtensorMap tm_p, const __grid_constant__ CUtensorMap tm_ds,
               const Rel p) {
  rb_pdl_wait();
  rb_pdl_launch();
  const int z = blockIdx.x / p.tiles;
  const int q0 = (int)(blockIdx.x % p.tiles) * kRows;
  const int b = z / p.heads, h = z - b * p.heads;
  const int len = p.lens[b];
  const int tid = threadIdx.x, wg = tid >> 7, r = tid & 127, lane = tid & 31;
  const int n_tiles = (len + 63) / 64;
  const int band_row = (h * p.batch + b) * p.lp + q0;
  const int n_rows_band = min(kRows, p.lp - q0);
  const int x0 = p.center - q0 - 127 + p.band_off;  // first column of the band that this tile of queries fills (a multiple of 8, not negative)
  // zeros in the columns of the band outside [lo, hi), a warp to a row
  auto band_zeros = [&](int lo, int hi) {
    for (int i = tid >> 5; i < n_rows_band; i += kThreads / 32) {
      uint4* dst = reinterpret_cast<uint4*>(p.band + (long long)(band_row + i) * p.band_w);
      for (int x = lane; x < p.band_w / 8; x += 32)
        if (x * 8 < lo || x * 8 >= hi) dst[x] = make_uint4(0u, 0u, 0u, 0u);
    }
  };
  if (q0 >= len) {  // no valid query
    if (tid >= kThreads || p.sparse) return;
    band_zeros(0, 0);
    for (int i = tid; i < n_rows_band * 8; i += kThreads) {
      const long long at = ((long long)b * p.lp + q0 + (i >> 3)) * (p.heads * 64) + h * 64 + (i & 7) * 8;
      *reinterpret_cast<uint4*>(p.dqu + at) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(p.dqv + at) = make_uint4(0u, 0u, 0u, 0u);
    }
    return;
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t* squ = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sqv = squ + kBig;
  uint8_t* sdo = sqv + kBig;
  uint8_t* sk = sdo + kBig;          // [3][64 keys]
  uint8_t* sv = sk + 3 * kSmall;     // [2][64 keys]
  uint8_t* spos = sv + 2 * kSmall;   // [5][64 positions]: blocks of the windows, tile t's are t to t + 2
  uint8_t* sds = spos + 5 * kSmall;  // [128 queries][64 keys]
  uint8_t* sdg = sds + kBig;         // ring of [4][128 queries][64 positions]; first the tile of O in 32 bits
  uint8_t* sp = sdg + 4 * kBig;      // [128 queries][64 keys] dropped probabilities
  const Pipe w = pipe_begin<512, 8, 2>(sp + kBig);  // `out`: the products, and the bulk stores have read their tiles
  const Cta& c = w.c;
  const int row = q0 + r;
  const int len64 = n_tiles * 64;
  const uint32_t t_lane = (uint32_t)(r & ~31) << 16;
  const uint32_t t_s = c.tmem, t_dp = c.tmem + 64, t_g = c.tmem + 128, t_dqu = c.tmem + 320, t_dqv = c.tmem + 384;
  if (tid >= kThreads) {
    auto load = [&](int t) {
      if (!elect_one()) return;
      const int s = t & 1;
      const int p0 = p.center - q0 - 127;  // first position of block 0
      mbar_expect_tx(&c.full[s], 3 * kSmall + (t == 0 ? 3 * kBig + 2 * kSmall : 0));
      if (t == 0) {
        tma_load_3d(squ, &tm_qu, h * 64, q0, b, &c.full[0]);
        tma_load_3d(sqv, &tm_qv, h * 64, q0, b, &c.full[0]);
        tma_load_3d(sdo, &tm_do, h * 64, q0, b, &c.full[0]);
        tma_load_2d(spos, &tm_pos, h * 64, p0, &c.full[0]);
        tma_load_2d(spos + kSmall, &tm_pos, h * 64, p0 + 64, &c.full[0]);
      }
      tma_load_3d(sk + t % 3 * kSmall, &tm_k, h * 64, t * 64, b, &c.full[s]);
      tma_load_3d(sv + s * kSmall, &tm_v, h * 64, t * 64, b, &c.full[s]);
      tma_load_2d(spos + (t + 2) % 5 * kSmall, &tm_pos, h * 64, p0 + (t + 2) * 64, &c.full[s]);
    };
    load(0);
    if (elect_one()) {
      mbar_expect_tx(c.extra, 2 * kBig);
      tma_load_3d(sdg, &tm_o, h * 64, q0, b, c.extra);
      tma_load_3d(sdg + kBig, &tm_o, h * 64 + 32, q0, b, c.extra);
    }
    if (n_tiles > 1) load(1);
    auto blocks_done = [&](int t) { return t + 1 < n_tiles ? 1 : 3; };  // blocks of the window that are complete
    pipe_issue_ahead(w, n_tiles, p.status, load,
               [&](int t) {
                 mma64_warp<false>(t_dp, sdo, sv + (t & 1) * kSmall, false);
                 if (SAVED) return;
                 mma64_warp<false>(t_s, squ, sk + t % 3 * kSmall, false);
                 for (int q = 0; q < 3; ++q) mma64_warp<false>(t_g + 64 * q, sqv, spos + (t + q) % 5 * kSmall, false);
               },
               [&](int t) {
                 mma64_warp<true>(t_dqu, sds, sk + t % 3 * kSmall, t > 0);
                 for (int q = 0; q < blocks_done(t); ++q) mma64_warp<true>(t_dqv, sdg + ((t + q) & 3) * kBig, spos + (t + q) % 5 * kSmall, t > 0 || q > 0);
               },
               [&](int t) {
                 if (!elect_one()) return;
                 for (int q = 0; q < blocks_done(t); ++q)
#pragma unroll
                   for (int half = 0; half < 2; ++half)
                     if (half * 64 < n_rows_band)
                       tma_store_2d(&tm_band, x0 + 64 * (t + q), band_row + half * 64, sdg + ((t + q) & 3) * kBig + half * kSmall);
                 // P and dS: the products over queries run in blocks of 64 rows, zeros up to there
#pragma unroll
                 for (int half = 0; half < 2; ++half) {
                   if (q0 + half * 64 >= len64) break;
                   tma_store_2d(&tm_ds, t * 64, z * p.lp + q0 + half * 64, sds + half * kSmall);
                   if (!SAVED) tma_store_2d(&tm_p, t * 64, z * p.lp + q0 + half * 64, sp + half * kSmall);
                 }
                 tma_store_commit();
                 tma_store_wait_read();
                 mbar_arrive_local(w.out);
               });
  } else {
    if (p.sparse) {  // up to the next tiles of 128 columns of the product over the band, half a warp to each side
      const int lo = x0 & ~127, hi = x0 + 64 * (n_tiles + 2), to = min((hi + 127) & ~127, p.band_w);
      const int x = lane < 16 ? lo + lane * 8 : hi + (lane - 16) * 8;
      if (x < (lane < 16 ? x0 : to))
        for (int i = tid >> 5; i < n_rows_band; i += kThreads / 32)
          *reinterpret_cast<uint4*>(p.band + (long long)(band_row + i) * p.band_w + x) = make_uint4(0u, 0u, 0u, 0u);
    } else {
      band_zeros(x0, x0 + 64 * (n_tiles + 2));
    }
    float lse = INFINITY, delta = 0.f;
    bool ok = pipe_wait(w, &c.full[0], 0, p.status, 26) && pipe_wait(w, c.extra, 0, p.status, 26);
    if (ok) {
      delta = dot_row64(sdg, sdo, r);
      if (!SAVED && row < len) lse = p.lse[(long long)z * p.lp + row];
    }
    rows_sync<kThreads>();
    for (int i = tid; i < 3 * kBig / 16; i += kThreads) reinterpret_cast<uint4*>(sdg)[i] = make_uint4(0u, 0u, 0u, 0u);
    rows_sync<kThreads>();
    const float cs = p.scale * kLog2e;
    const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
    uint4 wv[4], wd[4];
    auto fetch_saved = [&](int t) {
      const long long at = ((long long)z * p.lp + row) * p.lp + t * 64 + wg * 32;  // this thread's 32 scores
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        wv[q] = *reinterpret_cast<const uint4*>(p.w + at + 8 * q);
        if (DROP) wd[q] = *reinterpret_cast<const uint4*>(p.p + at + 8 * q);
      }
    };
    if (SAVED && row < len) fetch_saved(0);
    for (int it = 0; it < n_tiles && ok; ++it) {
      uint32_t bits = 0u;
      if (DROP && !SAVED && row < len) bits = p.keep[((long long)z * p.lp + row) * p.words + it * 2 + wg];
      ok = pipe_wait(w, w.scores, it, p.status, 27);
      if (!ok) break;
      float s[64], a[32], dp[32];
      if (!SAVED) {
        const uint32_t g0 = t_g + t_lane + (uint32_t)(96 - (r & ~31) + wg * 32);
        tmem_ld32(g0, reinterpret_cast<uint32_t*>(s));
        tmem_ld32(g0 + 32, reinterpret_cast<uint32_t*>(s) + 32);
        tmem_ld32(t_s + t_lane + wg * 32, reinterpret_cast<uint32_t*>(a));
      }
      tmem_ld32(t_dp + t_lane + wg * 32, reinterpret_cast<uint32_t*>(dp));
      tmem_wait_ld();
      pipe_arrive(w.taken);
      if (!SAVED) shift_down<32>(s, 31 - lane);
      const int left = row < len ? len - (it * 64 + wg * 32) : 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const bool vis = j < left;
        float d = dp[j];
        if (SAVED) {
          const uint32_t word = reinterpret_cast<const uint32_t*>(wv)[j >> 1];
          if (DROP) {  // a dropped probability is zero; where the probability itself is, its gradient is too
            const uint32_t kept = reinterpret_cast<const uint32_t*>(wd)[j >> 1];
            d = ((j & 1 ? kept >> 16 : kept) & 0x7fffu) ? d * keep_scale : 0.f;
          }
          a[j] = vis ? __uint_as_float(j & 1 ? word & 0xffff0000u : word << 16) * (d - delta) : 0.f;
        } else {
          const float pr = vis ? ex2(fmaf(a[j] + s[j], cs, -lse)) : 0.f;
          float pd = pr;
          if (DROP) {
            const bool k = (bits >> j) & 1u;
            d = k ? d * keep_scale : 0.f;
            pd = k ? pr * keep_scale : 0.f;
          }
          a[j] = vis ? pr * (d - delta) : 0.f;
          s[j] = pd;
        }
      }
      if (SAVED && row < len && it + 1 < n_tiles) fetch_saved(it + 1);  // (on their way until the next tile's scores are there)
      if (it > 0) {
        ok = pipe_wait(w, w.out, it - 1, p.status, 28);  // what the tile before has put has been read
        if (!ok) break;
      }
      uint4 pk[4], dk[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (!SAVED) pk[q] = make_uint4(pack2(s[8 * q], s[8 * q + 1]), pack2(s[8 * q + 2], s[8 * q + 3]), pack2(s[8 * q + 4], s[8 * q + 5]), pack2(s[8 * q + 6], s[8 * q + 7]));
        dk[q] = make_uint4(pack2(a[8 * q], a[8 * q + 1]), pack2(a[8 * q + 2], a[8 * q + 3]), pack2(a[8 * q + 4], a[8 * q + 5]), pack2(a[8 * q + 6], a[8 * q + 7]));
        const int slot = r * 128 + (((wg * 4 + q) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(sds + slot) = dk[q];
        if (!SAVED) *reinterpret_cast<uint4*>(sp + slot) = pk[q];
      }
      // shifted back: key j of the tile lies at column 127 - r + j of the window. 32 columns from c0 on as pairs; where c0 is odd, the first and
      // the last by themselves
      {
        const uint32_t* d = reinterpret_cast<const uint32_t*>(dk);
        const int c0 = 127 - r + wg * 32, odd = c0 & 1;
        uint8_t* base = sdg + r * 128;
        auto at_col = [&](int col) { return base + ((it + (col >> 6)) & 3) * kBig + ((((col & 63) >> 3) ^ (r & 7)) << 4) + (col & 7) * 2; };
#pragma unroll
        for (int j = 0; j < 15; ++j) *reinterpret_cast<uint32_t*>(at_col(c0 + odd + 2 * j)) = odd ? __funnelshift_r(d[j], d[j + 1], 16) : d[j];
        if (odd) {
          *reinterpret_cast<unsigned short*>(at_col(c0)) = (unsigned short)(d[0] & 0xffffu);
          *reinterpret_cast<unsigned short*>(at_col(c0 + 31)) = (unsigned short)(d[15] >> 16);
        } else {
          *reinterpret_cast<uint32_t*>(at_col(c0 + 30)) = d[15];
        }
      }
      // the block that joins the window with the next tile; the last two are filled in part
      if (it + 3 >= n_tiles && it + 3 <= n_tiles + 1) {
#pragma unroll
        for (int q = 0; q < kBig / 16 / kThreads; ++q) reinterpret_cast<uint4*>(sdg + ((it + 3) & 3) * kBig)[q * kThreads + tid] = make_uint4(0u, 0u, 0u, 0u);
      }
      fence_proxy_async_smem();
      pipe_arrive(w.put);
    }
    ok = ok && pipe_wait(w, w.out, n_tiles - 1, p.status, 29);
    rows_sync<kThreads>();
    if (ok && !*c.abort_flag) {
      float s[64];
      tmem_ld64((wg ? t_dqv : t_dqu) + t_lane, s);
#pragma unroll
      for (int j = 0; j < 64; ++j) s[j] *= p.scale;
      store_row64(wg ? sqv : squ, r, s);
      fence_proxy_async_smem();
      rows_sync<kThreads>();
      if (tid == 0) {
        tma_store_3d(&tm_dqu, h * 64, q0, b, squ);
        tma_store_3d(&tm_dqv, h * 64, q0, b, sqv);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }
  cta_end<512>(c);
}

// sum of the slices of a split product in their order, fp32 [slices][n] -> bf16 or fp32 [n], n a multiple of 4
__device__ __forceinline__ void store4(uint2* y, const float4& s) { *y = make_uint2(pack2(s.x, s.y), pack2(s.z, s.w)); }
__device__ __forceinline__ void store4(float4* y, const float4& s) { *y = s; }

template <typename Out>
__global__ void __launch_bounds__(256)
sum_slices_kernel(const float4* __restrict__ x, Out* __restrict__ y, int slices, long long n4) {
  rb_pdl_wait();
  rb_pdl_launch();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  float4 s = x[i];
#pragma unroll 8  // (loads ahead of the sums, which keep their order)
  for (int k = 1; k < slices; ++k) {
    const float4 v = x[k * n4 + i];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  store4(y + i, s);
}

template <typename Out>
int sum_slices(const float* x, void* y, int slices, long long n, cudaStream_t stream) {
  if (n <= 0 || slices <= 0) return RB_OK;
  if (n % 4) {
    rb_set_error("sum_slices: n=%lld must be a multiple of 4", n);
    return RB_ERR_ARG;
  }
  rb_launch_pdl(sum_slices_kernel<Out>, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, stream, (const float4*)x, (Out*)y, slices, n / 4);
  return rb_check_launch("sum_slices");
}

constexpr int kFwdSmem = 12 * kBig + 64 + 1024;
constexpr int kBwdSmem = 9 * kBig + 10 * kSmall + 64 + 1024;
static_assert(kFwdSmem <= 227 * 1024 && kBwdSmem <= 227 * 1024, "shared memory");

// positions [r_rows, HD]: boxes of `box` rows, 64 columns
int map_pos(CUtensorMap* m, const void* pos, int r_rows, int hd, int box) { return make_map(m, pos, hd, r_rows, hd, 64, box); }

int failed(const char* what, cudaError_t e) {
  rb_set_error("%s: %s", what, cudaGetErrorString(e));
  return RB_ERR_LAUNCH;
}

}  // namespace

// qu, qv, k, v: bf16 [B, Lp, H*64], rows past a sequence's length zero; pos [R, H*64]; keep words per row: 4 * ceil(Lp / 128); lse [B*H, Lp];
// o: fp32 [B, Lp, H*64], rows past a sequence's length unspecified. In 32 bits because the row sums dO . O of the backward pass are taken from
// it: the rounding of 16-bit values would be the same for a whole row of dS, which is far more than dS where the values share an offset
// (300 frames, values 24 + n(0, 1), keys 4 + n(0, 1): error of dQ 2.40, from 32 bits 0.12, as from the sums over P * dP; a training pass 398 -> 401 us at 36 x 333 x 8 heads)
// o [B, Lp, H*64] (fp32): valid rows written, and the last tile's zeros; out [N, H*64] (bf16, 16-byte aligned): the same rows, packed
RB_EXPORT int rb200_rel_flash_fwd(const void* qu, const void* qv, const void* k, const void* v, const void* pos, float* o, void* out, float* lse, void* keep,
                                  const int* lens, int batch, int heads, int lp, int r_rows, int center, float scale, float p_drop,
                                  const long long* seed, const long long* offset, int* status, cudaStream_t stream) {
  if (batch <= 0 || heads <= 0 || lp <= 0) return RB_OK;
  const int hd = heads * 64;
  Rel p = {};
  p.out = (__nv_bfloat16*)out;
  p.lens = lens; p.lse = lse; p.keep = (uint32_t*)keep; p.seed = seed; p.offset = offset; p.status = status;
  p.batch = batch; p.heads = heads; p.lp = lp; p.center = center; p.scale = scale; p.p_drop = p_drop;
  p.tiles = (lp + kRows - 1) / kRows;
  p.words = 4 * ((lp + 127) / 128);
  CUtensorMap a, b, c, d, e, f;
  const long long bp = (long long)lp * hd;
  int st = make_map_3d(&a, qu, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&b, qv, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&c, k, hd, lp, batch, hd, bp, 128);
  if (!st) st = make_map_3d(&d, v, hd, lp, batch, hd, bp, 128);
  if (!st) st = map_pos(&e, pos, r_rows, hd, 128);
  if (!st) st = make_map_3d(&f, o, hd, lp, batch, hd, bp, kRows, true);
  if (st) return st;
  auto kernel = p_drop > 0.f ? rel_fwd_kernel<true> : rel_fwd_kernel<false>;
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  if (err != cudaSuccess) return failed("rel_flash_fwd", err);
  rb_launch_pdl(kernel, dim3((unsigned)(p.tiles * batch * heads)), dim3(kCta), kFwdSmem, stream, a, b, c, d, e, f, p);
  return rb_check_launch("rel_flash_fwd");
}

// Column of the band that position row 0 has, such that every tile's first column is a multiple of 8 and none is negative; *width: columns
// of the band. (Lp a multiple of 64.)
RB_EXPORT int rb200_rel_flash_band(int lp, int center, int* off, int* width) {
  const int tiles = (lp + kRows - 1) / kRows;
  int o = (tiles - 1) * kRows + 127 - center;
  if (o < 0) o = 0;
  while ((center - 127 + o) & 7) ++o;
  *off = o;
  *width = (center + lp - 64 - 127 + o + 192 + 63) / 64 * 64;
  return RB_OK;
}

// dqu, dqv [B, Lp, H*64] and band [H, B, Lp, band_width]: written whole, zeros in the padding; pw, ds [B*H, Lp, Lp]: written for the first
// 64 * ceil(len / 64) rows and columns of each sequence. With saved probabilities `w` (else null; lse and keep are not read then) pw is read:
// the dropped probabilities, or anything without dropout
static int rel_flash_bwd(int sparse, const void* qu, const void* qv, const void* k, const void* v, const void* pos, const float* o, const void* d_o,
                                  void* dqu, void* dqv, const void* w, void* pw, void* ds, void* band, float* lse, void* keep, const int* lens, int batch,
                                  int heads, int lp, int r_rows, int center, float scale, float p_drop, int* status, cudaStream_t stream) {
  if (batch <= 0 || heads <= 0 || lp <= 0) return RB_OK;
  const int hd = heads * 64;
  Rel p = {};
  p.sparse = sparse;
  p.lens = lens; p.lse = lse; p.keep = (uint32_t*)keep; p.status = status; p.w = (const __nv_bfloat16*)w; p.p = (__nv_bfloat16*)pw;
  p.dqu = (__nv_bfloat16*)dqu; p.dqv = (__nv_bfloat16*)dqv; p.band = (__nv_bfloat16*)band;
  p.batch = batch; p.heads = heads; p.lp = lp; p.center = center; p.scale = scale; p.p_drop = p_drop;
  p.tiles = (lp + kRows - 1) / kRows;
  p.words = 4 * ((lp + 127) / 128);
  rb200_rel_flash_band(lp, center, &p.band_off, &p.band_w);
  const int width = p.band_w;
  CUtensorMap a, b, c, d, e, f, g, h, i, j, map_p, map_ds;
  const long long bp = (long long)lp * hd;
  int st = make_map_3d(&a, qu, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&b, qv, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&c, k, hd, lp, batch, hd, bp, 64);
  if (!st) st = make_map_3d(&d, v, hd, lp, batch, hd, bp, 64);
  if (!st) st = map_pos(&e, pos, r_rows, hd, 64);
  if (!st) st = make_map_3d(&f, o, hd, lp, batch, hd, bp, kRows, true);
  if (!st) st = make_map_3d(&g, d_o, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&h, dqu, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map_3d(&i, dqv, hd, lp, batch, hd, bp, kRows);
  if (!st) st = make_map(&j, band, width, (long long)heads * batch * lp, width, 64, 64);
  if (!st) st = make_map(&map_p, pw, lp, (long long)batch * heads * lp, lp, 64, 64);
  if (!st) st = make_map(&map_ds, ds, lp, (long long)batch * heads * lp, lp, 64, 64);
  if (st) return st;
  auto kernel = p_drop > 0.f ? (w ? rel_bwd_kernel<true, true> : rel_bwd_kernel<true, false>) : (w ? rel_bwd_kernel<false, true> : rel_bwd_kernel<false, false>);
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem);
  if (err != cudaSuccess) return failed("rel_flash_bwd", err);
  rb_launch_pdl(kernel, dim3((unsigned)(p.tiles * batch * heads)), dim3(kCta), kBwdSmem, stream, a, b, c, d, e, f, g, h, i, j, map_p, map_ds, p);
  return rb_check_launch("rel_flash_bwd");
}

RB_EXPORT int rb200_rel_flash_bwd(const void* qu, const void* qv, const void* k, const void* v, const void* pos, const float* o, const void* d_o,
                                  void* dqu, void* dqv, const void* w, void* pw, void* ds, void* band, float* lse, void* keep, const int* lens, int batch,
                                  int heads, int lp, int r_rows, int center, float scale, float p_drop, int* status, cudaStream_t stream) {
  return rel_flash_bwd(0, qu, qv, k, v, pos, o, d_o, dqu, dqv, w, pw, ds, band, lse, keep, lens, batch, heads, lp, r_rows, center, scale, p_drop, status, stream);
}

// The same, of the padding only what rel_flash_dpos reads of it: the rest of the band and the rows of dqu and dqv in tiles without a valid query are
// left as they are (zeros there were 100 of 270 MB at 36 x 334 frames of which 57 % are valid, 8 heads; kernel with saved probabilities
// 87 -> 68 us, with the probabilities of a tile fetched during the one before 64; with recomputed ones at 36 x 333 frames 102 -> 90)
RB_EXPORT int rb200_rel_flash_bwd_sparse(const void* qu, const void* qv, const void* k, const void* v, const void* pos, const float* o, const void* d_o,
                                  void* dqu, void* dqv, const void* w, void* pw, void* ds, void* band, float* lse, void* keep, const int* lens, int batch,
                                  int heads, int lp, int r_rows, int center, float scale, float p_drop, int* status, cudaStream_t stream) {
  return rel_flash_bwd(1, qu, qv, k, v, pos, o, d_o, dqu, dqv, w, pw, ds, band, lse, keep, lens, batch, heads, lp, r_rows, center, scale, p_drop, status, stream);
}

// slices that the product of the position gradient, [band_width, rows] x [rows, 64] per head, is cut into: it has few output tiles and
// B * Lp rows to sum over (48 tiles of 13824 rows for a full Conformer batch: a third of the SMs for 90 us); two waves of CTAs, equal slices
// of whole 64-row blocks
RB_EXPORT int rb200_rel_flash_slices(long long rows, int width, int heads) {
  const long long blocks = rows / 64, tiles = (long long)((width + 127) / 128) * heads;
  long long n = 296 / (tiles > 0 ? tiles : 1);
  if (n > blocks / 4) n = blocks / 4;
  while (n > 1 && blocks % n) --n;
  return n > 1 ? (int)n : 1;
}

// position gradient: part [slices][band_width][heads * 64] (fp32; one slice: bf16) = scale * band^T qv over the rows of the slice. Only the blocks
// of the band that rel_flash_bwd filled for the tile's positions are read: about a third of 36 x 333 frames (whole: 26 us of products, 170 MB)
RB_EXPORT int rb200_rel_flash_dpos(const void* band, const void* qv, void* part, const int* lens, int batch, int heads, int lp, int center, float scale,
                                   int slices, int* status, cudaStream_t stream) {
  if (batch <= 0 || heads <= 0 || lp <= 0) return RB_OK;
  const int hd = heads * 64;
  const long long rows = (long long)batch * lp;
  if (slices <= 0 || rows % slices || rows / slices % 64 || lp % 64 || rows * heads > 0x7fffffffLL) {
    rb_set_error("rel_flash_dpos: %lld rows in %d slices", rows, slices);
    return RB_ERR_ARG;
  }
  int off = 0, width = 0;
  rb200_rel_flash_band(lp, center, &off, &width);
  RbGemm g;
  g.a = band; g.b = qv; g.c = part; g.m = width; g.n = 64; g.k = (int)(rows / slices); g.lda = width; g.ldb = hd; g.ldc = hd;
  g.a_mn_major = 1; g.b_mn_major = 1; g.alpha = scale; g.out_fp32 = slices > 1; g.status = status;
  g.batch = slices * heads; g.heads = heads;
  g.a_rb = g.k; g.a_rh = rows; g.b_rb = g.k; g.b_ch = 64; g.c_sb = (long long)width * hd; g.c_sh = 64;
  g.a_rows = rows * heads; g.a_cols = width; g.b_rows = rows; g.b_cols = hd;
  g.win = 2; g.win_center = center + off; g.win_lp = lp; g.win_lens = lens;
  return rb_gemm(g, stream);
}

RB_EXPORT int rb200_sum_slices(const float* x, void* y, int slices, long long n, cudaStream_t stream) { return sum_slices<uint2>(x, y, slices, n, stream); }
RB_EXPORT int rb200_sum_slices_f32(const float* x, float* y, int slices, long long n, cudaStream_t stream) {
  return sum_slices<float4>(x, y, slices, n, stream);
}

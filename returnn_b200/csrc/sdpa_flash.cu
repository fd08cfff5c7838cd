// Scaled-dot-product attention in one kernel per pass for head dim 64: scores, mask, softmax, dropout and the product with the values
// stay on the SM, so no [Tq, Tk] matrix is written to memory.
//
//   flash_fwd     one CTA per (batch entry, head, 128 queries): a loop over tiles of 64 keys, online softmax
//   flash_bwd_q   the same split: recomputes the scores from the saved log-sum, dS = P * (dP - delta), dQ = scale * dS K
//   flash_bwd_kv  one CTA per (batch entry, head, 128 keys): a loop over tiles of 64 queries, transposed scores, dK and dV
//   flash_bwd_small  up to 128 queries and keys: both in one
//
// A CTA has 128 row threads = the 128 lanes of tensor memory: a thread owns one row of the score tile (a query; in flash_bwd_kv a key) and
// needs no exchange with others for maximum and sum. A warp of its own issues the TMA loads (two stages) and the tcgen05.mma and meets the rows
// at mbarriers only (see Pipe in flash.cuh). The chain product -> softmax -> product of one CTA is serial; three (backward: two) CTAs per SM fill
// each other's gaps. That is why the tiles are
// 64 wide: 128 TMEM columns and 67 KB of shared memory per CTA (backward 256 columns and 99 / 102 KB). The two-pass backward (dQ apart from
// dK / dV) repeats two of five products, which cost little here, and needs neither atomics nor an fp32 copy of dQ.
// The kernels are bound by the row work of a tile (about 1450 to 1750 cycles for 64 columns: issue slots and exponentials; two threads to a row
// gain nothing) and the length of the chain. 8 x 1000 causal, 8 heads, within a pass: 23 + 37 + 48 us with one of the row threads issuing and block
// barriers, 20 + 32 + 41 with the issuing warp. The forward kernel scales its output in tensor memory, see tmem_scale64: in a row of calls 30.6 us (with
// the output in registers 37.7). With dropout its decisions are drawn while the scores are multiplied, before those take up the registers: 61 us (after the
// exponentials, with spills: 90).
//
// Visible keys, the dropout rate and the layouts are those of sdpa.cu. The dropout decisions of the forward pass are kept as one bit per
// score. They come from a stream of the generator of their own (tag 0x53; sdpa.cu and attention.cu draw from 0x51, rel_pos_flash.cu from
// 0x52): the counter here steps in scores, theirs in groups of four, so that on one tag a later site would draw these words again.
#include "flash.cuh"

using namespace rbf;

namespace {

constexpr int kThreads = 128;

struct Flash {
  const int* k_lens;
  float* lse;    // [B*H, tq] log2 of the softmax denominator, maximum included; +inf: no visible key
  float* delta;  // [B*H, tq] sum_d dO * O
  uint32_t* keep;  // [B*H, tq, words] dropout: bit j of word w = key 32 w + j is kept
  const long long* seed;
  const long long* offset;
  int* status;
  int heads, bh, tq, tk, causal, shift, tiles, hq, hk, hv, hdo, words, tqp, tkp;
  int save;  // (forward) the output is kept in 32 bits for the backward pass
  float scale, p_drop;
};

__device__ __forceinline__ int visible(const Flash& p, int i, int klen) {
  int n = klen;
  if (p.causal) n = min(n, i + p.shift + 1);
  return max(n, 0);
}

constexpr int kCta = kThreads + 32;  // and the warp that issues (see Pipe)

template <bool DROP>
__global__ void __launch_bounds__(kCta, 3)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const __grid_constant__ CUtensorMap tm_o, const __grid_constant__ CUtensorMap tm_o32, const Flash p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sk = sq + kBig;
  uint8_t* sv = sk + 2 * kSmall;
  uint8_t* sp = sv + 2 * kSmall;
  const Pipe w = pipe_begin<128, 4>(sp + kBig);
  const Cta& c = w.c;
  rb_pdl_wait();
  rb_pdl_launch();
  const int tid = threadIdx.x;
  // the tiles of all heads side by side, causal the ones with the most keys first: the last wave of CTAs is then made of the short ones
  const int z = blockIdx.x % p.bh;
  const int q0 = (p.tiles - 1 - (int)(blockIdx.x / p.bh)) * kRows;
  const int b = z / p.heads, h = z - b * p.heads;
  const int klen = p.k_lens ? min(p.k_lens[b], p.tk) : p.tk;
  const int n_tiles = (visible(p, min(q0 + kRows, p.tq) - 1, klen) + kTile - 1) / kTile;
  const uint32_t t_s = c.tmem, t_o = c.tmem + 64;
  if (tid >= kThreads) {
    auto load = [&](int t) {
      if (!elect_one()) return;
      const int st = t & 1;
      mbar_expect_tx(&c.full[st], 2 * kSmall + (t == 0 ? kBig : 0));
      if (t == 0) tma_load_3d(sq, &tm_q, h * p.hq, q0, b, &c.full[0]);
      tma_load_3d(sk + st * kSmall, &tm_k, h * p.hk, t * kTile, b, &c.full[st]);
      tma_load_3d(sv + st * kSmall, &tm_v, h * p.hv, t * kTile, b, &c.full[st]);
    };
    if (n_tiles > 0) load(0);
    if (n_tiles > 1) load(1);
    if (n_tiles > 0)
      pipe_issue(w, n_tiles, p.status, load, [&](int t) { mma64_warp<false>(t_s, sq, sk + (t & 1) * kSmall, false); },
                 [&](int t) { mma64_warp<true>(t_o, sp, sv + (t & 1) * kSmall, t > 0); }, [](int) {});
  } else {
    const int row = q0 + tid;
    const int n = row < p.tq ? visible(p, row, klen) : 0;
    const uint32_t t_row = c.tmem + ((uint32_t)(tid & ~31) << 16);
    const float cs = p.scale * kLog2e;
    const uint64_t sd = DROP ? (uint64_t)p.seed[0] : 0, off = DROP ? (uint64_t)p.offset[0] : 0;
    const uint32_t thresh = DROP ? (uint32_t)(p.p_drop * 4294967296.0) : 0u;
    const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
    float m = -INFINITY, l = 0.f;
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      uint32_t bits[2] = {0u, 0u};
      if constexpr (DROP) {  // while the scores are multiplied, and before they take up the registers
        const uint64_t base = off + ((uint64_t)z * p.tqp + row) * p.tkp + it * kTile;
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
          const uint64_t ctr = base + j;
          const uint4 r = philox4x32(make_uint2((uint32_t)sd, (uint32_t)(sd >> 32)), make_uint4((uint32_t)ctr, (uint32_t)(ctr >> 32), 0x53u, 0u));
          const uint32_t x[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (x[e] >= thresh) bits[(j + e) >> 5] |= 1u << ((j + e) & 31);
        }
        if (row < p.tq) *reinterpret_cast<uint2*>(p.keep + ((long long)z * p.tq + row) * p.words + it * 2) = make_uint2(bits[0], bits[1]);
      }
      ok = pipe_wait(w, w.scores, it, p.status, 6);
      if (!ok) break;
      float s[64];
      tmem_ld64(t_row, s);
      pipe_arrive(w.taken);
      const int left = n - it * kTile;  // visible keys of this row in this tile
      float mx = -INFINITY;
      if (__all_sync(0xffffffffu, left >= kTile)) {
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          s[j] *= cs;
          mx = fmaxf(mx, s[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          s[j] = j < left ? s[j] * cs : -INFINITY;
          mx = fmaxf(mx, s[j]);
        }
      }
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
        ok = pipe_wait(w, w.out, it - 1, p.status, 7);  // P of the tile before has been read, its product is in the output
        if (!ok) break;
        if (__any_sync(0xffffffffu, grow)) tmem_scale64(t_row + 64, corr);
      }
      store_row64(sp, tid, s);
      fence_proxy_async_smem();
      pipe_arrive(w.put);
    }
    if (ok && n_tiles > 0) ok = pipe_wait(w, w.out, n_tiles - 1, p.status, 8);
    if (ok) {
      float s[64];
      if (n_tiles > 0) tmem_ld64(t_row + 64, s);
      const float inv = n > 0 ? 1.f / l : 0.f;
#pragma unroll
      for (int j = 0; j < 64; ++j) s[j] = n > 0 ? s[j] * inv : 0.f;
      store_row64(sq, tid, s);
      if (p.save) store_row64_f32(sk, tid, s);  // the tiles of keys and values are not needed any more
      if (row < p.tq) p.lse[(long long)z * p.tq + row] = n > 0 ? m + __log2f(l) : INFINITY;
      fence_proxy_async_smem();
    }
    rows_sync<kThreads>();
    if (tid == 0 && ok && !*c.abort_flag) {
      tma_store_3d(&tm_o, h * kTile, q0, b, sq);
      if (p.save) {
        tma_store_3d(&tm_o32, h * kTile, q0, b, sk);
        tma_store_3d(&tm_o32, h * kTile + 32, q0, b, sk + kBig);
      }
      tma_store_commit();
      tma_store_wait_read();  // (the writes complete like any other store of the grid)
    }
  }
  cta_end<128>(c);
}

template <bool DROP>
__global__ void __launch_bounds__(kCta, 2)
flash_bwd_q_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const __grid_constant__ CUtensorMap tm_o32, const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_dq,
                   const Flash p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sdo = sq + kBig;
  uint8_t* sk = sdo + kBig;
  uint8_t* sv = sk + 2 * kSmall;
  uint8_t* sds = sv + 2 * kSmall;  // first, with the kBig bytes behind it, the tile of O in 32 bits
  const Pipe w = pipe_begin<256, 4>(sds + 2 * kBig);
  const Cta& c = w.c;
  rb_pdl_wait();
  rb_pdl_launch();
  const int tid = threadIdx.x;
  const int z = blockIdx.x % p.bh;
  const int q0 = (p.tiles - 1 - (int)(blockIdx.x / p.bh)) * kRows;
  const int b = z / p.heads, h = z - b * p.heads;
  const int klen = p.k_lens ? min(p.k_lens[b], p.tk) : p.tk;
  const int n_tiles = (visible(p, min(q0 + kRows, p.tq) - 1, klen) + kTile - 1) / kTile;
  const uint32_t t_s = c.tmem, t_dp = c.tmem + 64, t_dq = c.tmem + 128;
  if (tid >= kThreads) {
    auto load = [&](int t) {
      if (!elect_one()) return;
      const int st = t & 1;
      mbar_expect_tx(&c.full[st], 2 * kSmall + (t == 0 ? 2 * kBig : 0));
      if (t == 0) {
        tma_load_3d(sq, &tm_q, h * p.hq, q0, b, &c.full[0]);
        tma_load_3d(sdo, &tm_do, h * p.hdo, q0, b, &c.full[0]);
      }
      tma_load_3d(sk + st * kSmall, &tm_k, h * p.hk, t * kTile, b, &c.full[st]);
      tma_load_3d(sv + st * kSmall, &tm_v, h * p.hv, t * kTile, b, &c.full[st]);
    };
    if (n_tiles > 0) {
      load(0);
      if (elect_one()) {
        mbar_expect_tx(c.extra, 2 * kBig);
        tma_load_3d(sds, &tm_o32, h * kTile, q0, b, c.extra);
        tma_load_3d(sds + kBig, &tm_o32, h * kTile + 32, q0, b, c.extra);
      }
      if (n_tiles > 1) load(1);
      pipe_issue(w, n_tiles, p.status, load,
                 [&](int t) {
                   mma64_warp<false>(t_s, sq, sk + (t & 1) * kSmall, false);
                   mma64_warp<false>(t_dp, sdo, sv + (t & 1) * kSmall, false);
                 },
                 [&](int t) { mma64_warp<true>(t_dq, sds, sk + (t & 1) * kSmall, t > 0); }, [](int) {});
    }
  } else {
    const int row = q0 + tid;
    const int n = row < p.tq ? visible(p, row, klen) : 0;
    const uint32_t t_row = c.tmem + ((uint32_t)(tid & ~31) << 16);
    float lse = INFINITY, delta = 0.f;
    bool ok = true;
    if (n_tiles > 0) {
      if (row < p.tq) lse = p.lse[(long long)z * p.tq + row];
      ok = pipe_wait(w, &c.full[0], 0, p.status, 9) && pipe_wait(w, c.extra, 0, p.status, 9);
      if (ok) {
        delta = dot_row64(sds, sdo, tid);
        if (row < p.tq) p.delta[(long long)z * p.tq + row] = delta;
      }
    }
    const float cs = p.scale * kLog2e;
    const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
    for (int it = 0; it < n_tiles && ok; ++it) {
      uint2 bits = make_uint2(0u, 0u);
      if (DROP && row < p.tq) bits = *reinterpret_cast<const uint2*>(p.keep + ((long long)z * p.tq + row) * p.words + it * 2);
      ok = pipe_wait(w, w.scores, it, p.status, 10);
      if (!ok) break;
      float s[64], dp[64];
      tmem_ld64(t_row, s);
      tmem_ld64(t_row + 64, dp);
      pipe_arrive(w.taken);
      const int left = n - it * kTile;
      auto grad = [&](int j) {
        float d = dp[j];
        if (DROP) d = (((j < 32 ? bits.x : bits.y) >> (j & 31)) & 1u) ? d * keep_scale : 0.f;
        return ex2(fmaf(s[j], cs, -lse)) * (d - delta);
      };
      if (__all_sync(0xffffffffu, left >= kTile)) {
#pragma unroll
        for (int j = 0; j < 64; ++j) s[j] = grad(j);
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j) s[j] = j < left ? grad(j) : 0.f;
      }
      if (it > 0) {
        ok = pipe_wait(w, w.out, it - 1, p.status, 11);  // dS of the tile before has been read
        if (!ok) break;
      }
      store_row64(sds, tid, s);
      fence_proxy_async_smem();
      pipe_arrive(w.put);
    }
    if (ok && n_tiles > 0) ok = pipe_wait(w, w.out, n_tiles - 1, p.status, 12);
    if (ok) {
      float s[64];
      if (n_tiles > 0) tmem_ld64(t_row + 128, s);
#pragma unroll
      for (int j = 0; j < 64; ++j) s[j] = n_tiles > 0 ? s[j] * p.scale : 0.f;
      store_row64(sq, tid, s);
      fence_proxy_async_smem();
    }
    rows_sync<kThreads>();
    if (tid == 0 && ok && !*c.abort_flag) {
      tma_store_3d(&tm_dq, h * kTile, q0, b, sq);
      tma_store_commit();
      tma_store_wait_read();
    }
  }
  cta_end<256>(c);
}

template <bool DROP>
__global__ void __launch_bounds__(kCta, 2)
flash_bwd_kv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                    const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                    const Flash p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sk = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sv = sk + kBig;
  uint8_t* sq = sv + kBig;
  uint8_t* sdo = sq + 2 * kSmall;
  uint8_t* sp = sdo + 2 * kSmall;
  uint8_t* sds = sp + kBig;
  // per warp of rows: (log-sum, delta) of the 64 queries of a tile, and the dropout bits of the warp's 32 keys
  float2* stat = reinterpret_cast<float2*>(sds + kBig) + (threadIdx.x >> 5) * 64;
  uint32_t* kept = reinterpret_cast<uint32_t*>(sds + kBig + 2048) + (threadIdx.x >> 5) * 64;
  const Pipe w = pipe_begin<256, 4>(sds + kBig + 2048 + 1024);
  const Cta& c = w.c;
  rb_pdl_wait();
  rb_pdl_launch();
  const int tid = threadIdx.x;
  const int z = blockIdx.x % p.bh;
  const int k0 = (int)(blockIdx.x / p.bh) * kRows;  // causal: the first keys have the most queries
  const int b = z / p.heads, h = z - b * p.heads;
  const int klen = p.k_lens ? min(p.k_lens[b], p.tk) : p.tk;
  const int first = p.causal ? max(0, k0 - p.shift) / kTile : 0;  // queries before cannot see the first key of the tile
  const int n_tiles = k0 < klen ? max(0, (p.tq + kTile - 1) / kTile - first) : 0;
  const uint32_t t_s = c.tmem, t_dp = c.tmem + 64, t_dv = c.tmem + 128, t_dk = c.tmem + 192;
  if (tid >= kThreads) {
    auto load = [&](int t) {
      if (!elect_one()) return;
      const int st = t & 1;
      mbar_expect_tx(&c.full[st], 2 * kSmall + (t == 0 ? 2 * kBig : 0));
      if (t == 0) {
        tma_load_3d(sk, &tm_k, h * p.hk, k0, b, &c.full[0]);
        tma_load_3d(sv, &tm_v, h * p.hv, k0, b, &c.full[0]);
      }
      tma_load_3d(sq + st * kSmall, &tm_q, h * p.hq, (first + t) * kTile, b, &c.full[st]);
      tma_load_3d(sdo + st * kSmall, &tm_do, h * p.hdo, (first + t) * kTile, b, &c.full[st]);
    };
    if (n_tiles > 0) {
      load(0);
      if (n_tiles > 1) load(1);
      pipe_issue(w, n_tiles, p.status, load,
                 [&](int t) {
                   mma64_warp<false>(t_s, sk, sq + (t & 1) * kSmall, false);
                   mma64_warp<false>(t_dp, sv, sdo + (t & 1) * kSmall, false);
                 },
                 [&](int t) {
                   mma64_warp<true>(t_dv, sp, sdo + (t & 1) * kSmall, t > 0);
                   mma64_warp<true>(t_dk, sds, sq + (t & 1) * kSmall, t > 0);
                 },
                 [](int) {});
    }
  } else {
    const int key = k0 + tid, lane = tid & 31;
    // queries that see this key: [lo, tq)
    const int lo = key < klen ? (p.causal ? max(0, key - p.shift) : 0) : p.tq;
    const uint32_t t_row = c.tmem + ((uint32_t)(tid & ~31) << 16);
    const float cs = p.scale * kLog2e;
    const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
    float2 ahead[2];     // of the queries lane and lane + 32 of the next tile
    uint32_t bits[2];
    auto fetch = [&](int t) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int q = (first + t) * kTile + lane + 32 * e;
        const long long at = (long long)z * p.tq + q;
        ahead[e] = q < p.tq ? make_float2(p.lse[at], p.delta[at]) : make_float2(INFINITY, 0.f);
        if (DROP) bits[e] = q < p.tq ? p.keep[at * p.words + k0 / 32 + (tid >> 5)] : 0u;
      }
    };
    if (n_tiles > 0) fetch(0);
    bool ok = true;
    for (int it = 0; it < n_tiles; ++it) {
      __syncwarp();  // the statistics of the tile before have been read
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        stat[lane + 32 * e] = ahead[e];
        if (DROP) kept[lane + 32 * e] = bits[e];
      }
      __syncwarp();
      if (it + 1 < n_tiles) fetch(it + 1);
      ok = pipe_wait(w, w.scores, it, p.status, 13);
      if (!ok) break;
      float s[64], dp[64];
      tmem_ld64(t_row, s);
      tmem_ld64(t_row + 64, dp);
      pipe_arrive(w.taken);
      const int q_base = (first + it) * kTile;
      auto both = [&](int j, bool vis) {
        const float2 ld = stat[j];
        float pr = ex2(fmaf(s[j], cs, -ld.x));
        float d = dp[j], pd = pr;
        if (DROP) {
          const bool k = (kept[j] >> lane) & 1u;
          d = k ? d * keep_scale : 0.f;
          pd = k ? pr * keep_scale : 0.f;
        }
        dp[j] = vis ? pr * (d - ld.y) : 0.f;
        s[j] = vis ? pd : 0.f;
      };
      if (__all_sync(0xffffffffu, q_base >= lo && q_base + kTile <= p.tq)) {
#pragma unroll
        for (int j = 0; j < 64; ++j) both(j, true);
      } else {
#pragma unroll
        for (int j = 0; j < 64; ++j) both(j, q_base + j >= lo && q_base + j < p.tq);
      }
      if (it > 0) {
        ok = pipe_wait(w, w.out, it - 1, p.status, 18);  // P and dS of the tile before have been read
        if (!ok) break;
      }
      store_row64(sp, tid, s);
      store_row64(sds, tid, dp);
      fence_proxy_async_smem();
      pipe_arrive(w.put);
    }
    if (ok && n_tiles > 0) ok = pipe_wait(w, w.out, n_tiles - 1, p.status, 19);
    if (ok) {
      float s[64], dp[64];
      if (n_tiles > 0) {
        tmem_ld64(t_row + 128, s);
        tmem_ld64(t_row + 192, dp);
      }
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        s[j] = n_tiles > 0 ? s[j] : 0.f;
        dp[j] = n_tiles > 0 ? dp[j] * p.scale : 0.f;
      }
      store_row64(sv, tid, s);
      store_row64(sk, tid, dp);
      fence_proxy_async_smem();
    }
    rows_sync<kThreads>();
    if (tid == 0 && ok && !*c.abort_flag) {
      tma_store_3d(&tm_dv, h * kTile, k0, b, sv);
      tma_store_3d(&tm_dk, h * kTile, k0, b, sk);
      tma_store_commit();
      tma_store_wait_read();
    }
  }
  cta_end<256>(c);
}

// Both gradients in one kernel where queries and keys fit one tile (at most 128 of each): one CTA per (batch entry, head), scores and dO V^T computed
// once, P and dS as operands of dV = P^T dO, dQ = scale dS K and dK = scale dS^T Q one after the other in the same 32 KB. A thread holds its row
// of P in registers, so the row sums of P * dP are taken from 32-bit values where they are used, and neither kernel of the two-pass form nor the
// 32-bit copy of the output is needed. 250 x 100 x 8 heads: 180 MB and 64 us in a profile that gave the two passes 56 + 74 (and the forward pass 5 us
// less without the copy): a training pass 399 -> 335 us; 250 x 20: 213 -> 143. Two CTAs per SM, bound by the chain load -> product -> row work ->
// products of each.
template <bool DROP>
__global__ void __launch_bounds__(kThreads, 2)
flash_bwd_small_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk,
                       const __grid_constant__ CUtensorMap tm_dv, const Flash p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sk = sq + kBig;
  uint8_t* sv = sk + kBig;
  uint8_t* sdo = sv + kBig;
  uint8_t* sx = sdo + kBig;  // P, then dS: two panels of 64 keys
  const Cta c = cta_begin<256>(sx + 2 * kBig);
  if (threadIdx.x == 0) {
    prefetch_map(&tm_q);
    prefetch_map(&tm_k);
    prefetch_map(&tm_v);
    prefetch_map(&tm_do);
  }
  rb_pdl_wait();
  rb_pdl_launch();
  const int tid = threadIdx.x;
  const int z = blockIdx.x, b = z / p.heads, h = z - b * p.heads;
  const int klen = p.k_lens ? max(0, min(p.k_lens[b], p.tk)) : p.tk;
  const int row = tid;
  const int n = row < p.tq ? visible(p, row, klen) : 0;
  // steps of 16 keys and queries; what lies behind the last step is not multiplied: padding that is not a number stays out as it does elsewhere
  const int key_steps = (visible(p, p.tq - 1, klen) + 15) / 16, query_steps = (p.tq + 15) / 16;
  const uint32_t t_row = c.tmem + ((uint32_t)(tid & ~31) << 16);
  const uint32_t t_s = c.tmem, t_dp = c.tmem + 128, t_dv = c.tmem, t_dq = c.tmem + 64, t_dk = c.tmem + 128;
  bool ok = true;
  const bool any = key_steps > 0;
  if (tid < 32 && any) {  // (loads and products: one lane of the first warp)
    if (elect_one()) {
      mbar_expect_tx(&c.full[0], 4 * kBig);
      tma_load_3d(sq, &tm_q, h * p.hq, 0, b, &c.full[0]);
      tma_load_3d(sk, &tm_k, h * p.hk, 0, b, &c.full[0]);
      tma_load_3d(sdo, &tm_do, h * p.hdo, 0, b, &c.full[0]);
      tma_load_3d(sv, &tm_v, h * p.hv, 0, b, &c.full[0]);
    }
    __syncwarp();
    ok = __all_sync(0xffffffffu, wait_or_abort(c, &c.full[0], 0, p.status, 14));
    if (ok) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(16 * key_steps >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) umma_f16_warp(t_s, desc_lo(smem_u32(sq), 16) + 2 * kk, desc_lo(smem_u32(sk), 16) + 2 * kk, idesc, kk > 0);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) umma_f16_warp(t_dp, desc_lo(smem_u32(sdo), 16) + 2 * kk, desc_lo(smem_u32(sv), 16) + 2 * kk, idesc, kk > 0);
      umma_commit_warp(c.done);
    }
  }
  const float lse = row < p.tq ? p.lse[(long long)z * p.tq + row] : INFINITY;
  uint4 bits = make_uint4(0u, 0u, 0u, 0u);
  if (DROP && row < p.tq) bits = *reinterpret_cast<const uint4*>(p.keep + ((long long)z * p.tq + row) * p.words);
  const uint32_t keep[4] = {bits.x, bits.y, bits.z, bits.w};
  const float keep_scale = DROP ? 1.f / (1.f - p.p_drop) : 1.f;
  const float cs = p.scale * kLog2e;
  if (any) {
    ok = ok && wait_or_abort(c, c.done, 0, p.status, 15);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    float pr[128], delta = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t s[32], d[32];
      tmem_ld32(t_row + 32 * q, s);
      tmem_ld32(t_row + 128 + 32 * q, d);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int key = 32 * q + j;
        const float v = key < n ? ex2(fmaf(__uint_as_float(s[j]), cs, -lse)) : 0.f;
        float g = __uint_as_float(d[j]);
        if (DROP) g = (keep[q] >> j & 1u) ? g * keep_scale : 0.f;
        pr[key] = v;
        if (key < n) delta = fmaf(v, g, delta);
      }
      if (q & 1) {
        float o[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const int key = 32 * (q - 1) + j;
          o[j] = DROP ? ((keep[key >> 5] >> (key & 31) & 1u) ? pr[key] * keep_scale : 0.f) : pr[key];
        }
        store_row64(sx + (q >> 1) * kBig, tid, o);
      }
    }
    fence_proxy_async_smem();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    ok = !__syncthreads_or(ok ? 0 : 1);
    // contraction over the queries: A [query][key] is M-major in two panels of 64 keys, B [query][64] N-major
    constexpr uint32_t idesc_t = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    constexpr uint32_t idesc_n = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint32_t x_t = desc_lo(smem_u32(sx), kBig), x_n = desc_lo(smem_u32(sx), 16);
    if (tid < 32 && ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int kk = 0; kk < query_steps; ++kk) umma_f16_warp(t_dv, x_t + 128 * kk, desc_lo(smem_u32(sdo), 8192) + 128 * kk, idesc_t, kk > 0);
      umma_commit_warp(c.done);
    }
    __syncwarp();
    uint32_t ds[64];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t d[32];
      tmem_ld32(t_row + 128 + 32 * q, d);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        float v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int key = 32 * q + j + e;
          float g = __uint_as_float(d[j + e]);
          if (DROP) g = (keep[q] >> (j + e) & 1u) ? g * keep_scale : 0.f;
          v[e] = key < n ? pr[key] * (g - delta) : 0.f;
        }
        ds[16 * q + j / 2] = pack2(v[0], v[1]);
      }
    }
    ok = ok && wait_or_abort(c, c.done, 1, p.status, 16);  // P has been read
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 16; ++q)
      *reinterpret_cast<uint4*>(sx + (q >> 3) * kBig + tid * 128 + (((q & 7) ^ (tid & 7)) << 4)) = make_uint4(ds[4 * q], ds[4 * q + 1], ds[4 * q + 2], ds[4 * q + 3]);
    fence_proxy_async_smem();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    ok = !__syncthreads_or(ok ? 0 : 1);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid < 32 && ok) {
      for (int kk = 0; kk < key_steps; ++kk)
        umma_f16_warp(t_dq, x_n + (kk >> 2) * (kBig >> 4) + (kk & 3) * 2, desc_lo(smem_u32(sk), 8192) + 128 * kk, idesc_n, kk > 0);
      for (int kk = 0; kk < query_steps; ++kk) umma_f16_warp(t_dk, x_t + 128 * kk, desc_lo(smem_u32(sq), 8192) + 128 * kk, idesc_t, kk > 0);
      umma_commit_warp(c.done);
    }
    __syncwarp();
    float o[64];
    if (ok) {
      tmem_ld64(t_row, o);
      store_row64(sv, tid, o);
    }
    ok = ok && wait_or_abort(c, c.done, 0, p.status, 17);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    if (ok) {
      tmem_ld64(t_row + 64, o);
#pragma unroll
      for (int j = 0; j < 64; ++j) o[j] *= p.scale;
      store_row64(sq, tid, o);
      tmem_ld64(t_row + 128, o);
#pragma unroll
      for (int j = 0; j < 64; ++j) o[j] *= p.scale;
      store_row64(sk, tid, o);
    }
  } else {
    float o[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) o[j] = 0.f;
    store_row64(sq, tid, o);
    store_row64(sk, tid, o);
    store_row64(sv, tid, o);
  }
  fence_proxy_async_smem();
  if (!__syncthreads_or(ok ? 0 : 1) && tid == 0) {
    tma_store_3d(&tm_dq, h * kTile, 0, b, sq);
    tma_store_3d(&tm_dk, h * kTile, 0, b, sk);
    tma_store_3d(&tm_dv, h * kTile, 0, b, sv);
    tma_store_commit();
    tma_store_wait_read();  // (the writes complete like any other store of the grid)
  }
  cta_end<256>(c);
}

constexpr int kFwdSmem = 2 * kBig + 4 * kSmall + 64 + 1024;
constexpr int kBwdQSmem = 4 * kBig + 4 * kSmall + 64 + 1024;
constexpr int kBwdSmallSmem = 6 * kBig + 64 + 1024;
constexpr int kBwdKvSmem = 4 * kBig + 4 * kSmall + 2048 + 1024 + 64 + 1024;

int launch_failed(const char* what, cudaError_t e) {
  rb_set_error("%s: %s", what, cudaGetErrorString(e));
  return RB_ERR_LAUNCH;
}

// geom: B, H, Tq, Tk, causal, causal shift, then row and head pitch (elements) of q, k, v, dO, Tqp, Tkp, dropout words per row
enum { G_B, G_H, G_TQ, G_TK, G_CAUSAL, G_SHIFT, G_RQ, G_HQ, G_RK, G_HK, G_RV, G_HV, G_RDO, G_HDO, G_TQP, G_TKP, G_WORDS };

Flash make_params(const int* g, const int* k_lens, float* lse, float* delta, void* keep, float scale, float p_drop, const long long* seed,
                  const long long* offset, int* status) {
  Flash p = {};
  p.k_lens = k_lens; p.lse = lse; p.delta = delta; p.keep = (uint32_t*)keep; p.seed = seed; p.offset = offset; p.status = status;
  p.heads = g[G_H]; p.bh = g[G_B] * g[G_H]; p.tq = g[G_TQ]; p.tk = g[G_TK]; p.causal = g[G_CAUSAL]; p.shift = g[G_SHIFT];
  p.hq = g[G_HQ]; p.hk = g[G_HK]; p.hv = g[G_HV]; p.hdo = g[G_HDO]; p.words = g[G_WORDS]; p.tqp = g[G_TQP]; p.tkp = g[G_TKP];
  p.scale = scale; p.p_drop = p_drop;
  return p;
}

int map_of(CUtensorMap* m, const void* base, const int* g, int t, int row_pitch, int head_pitch, int box_rows) {
  return make_map_3d(m, base, (long long)(g[G_H] - 1) * head_pitch + kTile, t, g[G_B], row_pitch, (long long)t * row_pitch, box_rows);
}

}  // namespace

// whether the backward pass runs as one kernel, which takes no 32-bit copy of the output
RB_EXPORT int rb200_flash_bwd_one_kernel(int tq, int tk) { return tq <= kRows && tk <= kRows; }

// o [B, Tq, H * 64] bf16; o32 (null: no backward pass follows) the same in fp32, for the row sums dO . O of the backward pass: from the 16-bit
// values those are off by 2^-9 of |dO| |O| in one direction for a whole row of dS, which is far more than dS where the values share an offset
// (512 keys, values 24 + n(0, 1), keys 4 + n(0, 1): error of dQ 3.07, from 32 bits 0.11; a training pass over 250 x 100 x 8 heads 164 -> 176 us)
RB_EXPORT int rb200_flash_fwd(const void* q, const void* k, const void* v, void* o, float* o32, float* lse, void* keep, const int* k_lens, const int* g, float scale,
                              float p_drop, const long long* seed, const long long* offset, int* status, cudaStream_t stream) {
  if (g[G_B] <= 0 || g[G_H] <= 0 || g[G_TQ] <= 0) return RB_OK;
  if (g[G_TK] <= 0) {
    rb_set_error("flash_fwd: no keys for %d queries", g[G_TQ]);
    return RB_ERR_ARG;
  }
  if (p_drop > 0.f && (!seed || !offset || !keep || !(p_drop < 1.f))) {
    rb_set_error("flash_fwd: dropout of %f needs seed, offset and a buffer for its decisions, and a rate below 1", p_drop);
    return RB_ERR_ARG;
  }
  Flash p = make_params(g, k_lens, lse, nullptr, keep, scale, p_drop, seed, offset, status);
  p.tiles = (p.tq + kRows - 1) / kRows;
  const long long ctas = (long long)p.tiles * g[G_B] * g[G_H];
  if (ctas > 0x7fffffffLL) {
    rb_set_error("flash_fwd: too many tiles");
    return RB_ERR_ARG;
  }
  const int hd = g[G_H] * kTile;
  p.save = o32 != nullptr;
  CUtensorMap tq, tk, tv, to, to32;
  int st = map_of(&tq, q, g, p.tq, g[G_RQ], g[G_HQ], kRows);
  if (!st) st = map_of(&tk, k, g, p.tk, g[G_RK], g[G_HK], kTile);
  if (!st) st = map_of(&tv, v, g, p.tk, g[G_RV], g[G_HV], kTile);
  if (!st) st = map_of(&to, o, g, p.tq, hd, kTile, kRows);
  to32 = to;
  if (!st && o32) st = make_map_3d(&to32, o32, hd, p.tq, g[G_B], hd, (long long)p.tq * hd, kRows, true);
  if (st) return st;
  auto kernel = p_drop > 0.f ? flash_fwd_kernel<true> : flash_fwd_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
  if (e != cudaSuccess) return launch_failed("flash_fwd", e);
  rb_launch_pdl(kernel, dim3((unsigned)ctas), dim3(kCta), kFwdSmem, stream, tq, tk, tv, to, to32, p);
  return rb_check_launch("flash_fwd");
}

RB_EXPORT int rb200_flash_bwd(const void* q, const void* k, const void* v, const float* o32, const void* d_o, void* dq, void* dk, void* dv, float* lse,
                              float* delta, void* keep, const int* k_lens, const int* g, float scale, float p_drop, int* status, cudaStream_t stream) {
  if (g[G_B] <= 0 || g[G_H] <= 0 || (g[G_TQ] <= 0 && g[G_TK] <= 0)) return RB_OK;
  if (g[G_TQ] <= 0 || g[G_TK] <= 0) {
    rb_set_error("flash_bwd: %d queries, %d keys", g[G_TQ], g[G_TK]);
    return RB_ERR_ARG;
  }
  if (p_drop > 0.f && (!keep || !(p_drop < 1.f))) {
    rb_set_error("flash_bwd: dropout of %f needs the decisions of the forward pass and a rate below 1", p_drop);
    return RB_ERR_ARG;
  }
  Flash p = make_params(g, k_lens, lse, delta, keep, scale, p_drop, nullptr, nullptr, status);
  const int hd = g[G_H] * kTile;
  const int tiles_q = (p.tq + kRows - 1) / kRows, tiles_k = (p.tk + kRows - 1) / kRows;
  const long long bh = (long long)g[G_B] * g[G_H];
  if (bh * tiles_q > 0x7fffffffLL || bh * tiles_k > 0x7fffffffLL) {
    rb_set_error("flash_bwd: too many tiles");
    return RB_ERR_ARG;
  }
  CUtensorMap tq, tk, tv, to, td, tg, tg2;
  if (rb200_flash_bwd_one_kernel(p.tq, p.tk)) {
    int st = map_of(&tq, q, g, p.tq, g[G_RQ], g[G_HQ], kRows);
    if (!st) st = map_of(&tk, k, g, p.tk, g[G_RK], g[G_HK], kRows);
    if (!st) st = map_of(&tv, v, g, p.tk, g[G_RV], g[G_HV], kRows);
    if (!st) st = map_of(&td, d_o, g, p.tq, g[G_RDO], g[G_HDO], kRows);
    if (!st) st = map_of(&to, dq, g, p.tq, hd, kTile, kRows);
    if (!st) st = map_of(&tg, dk, g, p.tk, hd, kTile, kRows);
    if (!st) st = map_of(&tg2, dv, g, p.tk, hd, kTile, kRows);
    if (st) return st;
    auto kernel = p_drop > 0.f ? flash_bwd_small_kernel<true> : flash_bwd_small_kernel<false>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmallSmem);
    if (e != cudaSuccess) return launch_failed("flash_bwd", e);
    rb_launch_pdl(kernel, dim3((unsigned)bh), dim3(kThreads), kBwdSmallSmem, stream, tq, tk, tv, td, to, tg, tg2, p);
    return rb_check_launch("flash_bwd_small");
  }
  if (!o32 || !delta) {
    rb_set_error("flash_bwd: %d queries, %d keys need the output in 32 bits", p.tq, p.tk);
    return RB_ERR_ARG;
  }
  int st = map_of(&tq, q, g, p.tq, g[G_RQ], g[G_HQ], kRows);
  if (!st) st = map_of(&tk, k, g, p.tk, g[G_RK], g[G_HK], kTile);
  if (!st) st = map_of(&tv, v, g, p.tk, g[G_RV], g[G_HV], kTile);
  if (!st) st = make_map_3d(&to, o32, hd, p.tq, g[G_B], hd, (long long)p.tq * hd, kRows, true);
  if (!st) st = map_of(&td, d_o, g, p.tq, g[G_RDO], g[G_HDO], kRows);
  if (!st) st = map_of(&tg, dq, g, p.tq, hd, kTile, kRows);
  if (st) return st;
  auto kq = p_drop > 0.f ? flash_bwd_q_kernel<true> : flash_bwd_q_kernel<false>;
  auto kkv = p_drop > 0.f ? flash_bwd_kv_kernel<true> : flash_bwd_kv_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kq, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdQSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kkv, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdKvSmem);
  if (e != cudaSuccess) return launch_failed("flash_bwd", e);
  p.tiles = tiles_q;
  rb_launch_pdl(kq, dim3((unsigned)(bh * tiles_q)), dim3(kCta), kBwdQSmem, stream, tq, tk, tv, to, td, tg, p);
  st = rb_check_launch("flash_bwd_q");
  if (!st) st = map_of(&tq, q, g, p.tq, g[G_RQ], g[G_HQ], kTile);
  if (!st) st = map_of(&tk, k, g, p.tk, g[G_RK], g[G_HK], kRows);
  if (!st) st = map_of(&tv, v, g, p.tk, g[G_RV], g[G_HV], kRows);
  if (!st) st = map_of(&td, d_o, g, p.tq, g[G_RDO], g[G_HDO], kTile);
  if (!st) st = map_of(&tg, dk, g, p.tk, hd, kTile, kRows);
  if (!st) st = map_of(&tg2, dv, g, p.tk, hd, kTile, kRows);
  if (st) return st;
  p.tiles = tiles_k;
  rb_launch_pdl(kkv, dim3((unsigned)(bh * tiles_k)), dim3(kCta), kBwdKvSmem, stream, tq, tk, tv, td, tg, tg2, p);
  return rb_check_launch("flash_bwd_kv");
}

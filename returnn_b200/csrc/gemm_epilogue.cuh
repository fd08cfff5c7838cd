// Epilogue and work-unit decoding shared by the persistent tcgen05 GEMM kernels (one-CTA and CTA-pair variants).
#pragma once
#include "tcgen05.cuh"
#include "gemm.h"

namespace rbg {

using namespace rbt;

constexpr int BK = 64;

struct Params {
  RbGemm g;
  int tiles_m, tiles_n, split, kb_per_split, num_kb, units;
  int vec_ok;    // all epilogue pointers 16-byte aligned and ldc % 8 == 0
  int bias_vec;  // fp32 bias, 16-byte aligned: read as two float4
  int tma_store; // the output leaves through shared memory and bulk tensor stores (tensor maps of c / c2 passed to the kernel)
  int step, step_sp, step_m, step_n;  // CTA-pair kernel: from a pair's unit to its next, and the same in slices, rows and columns of tiles
  int seg_kb;    // CTA-pair kernel: K blocks per product of split operands (0: not split)
  long long c_next;   // c_next - c in elements (a_next: g.alpha is 1, and alpha_first that of the first problems)
  float alpha_first;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ float act_grad(float z, int act) {
  if (act == 1) return z > 0.f ? 1.f : 0.f;
  if (act == 2) {
    float s = __fdividef(1.f, 1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
  }
  if (act == 3) {
    float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
    float pdf = __expf(-0.5f * z * z) * 0.3989422804014327f;
    return cdf + z * pdf;
  }
  return 1.f;
}

// The activation (or its derivative) on 8 values. The kind is uniform over the kernel: it is tested ONCE per group, outside the
// element loops, so that the cheap kinds do not carry the instructions of the expensive one (erf) as predicated code.
__device__ __forceinline__ float silu_tanh(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return x * (0.5f + 0.5f * t);  // x * sigmoid(x), sigmoid(x) = (1 + tanh(x / 2)) / 2: one special-function instruction
}
__device__ __forceinline__ void act8(float* v, int act) {
  if (act == 2) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = silu_tanh(v[i]);
  } else if (act == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = fmaxf(v[i], 0.f);
  } else if (act == 3) {
#pragma unroll  // no rolled loop here: a dynamically indexed v[] would move the array, for every kind, from registers to local memory
    for (int i = 0; i < 8; ++i) v[i] = 0.5f * v[i] * (1.f + erff(v[i] * 0.70710678118654752f));
  }
}
__device__ __forceinline__ void act_grad8(float* v, const float* z, int act) {
  if (act == 2) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float t;
      asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * z[i]));
      const float s = 0.5f + 0.5f * t;
      v[i] *= s * (1.f + z[i] * (1.f - s));
    }
  } else if (act == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = z[i] > 0.f ? v[i] : 0.f;
  } else if (act == 3) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] *= act_grad(z[i], 3);
  }
}

__device__ __forceinline__ void load8_bf16(const void* base, size_t off, bool vec, int nvalid, float* out) {
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(base) + off;
  if (vec) {
    uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(h[i]);
      out[2 * i] = f.x;
      out[2 * i + 1] = f.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = i < nvalid ? __bfloat162float(p[i]) : 0.f;
  }
}

__device__ __forceinline__ void store8_bf16(void* base, size_t off, bool vec, int nvalid, const float* v) {
  __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(base) + off;
  if (vec) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = u;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < nvalid) p[i] = __float2bfloat16(v[i]);
  }
}

// one lane's share of the epilogue: 8 consecutive columns [col, col+8) of one output row.
// FULL = false compiles the common case only (scale, bias, activation, store): no activation gradient, dropout or residual,
// which keeps the instruction stream of the epilogue warps short.
template <bool FULL>
__device__ __forceinline__ void epilogue_group(const Params& p, int row, int col, int n_extent, size_t c_off, float* v) {
  const RbGemm& g = p.g;
  const int nvalid = min(8, n_extent - col);
  const bool vec = p.vec_ok && nvalid == 8 && (c_off & 7) == 0;
  const size_t off = c_off + (size_t)row * g.ldc + col;
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] *= g.alpha;
  if (g.bias && p.bias_vec && nvalid == 8) {
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.bias) + col));
    const float4 b1 = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.bias) + col) + 1);
    v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
    v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
  } else if (g.bias) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < nvalid) {
        v[i] += g.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g.bias)[col + i])
                            : __ldg(reinterpret_cast<const float*>(g.bias) + col + i);
      }
    }
  }
  float pre[8];
  if (FULL && g.dact_z) {
    float z[8];
    load8_bf16(g.dact_z, off, vec, nvalid, z);
    act_grad8(v, z, g.act);
  } else if (g.act) {
#pragma unroll
    for (int i = 0; i < 8; ++i) pre[i] = v[i];
    act8(v, g.act);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) pre[i] = v[i];
  }
  if (FULL && g.drop_p > 0.f) {
    const uint64_t sd = (uint64_t)g.seed[0];
    const uint64_t c = (uint64_t)g.offset[0] + g.drop_site + (uint64_t)off;
    rb_dropout_apply8(make_uint2((uint32_t)sd, (uint32_t)(sd >> 32)), c, rb_dropout_thresh16(g.drop_p), 1.f / (1.f - g.drop_p), v);
  }
  if (FULL && g.resid) {
    float rs[8];
    load8_bf16(g.resid, off, vec, nvalid, rs);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = rs[i] + g.res_scale * v[i];
  }
  if (g.out_fp32) {
    float* c = reinterpret_cast<float*>(g.c) + off;
    if (g.accumulate == 2) {
      if (vec) {
        atomicAdd(reinterpret_cast<float4*>(c), make_float4(v[0], v[1], v[2], v[3]));
        atomicAdd(reinterpret_cast<float4*>(c) + 1, make_float4(v[4], v[5], v[6], v[7]));
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < nvalid) atomicAdd(c + i, v[i]);
      }
    } else if (vec) {
      float4 a = make_float4(v[0], v[1], v[2], v[3]), b = make_float4(v[4], v[5], v[6], v[7]);
      if (g.accumulate == 1) {
        float4 oa = reinterpret_cast<float4*>(c)[0], ob = reinterpret_cast<float4*>(c)[1];
        a.x += oa.x; a.y += oa.y; a.z += oa.z; a.w += oa.w;
        b.x += ob.x; b.y += ob.y; b.z += ob.z; b.w += ob.w;
      }
      reinterpret_cast<float4*>(c)[0] = a;
      reinterpret_cast<float4*>(c)[1] = b;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < nvalid) c[i] = g.accumulate == 1 ? c[i] + v[i] : v[i];
    }
  } else if (g.c2) {
    store8_bf16(g.c, off, vec, nvalid, pre);
    store8_bf16(g.c2, off, vec, nvalid, v);
  } else {
    store8_bf16(g.c, off, vec, nvalid, v);
  }
}

// one work unit: output tile (m0, n0) of problem z, K blocks [kb0, kb1)
struct Unit {
  int m0, n0, kb0, kb1, M, N;
  int c_r0;  // row of the stored output that row 0 of this unit's product is (slices one behind the other)
  int a_r0, a_c0, b_r0, b_c0;
  size_t c_off;
  bool valid, next;  // next: of the problems a_next, b_next, c_next
};

template <int BM, int BN>
__device__ __forceinline__ Unit decode_unit(const Params& p, int u) {
  const RbGemm& g = p.g;
  Unit w;
  w.c_r0 = 0;
  w.next = false;
  const int tiles = p.tiles_m * p.tiles_n;
  if (g.batch > 0) {
    int z = u / tiles;
    const int t = u % tiles;
    if (z >= g.batch) {
      w.next = true;
      z -= g.batch;
    }
    const int zb = z / g.heads, zh = z % g.heads;
    const int len = g.lens ? g.lens[zb] : 0;
    w.M = g.m_from_lens ? len : g.m;
    w.N = g.n_from_lens ? len : g.n;
    const int K = g.k_from_lens ? len : g.k;
    w.m0 = (t / p.tiles_n) * BM;
    w.n0 = (t % p.tiles_n) * BN;
    w.kb0 = 0;
    w.kb1 = K > 0 ? (K + BK - 1) / BK : 0;
    w.a_r0 = (int)(zb * g.a_rb + zh * g.a_rh); w.a_c0 = (int)(zb * g.a_cb + zh * g.a_ch);
    w.b_r0 = (int)(zb * g.b_rb + zh * g.b_rh); w.b_c0 = (int)(zb * g.b_cb + zh * g.b_ch);
    w.c_off = (size_t)zb * g.c_sb + (size_t)zh * g.c_sh + (w.next ? (size_t)p.c_next : 0);
    w.valid = w.m0 < w.M && w.n0 < w.N && w.kb1 > 0;
    if (g.win == 1) w.valid = w.valid && w.n0 < g.win_center - w.m0 + len && w.n0 + BN > g.win_center - (min(w.m0 + BM, len) - 1);
  } else {
    const int sp = u / tiles, t = u % tiles;
    w.M = g.m; w.N = g.n;
    w.m0 = (t / p.tiles_n) * BM;
    w.n0 = (t % p.tiles_n) * BN;
    w.kb0 = sp * p.kb_per_split;
    w.kb1 = min(p.num_kb, w.kb0 + p.kb_per_split);
    w.a_r0 = w.a_c0 = w.b_r0 = w.b_c0 = 0;
    w.c_off = 0;
    w.valid = true;
  }
  return w;
}

// Walks over the K blocks of a unit whose A is a band (win = 2): which of them have a column of the tile in their window. The first is always
// taken (it starts the accumulator), as zeros where it has none. Producer and MMA issuer walk alike.
struct BandWalk {
  const RbGemm& g;
  int b, i0, len, m0, m1;
  bool zeros = false;
  __device__ __forceinline__ BandWalk(const RbGemm& g_, const Unit& w, int bm) : g(g_), b(0), i0(0), len(0), m0(w.a_c0 + w.m0), m1(w.a_c0 + w.m0 + bm) {
    if (g.win != 2) return;
    const int rows = g.heads > 0 ? (int)(w.a_r0 % ((long long)g.batch / g.heads * g.k)) : 0;  // row within the band of one head
    b = rows / g.win_lp;
    i0 = rows - b * g.win_lp - BK;
    len = g.win_lens[b];
  }
  __device__ __forceinline__ bool skip(bool first) {  // called once per K block
    if (g.win != 2) return false;
    i0 += BK;
    if (i0 == g.win_lp) {
      i0 = 0;
      len = g.win_lens[++b];
    }
    const bool out = i0 >= len || g.win_center - i0 + len <= m0 || g.win_center - min(i0 + BK, len) + 1 >= m1;
    zeros = first && out;
    return !first && out;
  }
};

// Epilogue of the accumulator columns [c_begin, c_end) of one 128-row tile by one warp (TMEM lane quarter q), in chunks of 16
// columns: tcgen05.ld -> registers -> this warp's 2 KB staging area (fp32 rows of 64 bytes, 16-byte chunk index xor-swizzled with
// the row so that neither direction has bank conflicts) -> every lane owns 8 consecutive columns of one row -> epilogue_group.
// `arrive` is called by lane 0 once the warp's last read of the accumulator has completed (hands the TMEM buffer back to the
// MMA issuer). Many narrow warps rather than few wide ones: the epilogue is latency-bound per warp (measured about 6 stall
// cycles per issued instruction), so its throughput scales with the number of warps the schedulers can switch between.
// NEXT: two sets of problems, each with its alpha.
template <bool FULL, bool NEXT = false, typename Arrive>
__device__ __forceinline__ void epilogue_columns(const Params& p, const Unit& w, int m0, int n0, uint32_t t_addr, int c_begin, int c_end, float* stg,
                                                 int lane, int q, Arrive arrive) {
#pragma unroll 1
  for (int c0 = c_begin; c0 < c_end; c0 += 16) {
    uint32_t r[16];
    tmem_ld16(t_addr + (uint32_t)c0, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (c0 + 16 >= c_end) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive();
    }
    float4* srow = reinterpret_cast<float4*>(stg + lane * 16);
    const int sw = (lane >> 1) & 3;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      srow[j ^ sw] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
    }
    __syncwarp();
    const int cg = lane & 1;
    const int col = n0 + c0 + cg * 8;
#pragma unroll
    for (int itr = 0; itr < 2; ++itr) {
      const int rl = itr * 16 + (lane >> 1);
      const int row = m0 + q * 32 + rl;
      const float4* rrow = reinterpret_cast<const float4*>(stg + rl * 16);
      const int sr = (rl >> 1) & 3;
      const float4 a = rrow[(2 * cg) ^ sr], b = rrow[(2 * cg + 1) ^ sr];
      if (row < w.M && col < w.N) {
        float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (NEXT && p.g.a_next) {
          const float alpha = w.next ? p.g.alpha_next : p.alpha_first;
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] *= alpha;
        }
        epilogue_group<FULL>(p, row, col, w.N, w.c_off, v);
      }
    }
    __syncwarp();
  }
}

// ---- row-owner epilogue with bulk tensor stores ---------------------------------------------------------------------------------
// Every lane owns ONE accumulator row (TMEM lane = row) and reads W consecutive columns of it with one or two tcgen05.ld.x32, so
// the accumulator buffer is handed back to the MMA issuer as soon as the values are in registers. Bias, activation, activation
// gradient, dropout and residual are computed on groups of 8 consecutive columns (the same grouping and dropout counters as
// epilogue_group). The results go to this warp's 4 KB box in shared memory in the swizzled layout of the output tensor map (rows
// of 128 bytes: 64 bf16 or 32 fp32 columns; 16-byte chunk j of row r sits at chunk position j ^ (r & 7), which also keeps the
// 32 lanes' 16-byte writes on distinct banks), and ONE bulk tensor store (or bulk reduce-add for accumulate != 0) per box moves
// them to global memory: full-line writes, no st.global from the warps, rows and columns outside the matrix clipped by the TMA
// unit. The next box is written only after the previous store has finished reading shared memory (wait_group.read).

// v[8] (accumulator values of columns col .. col+7 of `row`) -> final values in v, pre-activation in pre. Loads of dact_z / resid
// only for valid elements. Same order of operations as epilogue_group.
__device__ __forceinline__ void unpack8_bf16(const uint4& u, float* out) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = __bfloat1622float2(h[i]);
    out[2 * i] = f.x;
    out[2 * i + 1] = f.y;
  }
}

// The epilogue's global input (dact_z if there is one, else resid) for the 16 columns col0 .. col0+15 of `row`, fetched into
// registers one phase ahead of its use: the first phase BEFORE the warp waits for the accumulator (the loads are in flight while
// the MMAs of the tile still run), every later phase before the arithmetic of the phase before it. Groups that are not completely
// inside the matrix are left to the in-line path of epilogue_math8 (their slot stays zero and is not used).
__device__ __forceinline__ void epilogue_prefetch16(const Params& p, int M, int N, int row, int col0, uint4& a, uint4& b) {
  const RbGemm& g = p.g;
  const void* src = g.dact_z ? g.dact_z : g.resid;
  a = make_uint4(0u, 0u, 0u, 0u);
  b = a;
  if (src == nullptr || row >= M) return;
  const __nv_bfloat16* base = reinterpret_cast<const __nv_bfloat16*>(src) + (size_t)row * g.ldc + col0;
  if (col0 + 8 <= N) a = *reinterpret_cast<const uint4*>(base);
  if (col0 + 16 <= N) b = *reinterpret_cast<const uint4*>(base + 8);
}

// in8 / in_valid: the group's prefetched input (see epilogue_prefetch_half), passed by value so that it stays in registers
template <bool FULL>
__device__ __forceinline__ void epilogue_math8(const Params& p, int row, int col, bool row_ok, int n_extent, float* v, float* pre,
                                               const uint4 in8 = make_uint4(0u, 0u, 0u, 0u), bool in_valid = false) {
  const RbGemm& g = p.g;
  const int nvalid = row_ok ? max(0, min(8, n_extent - col)) : 0;
  const bool have_in = FULL && in_valid && nvalid == 8;
  const size_t off = (size_t)row * g.ldc + col;
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] *= g.alpha;
  if (g.bias && nvalid == 8) {
    if (p.bias_vec) {
      const float4 b0 = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.bias) + col));
      const float4 b1 = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.bias) + col) + 1);
      v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
      v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] += g.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g.bias)[col + i])
                            : __ldg(reinterpret_cast<const float*>(g.bias) + col + i);
      }
    }
  } else if (g.bias) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i < nvalid) {
        v[i] += g.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g.bias)[col + i])
                            : __ldg(reinterpret_cast<const float*>(g.bias) + col + i);
      }
    }
  }
  if (FULL && g.dact_z) {
    float z[8];
    if (have_in) unpack8_bf16(in8, z);
    else load8_bf16(g.dact_z, off, nvalid == 8, nvalid, z);
    act_grad8(v, z, g.act);
  } else if (g.act) {
#pragma unroll
    for (int i = 0; i < 8; ++i) pre[i] = v[i];
    act8(v, g.act);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) pre[i] = v[i];
  }
  if (FULL && g.drop_p > 0.f) {
    const uint64_t sd = (uint64_t)g.seed[0];
    const uint64_t c = (uint64_t)g.offset[0] + g.drop_site + (uint64_t)off;
    rb_dropout_apply8(make_uint2((uint32_t)sd, (uint32_t)(sd >> 32)), c, rb_dropout_thresh16(g.drop_p), 1.f / (1.f - g.drop_p), v);
  }
  if (FULL && g.resid) {
    float rs[8];
    if (have_in && g.dact_z == nullptr) unpack8_bf16(in8, rs);
    else load8_bf16(g.resid, off, nvalid == 8, nvalid, rs);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = rs[i] + g.res_scale * v[i];
  }
}

__device__ __forceinline__ uint4 pack8_bf16(const float* v) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return u;
}

// Column sums of a box of 64 bf16 columns as it was rounded, added onto `sum`: a lane reads two columns down its rows (the 32 lanes cover a row's 128
// bytes: no bank conflicts) while the bulk store reads the same memory. As a kernel of its own that read the output again: 14.7 us at 6740 x 2048.
__device__ __forceinline__ void epilogue_column_sums(const uint8_t* box, int n_rows, int col, int n, float* sum, int lane) {
  float s0 = 0.f, s1 = 0.f;
  const uint8_t* at = box + (lane & 3) * 4;
  for (int i = 0; i < n_rows; ++i) {
    const uint32_t u = *reinterpret_cast<const uint32_t*>(at + i * 128 + (((lane >> 2) ^ (i & 7)) << 4));
    s0 += __uint_as_float(u << 16);
    s1 += __uint_as_float(u & 0xffff0000u);
  }
  if (col < n) atomicAdd(sum + col, s0);
  if (col + 1 < n) atomicAdd(sum + col + 1, s1);
}

// One warp's share of a tile: rows m0 + q*32 .. +31 (lane = row), accumulator columns [c_begin, c_begin + 64) at TMEM address
// t_addr (lane quarter already applied). box: this warp's 4 KB of shared memory, 1024-byte aligned. tm_c / tm_c2: tensor maps of the
// outputs with boxes of 32 rows x 128 bytes (64 bf16 or 32 fp32 columns; with a second output c2: 32 rows x 64 bytes, 64-byte swizzle). `arrive` hands the accumulator buffer back (lane 0).
// One warp's share of a tile in four phases of 16 columns (a rolled loop: the body is small enough to stay in the instruction
// cache, which an unrolled 64-column body is not; with 16 warps walking through it once per tile, instruction fetch was the
// largest stall reason of the unrolled form). A phase: tcgen05.ld of 16 accumulator values, request of the NEXT phase's global
// input (full epilogue), arithmetic on two groups of 8 columns, 16-byte writes into the box. The accumulator buffer is released
// after the last phase's tcgen05.ld. A box is handed to the TMA unit when it is complete: after 64 bf16 columns (one output),
// after 32 columns for fp32 outputs and for two outputs (then a pair of boxes with 64-byte rows, 64-byte swizzle: chunk j of row r
// at position j ^ ((r >> 1) & 3)), and it is written again only after that store has finished reading it.
// in_a / in_b: the prefetched input of phase 0 (valid if have_in).
template <bool FULL, typename Arrive>
__device__ __forceinline__ void epilogue_rows_tma(const Params& p, const Unit& w, int m0, int n0, uint32_t t_addr, int c_begin, uint8_t* box,
                                                  const CUtensorMap* tm_c, const CUtensorMap* tm_c2, int lane, int q, Arrive arrive,
                                                  uint4 in_a, uint4 in_b, bool have_in) {
  const RbGemm& g = p.g;
  const int row0 = m0 + q * 32;
  const int row = row0 + lane;
  const bool row_ok = row < w.M;
  const int col0 = n0 + c_begin;
  auto release = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) arrive();
  };
  if (row0 >= w.M || col0 >= w.N) {  // nothing of this warp's box lies inside the matrix (warp-uniform): nothing to read
    release();
    return;
  }
  const bool two_out = g.c2 != nullptr;
  const bool fp32 = g.out_fp32 != 0;
  const bool half_boxes = two_out || fp32;  // a box (or pair of boxes) is complete after 32 columns
  uint8_t* my_row = box + lane * 128;
  uint8_t* row_pre = box + lane * 64;
  uint8_t* row_fin = box + 2048 + lane * 64;
  const int sw = lane & 7, sw64 = (lane >> 1) & 3;
#pragma unroll 1
  for (int ph = 0; ph < 4; ++ph) {
    uint32_t r[16];
    tmem_ld16(t_addr + (uint32_t)(c_begin + 16 * ph), r);
    uint4 nx_a = make_uint4(0u, 0u, 0u, 0u), nx_b = nx_a;
    if (FULL && ph < 3 && have_in) epilogue_prefetch16(p, w.M, w.N, row, col0 + 16 * (ph + 1), nx_a, nx_b);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (ph == 3) release();
    if (ph == 0 || (half_boxes && ph == 2)) {
      if (lane == 0) tma_store_wait_read();
      __syncwarp();
    }
    const bool cols_in = col0 + 16 * ph < w.N;
#pragma unroll
    for (int gi = 0; gi < 2; ++gi) {
      float v[8], pre[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * gi + i]);
      epilogue_math8<FULL>(p, row, col0 + 16 * ph + 8 * gi, row_ok && cols_in, w.N, v, pre, gi == 0 ? in_a : in_b, have_in);
      if (fp32) {
        const int c8 = 4 * (ph & 1) + 2 * gi;  // 16-byte chunk within the 32-column box
        *reinterpret_cast<float4*>(my_row + ((c8 ^ sw) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(my_row + (((c8 + 1) ^ sw) << 4)) = make_float4(v[4], v[5], v[6], v[7]);
      } else if (two_out) {
        const int c4 = 2 * (ph & 1) + gi;
        *reinterpret_cast<uint4*>(row_pre + ((c4 ^ sw64) << 4)) = pack8_bf16(pre);
        *reinterpret_cast<uint4*>(row_fin + ((c4 ^ sw64) << 4)) = pack8_bf16(v);
      } else {
        *reinterpret_cast<uint4*>(my_row + (((2 * ph + gi) ^ sw) << 4)) = pack8_bf16(v);
      }
    }
    in_a = nx_a;
    in_b = nx_b;
    if (ph == 3 || (half_boxes && ph == 1)) {
      const int cbox = half_boxes ? col0 + 32 * (ph >> 1) : col0;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && cbox < w.N) {
        if (fp32 && g.accumulate) {
          tma_reduce_add_2d(tm_c, cbox, row0, box);
        } else {
          tma_store_2d(tm_c, cbox, row0, box);
          if (two_out) tma_store_2d(tm_c2, cbox, row0, box + 2048);
        }
        tma_store_commit();
      }
      if (FULL && g.colsum && ph == 3) epilogue_column_sums(box, min(32, w.M - row0), col0 + 2 * lane, w.N, g.colsum, lane);
    }
  }
}

// ---- the epilogues that the layers use, each in a form of its own -------------------------------------------------------------------
// epilogue_rows_tma asks in every group of 8 columns what there is to do, and the 16 warps of a CTA issue all of that: 600 to 840 cycles per
// phase of 16 columns where the plain form needs about 250 (6912 x 512 x 512: 2.9 us between the last product of a tile and its last store, now
// 1.2). KIND is chosen by the launcher (epilogue_kind); whatever has no form of its own takes epilogue_rows_tma or epilogue_columns.
// All: output through bulk tensor stores, n a multiple of 8, fp32 bias on a 16-byte boundary or none.
enum EpiKind {
  kEpiSome,      // without activation gradient, dropout, residual: any of the rest
  kEpiAny,       // anything
  kEpiPlain,     // bf16: [bias], [activation]
  kEpiF32,       // fp32, stored or added
  kEpiTwo,       // pre-activation and activation
  kEpiTwoDrop,   // ... with dropout on the second
  kEpiResid,     // residual + res_scale * (value [+ bias])
  kEpiResidDrop, // ... with dropout on the value
  kEpiDact,      // value * act'(z), column sums where wanted
  kEpiDactDrop   // ... with dropout
};
constexpr bool epi_generic(int kind) { return kind == kEpiSome || kind == kEpiAny; }
constexpr bool epi_drops(int kind) { return kind == kEpiTwoDrop || kind == kEpiResidDrop || kind == kEpiDactDrop; }
constexpr bool epi_has_input(int kind) { return kind == kEpiResid || kind == kEpiResidDrop || kind == kEpiDact || kind == kEpiDactDrop; }

inline int epilogue_kind(const Params& p) {
  const RbGemm& g = p.g;
  const bool full = g.dact_z != nullptr || g.drop_p > 0.f || g.resid != nullptr;
  const int generic = full ? kEpiAny : kEpiSome;
  if (!p.tma_store || g.n % 8 || (g.bias && !p.bias_vec)) return generic;
  const bool drop = g.drop_p > 0.f;
  // (sums that are added onto a matrix beyond the L2 leave in boxes of whole lines: 8000 x 8000 x 1000 170 us in the narrow boxes of kEpiF32, 157 in those;
  // 6000 x 8000 x 512 95.7 / 93.7, 4096 x 8000 x 512 64.0 / 64.1; stores are faster in the narrow ones throughout)
  const bool large_sum = g.accumulate && (long long)g.m * g.n >= 40000000;
  if (g.out_fp32) return full || g.bias || g.act || g.c2 || large_sum ? generic : kEpiF32;
  if (g.dact_z) return g.resid || g.bias || g.c2 ? generic : drop ? kEpiDactDrop : kEpiDact;
  if (g.resid) return g.act || g.c2 || g.colsum ? generic : drop ? kEpiResidDrop : kEpiResid;
  if (g.c2) return drop ? kEpiTwoDrop : kEpiTwo;
  return drop ? generic : kEpiPlain;
}

// the generator's key and first counter of a product, read once per warp
struct EpiRng {
  uint2 key;
  uint64_t base;
  uint32_t thresh;
  float scale;
  template <int KIND>
  __device__ __forceinline__ static EpiRng load(const RbGemm& g) {
    EpiRng r = {};
    if constexpr (epi_drops(KIND)) {
      const uint64_t sd = (uint64_t)g.seed[0];
      r.key = make_uint2((uint32_t)sd, (uint32_t)(sd >> 32));
      r.base = (uint64_t)g.offset[0] + g.drop_site;
      r.thresh = rb_dropout_thresh16(g.drop_p);
      r.scale = 1.f / (1.f - g.drop_p);
    }
    return r;
  }
};

// Arguments as epilogue_rows_tma. fp32 outputs leave in boxes of 32 rows x 16 columns, two of them in turn in the warp's 4 KB: a bulk add
// takes about 2000 cycles to read its box, and with one box of 32 columns the second half of a tile waited for that.
template <int KIND, typename Arrive>
__device__ __forceinline__ void epilogue_kind_tma(const Params& p, const Unit& w, int m0, int n0, uint32_t t_addr, int c_begin, uint8_t* box,
                                                  const CUtensorMap* tm_c, const CUtensorMap* tm_c2, int lane, int q, Arrive arrive, uint4 in_a, uint4 in_b,
                                                  const EpiRng& rng) {
  constexpr bool F32 = KIND == kEpiF32, TWO = KIND == kEpiTwo || KIND == kEpiTwoDrop, DROP = epi_drops(KIND), INPUT = epi_has_input(KIND);
  constexpr bool DACT = KIND == kEpiDact || KIND == kEpiDactDrop, RESID = INPUT && !DACT;
  const RbGemm& g = p.g;
  const int row0 = m0 + q * 32;
  const int row = row0 + lane;
  const int col0 = n0 + c_begin;
  auto release = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) arrive();
  };
  if (row0 >= w.M || col0 >= w.N) {  // nothing of this warp's box lies inside the matrix (warp-uniform): nothing to read
    release();
    return;
  }
  const int sw = lane & 7, sw64 = (lane >> 1) & 3;
  const float alpha = g.alpha;
  const float* bias = F32 || DACT ? nullptr : reinterpret_cast<const float*>(g.bias);
#pragma unroll 1
  for (int ph = 0; ph < 4; ++ph) {
    const int col = col0 + 16 * ph;
    uint32_t r[16];
    tmem_ld16(t_addr + (uint32_t)(c_begin + 16 * ph), r);
    uint4 nx_a = make_uint4(0u, 0u, 0u, 0u), nx_b = nx_a;
    if (INPUT && ph < 3) epilogue_prefetch16(p, w.M, w.N, row, col + 16, nx_a, nx_b);
    float4 b[4];
    if (bias) {
#pragma unroll
      for (int i = 0; i < 4; ++i) b[i] = col + 8 * (i >> 1) < w.N ? __ldg(reinterpret_cast<const float4*>(bias + col) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (ph == 3) release();
    if (F32 || ph == 0 || (TWO && ph == 2)) {  // the box was handed to the TMA unit before: it must have been read
      if (lane == 0) {
        if (F32) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        else tma_store_wait_read();
      }
      __syncwarp();
    }
#pragma unroll
    for (int gi = 0; gi < 2; ++gi) {
      float v[8], pre[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * gi + i]) * alpha;
      if (bias) {
        const float4 b0 = b[2 * gi], b1 = b[2 * gi + 1];
        v[0] += b0.x; v[1] += b0.y; v[2] += b0.z; v[3] += b0.w;
        v[4] += b1.x; v[5] += b1.y; v[6] += b1.z; v[7] += b1.w;
      }
      if constexpr (TWO) {
#pragma unroll
        for (int i = 0; i < 8; ++i) pre[i] = v[i];
      }
      if constexpr (DACT) {
        float z[8];
        unpack8_bf16(gi == 0 ? in_a : in_b, z);
        act_grad8(v, z, g.act);
      } else if constexpr (TWO || KIND == kEpiPlain) {
        if (g.act) act8(v, g.act);
      }
      if constexpr (DROP) rb_dropout_apply8(rng.key, rng.base + (uint64_t)((size_t)row * g.ldc + col + 8 * gi), rng.thresh, rng.scale, v);
      if constexpr (RESID) {
        float rs[8];
        unpack8_bf16(gi == 0 ? in_a : in_b, rs);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = rs[i] + g.res_scale * v[i];
      }
      if constexpr (F32) {
        uint8_t* at = box + (ph & 1) * 2048 + lane * 64;
        *reinterpret_cast<float4*>(at + (((2 * gi) ^ sw64) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(at + (((2 * gi + 1) ^ sw64) << 4)) = make_float4(v[4], v[5], v[6], v[7]);
      } else if constexpr (TWO) {
        uint8_t* at = box + lane * 64 + (((2 * (ph & 1) + gi) ^ sw64) << 4);
        *reinterpret_cast<uint4*>(at) = pack8_bf16(pre);
        *reinterpret_cast<uint4*>(at + 2048) = pack8_bf16(v);
      } else {
        *reinterpret_cast<uint4*>(box + lane * 128 + (((2 * ph + gi) ^ sw) << 4)) = pack8_bf16(v);
      }
    }
    if constexpr (INPUT) {
      in_a = nx_a;
      in_b = nx_b;
    }
    if (F32 || ph == 3 || (TWO && ph == 1)) {
      const int cbox = F32 ? col : TWO ? col0 + 32 * (ph >> 1) : col0;
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (cbox < w.N) {
          const uint8_t* from = F32 ? box + (ph & 1) * 2048 : box;
          if (F32 && g.accumulate) tma_reduce_add_2d(tm_c, cbox, row0, from);
          else tma_store_2d(tm_c, cbox, F32 ? w.c_r0 + row0 : row0, from);
          if (TWO) tma_store_2d(tm_c2, cbox, row0, box + 2048);
        }
        tma_store_commit();
      }
    }
  }
  if constexpr (DACT) {
    if (g.colsum) epilogue_column_sums(box, min(32, w.M - row0), col0 + 2 * lane, w.N, g.colsum, lane);
  }
}

// One warp's 32 rows x 64 columns [c_begin, c_begin + 64) of a problem that owns whole rows of the output (c_rows > 0): alpha only, bf16, in one box of
// 4 KB (rows of 128 bytes, 128-byte swizzle) and one bulk store. c_row: row of the output matrix that the problem's row 0 is. Attention scores are
// products over one block of 64: the epilogue is all of their time. The accumulator is given back as soon as it is in registers, and the box is
// waited for only when the next unit's values are there: with two boxes of half the width, one staging area and a wait in between, the scores of
// 36 x 333 frames with 8 heads took 23 us, now 16.7.
template <typename Arrive>
__device__ __forceinline__ void epilogue_boxes(const Params& p, const Unit& w, int c_row, uint32_t t_addr, int c_begin, uint8_t* box, const CUtensorMap* tm_c,
                                               int lane, int q, Arrive arrive) {
  const int row0 = w.m0 + q * 32, col0 = w.n0 + c_begin;
  auto release = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) arrive();
  };
  if (row0 >= w.M || col0 >= w.N) {
    release();
    return;
  }
  uint32_t r[64];
  tmem_ld32(t_addr + (uint32_t)c_begin, r);
  tmem_ld32(t_addr + (uint32_t)c_begin + 32, r + 32);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  release();
  if (lane == 0) tma_store_wait_read();
  __syncwarp();
#pragma unroll
  for (int gi = 0; gi < 8; ++gi) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * gi + i]) * p.g.alpha;
    *reinterpret_cast<uint4*>(box + lane * 128 + ((gi ^ (lane & 7)) << 4)) = pack8_bf16(v);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_2d(tm_c, col0, c_row + row0, box);
    tma_store_commit();
  }
}

constexpr int kEpilogueWarps = 16;                        // four per TMEM lane quarter: each takes a quarter of the tile's columns
constexpr int kGemmThreads = 64 + kEpilogueWarps * 32;    // + TMA producer warp + MMA warp
constexpr int kStagingBytesPerWarp = 32 * 16 * 4;
constexpr int kStoreBoxBytesPerWarp = 32 * 128;           // row-owner epilogue: one box of 32 rows x 128 bytes per warp

}  // namespace rbg

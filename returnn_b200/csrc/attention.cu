// Relative-position self-attention on packed sequences: the non-GEMM stages.
//
// The contraction stages (Qu·K^T, Qv·P^T, W·V and the six backward products) run on the batched tcgen05 GEMM
// (gemm_tcgen05.cu) over zero-padded per-sequence buffers; the kernels here do the rest:
//   att_prepare      packed qkv [N, H*3*D] -> padded Qu = q+u, Qv = q+v, K, V  [B*Lp, H*D], zeros in the padding
//   att_softmax_fwd  scores = S_ac[i,j] + G[i, j-i+center] (the Transformer-XL shift as an index), masked softmax over the
//                    valid keys, dropout with a replayable counter-based RNG; writes probabilities W and dropped Wd
//   att_softmax_bwd  dS = W * (dW - delta) with the exact delta = sum_j W*dW, and dG = the un-shifted dS
//   att_pack_dqkv    padded dQu+dQv, dK, dV -> packed dqkv [N, H*3*D], and their column sums
// Row length (keys per query) is limited to 512: one warp holds a row in registers.
#include "common.cuh"

namespace {

__device__ __forceinline__ float score_f(float x) { return x; }
__device__ __forceinline__ float score_f(__nv_bfloat16 x) { return __bfloat162float(x); }

constexpr int kMaxPerLane = 16;  // 32 lanes * 16 = 512 keys

// First packed row of sequence b (the sequences lie back to back): the sum of the lengths before it, by every warp for itself.
__device__ __forceinline__ int seq_start(const int* __restrict__ lens, int b) {
  int s = 0;
  for (int i = threadIdx.x & 31; i < b; i += 32) s += lens[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The two kernels that fill padded buffers write the padding too: fills of the buffers in front of them took as long as the copies (17 us for
// the 85 MB of a batch of 36 x 333 frames with 8 heads, 13 us for 42 MB). A CTA owns kPadRows padded rows of one sequence, so that a full batch is
// one wave of CTAs, and a thread has four 16-byte loads in flight (one item per thread and ten thousand CTAs: 28 us, now 23).
constexpr int kPadRows = 16;
constexpr int kPadLoads = 4;

// A thread keeps 8 columns of a row of qkv (one of q/k/v of one head) and goes down the rows, so that the position biases are read once: with items in
// the order of memory every item of q read 16 numbers of them, 32 bytes apart from lane to lane. 8 heads of 64, 36 sequences, 7865 of 12024 rows:
// 23.1 -> 15.2 us (out of DRAM 26.8 -> 20.4), all 12024 rows 24.8 -> 17.4, 4 x 50 rows 7.7 -> 5.0. 32 rows to a CTA: 17.6, 18.2 and 8.2 us.
__global__ void __launch_bounds__(256)
att_prepare_kernel(const __nv_bfloat16* __restrict__ qkv, const float* __restrict__ u, const float* __restrict__ v,
                   const int* __restrict__ lens, __nv_bfloat16* __restrict__ qu, __nv_bfloat16* __restrict__ qv, __nv_bfloat16* __restrict__ kk,
                   __nv_bfloat16* __restrict__ vv, int heads, int dim, int lp, int ctas) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const int b = blockIdx.x / ctas;
  const int row0 = (blockIdx.x - b * ctas) * kPadRows;
  const int hd = heads * dim;
  const int rows = min(kPadRows, lp - row0), valid = min(rows, lens[b] - row0);
  const __nv_bfloat16* src = qkv + ((long long)seq_start(lens, b) + row0) * 3 * hd;
  const long long dst0 = ((long long)b * lp + row0) * hd;
  for (int g = threadIdx.x; g < 3 * hd / 8; g += blockDim.x) {
    const int h = g * 8 / (3 * dim), in_head = g * 8 - h * 3 * dim, part = in_head / dim;
    const int c0 = h * dim + in_head - part * dim;
    const __nv_bfloat16* from = src + g * 8;
    float bu[8], bv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      bu[i] = part == 0 && u ? u[c0 + i] : 0.f;
      bv[i] = part == 0 && v ? v[c0 + i] : 0.f;
    }
    __nv_bfloat16* to = (part == 0 ? qu : part == 1 ? kk : vv) + dst0 + c0;
    __nv_bfloat16* to_v = qv + dst0 + c0;
    for (int r0 = 0; r0 < rows; r0 += kPadLoads) {
      uint4 raw[kPadLoads];
#pragma unroll
      for (int k = 0; k < kPadLoads; ++k) {
        raw[k] = make_uint4(0u, 0u, 0u, 0u);
        if (r0 + k < valid) raw[k] = *reinterpret_cast<const uint4*>(from + (long long)(r0 + k) * 3 * hd);
      }
#pragma unroll
      for (int k = 0; k < kPadLoads; ++k) {
        if (r0 + k >= rows) break;
        const long long at = (long long)(r0 + k) * hd;
        if (part == 0) {
          const bool in = r0 + k < valid;
          F8 a, c;
          const F8 x = load8(&raw[k], 0, 1);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            a.v[i] = in ? x.v[i] + bu[i] : 0.f;
            c.v[i] = in ? x.v[i] + bv[i] : 0.f;
          }
          store8(to, at, a, 1);
          store8(to_v, at, c, 1);
        } else {
          *reinterpret_cast<uint4*>(to + at) = raw[k];
        }
      }
    }
  }
}

// rows [N, width] packed -> [B*Lp, width], zeros in the padding
__global__ void __launch_bounds__(256)
att_rows_pad_kernel(const __nv_bfloat16* __restrict__ src, __nv_bfloat16* __restrict__ dst, const int* __restrict__ lens, int width, int lp, int ctas) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const int b = blockIdx.x / ctas;
  const int row0 = (blockIdx.x - b * ctas) * kPadRows;
  const __nv_bfloat16* from = src + ((long long)seq_start(lens, b) + row0) * width;
  __nv_bfloat16* to = dst + ((long long)b * lp + row0) * width;
  const uint32_t items = min(kPadRows, lp - row0) * (width / 8);
  const uint32_t valid = max(0, min(kPadRows, lens[b] - row0)) * (width / 8);  // rows lie one after the other on both sides
  for (uint32_t it0 = threadIdx.x; it0 < items; it0 += kPadLoads * 256) {
    uint4 raw[kPadLoads];
#pragma unroll
    for (int k = 0; k < kPadLoads; ++k) {
      const uint32_t it = it0 + k * 256;
      raw[k] = make_uint4(0u, 0u, 0u, 0u);
      if (it < valid) raw[k] = *reinterpret_cast<const uint4*>(from + (long long)it * 8);
    }
#pragma unroll
    for (int k = 0; k < kPadLoads; ++k) {
      const uint32_t it = it0 + k * 256;
      if (it < items) *reinterpret_cast<uint4*>(to + (long long)it * 8) = raw[k];
    }
  }
}

__device__ __forceinline__ uint32_t rng_u32(uint64_t seed, uint64_t idx) {
  uint4 r = philox4x32(make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)), make_uint4((uint32_t)(idx >> 2), (uint32_t)(idx >> 34), 0x51u, 0u));
  const uint32_t sel = (uint32_t)(idx & 3);
  return sel == 0 ? r.x : sel == 1 ? r.y : sel == 2 ? r.z : r.w;
}

// grid: (ceil(Lp / warps_per_cta), B*H); one warp per query row
template <typename TS>
__global__ void __launch_bounds__(128)
att_softmax_fwd_kernel(const TS* __restrict__ s_ac, const TS* __restrict__ g, __nv_bfloat16* __restrict__ w,
                       __nv_bfloat16* __restrict__ wd, const int* __restrict__ lens, int batch, int heads, int lp, int rp, int center,
                       float p_drop, const long long* __restrict__ seed, const long long* __restrict__ offset) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int z = blockIdx.y;
  const int b = z / heads, h = z % heads;
  const int len = lens[b];
  // the GEMMs that consume w / wd contract over rows or columns up to the next multiple of 64: that margin is zeroed here,
  // nothing beyond it is ever read, so the buffers need no memset
  const int len64 = min(lp, (len + 63) & ~63);
  if (i >= len64) return;
  const long long srow = ((long long)z * lp + i) * lp;
  if (i >= len) {
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int j = lane; j < len64; j += 32) {
      w[srow + j] = zero;
      if (p_drop > 0.f) wd[srow + j] = zero;
    }
    return;
  }
  const long long grow = (((long long)h * batch + b) * lp + i) * rp;
  float x[kMaxPerLane];
  float mx = -INFINITY;
#pragma unroll
  for (int t = 0; t < kMaxPerLane; ++t) {
    const int j = lane + 32 * t;
    if (j < len) {
      x[t] = score_f(s_ac[srow + j]) + score_f(g[grow + (j - i + center)]);
      mx = fmaxf(mx, x[t]);
    } else {
      x[t] = -INFINITY;
    }
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int t = 0; t < kMaxPerLane; ++t) {
    x[t] = (lane + 32 * t < len) ? __expf(x[t] - mx) : 0.f;
    sum += x[t];
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  const bool drop = p_drop > 0.f;
  const uint64_t sd = drop ? (uint64_t)seed[0] : 0;
  const uint64_t off = drop ? (uint64_t)offset[0] : 0;
  const uint32_t thresh = drop ? (uint32_t)(p_drop * 4294967296.0) : 0u;
  const float keep_scale = drop ? 1.f / (1.f - p_drop) : 1.f;
#pragma unroll
  for (int t = 0; t < kMaxPerLane; ++t) {
    const int j = lane + 32 * t;
    if (j < len64) {
      const float pr = j < len ? x[t] * inv : 0.f;
      w[srow + j] = __float2bfloat16(pr);
      if (drop) {
        const bool keep = rng_u32(sd, off + (uint64_t)(srow + j)) >= thresh;
        wd[srow + j] = __float2bfloat16(keep ? pr * keep_scale : 0.f);
      }
    }
  }
}

template <typename TS>
__global__ void __launch_bounds__(128)
att_softmax_bwd_kernel(const __nv_bfloat16* __restrict__ w, const TS* __restrict__ dwd, __nv_bfloat16* __restrict__ ds,
                       __nv_bfloat16* __restrict__ dg, const int* __restrict__ lens, int batch, int heads, int lp, int rp, int center,
                       float p_drop, const long long* __restrict__ seed, const long long* __restrict__ offset) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int z = blockIdx.y;
  const int b = z / heads, h = z % heads;
  const int len = lens[b];
  const int len64 = min(lp, (len + 63) & ~63);  // see the forward kernel
  if (i >= len64) return;
  const long long srow = ((long long)z * lp + i) * lp;
  if (i >= len) {
    for (int j = lane; j < len64; j += 32) ds[srow + j] = __float2bfloat16(0.f);
    return;
  }
  const long long grow = (((long long)h * batch + b) * lp + i) * rp;
  const bool drop = p_drop > 0.f;
  const uint64_t sd = drop ? (uint64_t)seed[0] : 0;
  const uint64_t off = drop ? (uint64_t)offset[0] : 0;
  const uint32_t thresh = drop ? (uint32_t)(p_drop * 4294967296.0) : 0u;
  const float keep_scale = drop ? 1.f / (1.f - p_drop) : 1.f;
  float pw[kMaxPerLane], dw[kMaxPerLane];
  float delta = 0.f;
#pragma unroll
  for (int t = 0; t < kMaxPerLane; ++t) {
    const int j = lane + 32 * t;
    if (j < len) {
      pw[t] = __bfloat162float(w[srow + j]);
      float d = score_f(dwd[srow + j]);
      if (drop) d = (rng_u32(sd, off + (uint64_t)(srow + j)) >= thresh) ? d * keep_scale : 0.f;
      dw[t] = d;
      delta += pw[t] * d;
    } else {
      pw[t] = 0.f;
      dw[t] = 0.f;
    }
  }
  delta = warp_sum(delta);
#pragma unroll
  for (int t = 0; t < kMaxPerLane; ++t) {
    const int j = lane + 32 * t;
    if (j < len) {
      const __nv_bfloat16 o = __float2bfloat16(pw[t] * (dw[t] - delta));
      ds[srow + j] = o;
      dg[grow + (j - i + center)] = o;
    } else if (j < len64) {
      ds[srow + j] = __float2bfloat16(0.f);
    }
  }
}

// ---- bf16-score versions with 16-byte accesses: a lane owns 8 consecutive keys per step (two steps cover 512 keys), one
// philox call serves 4 keys (the scalar kernels above draw one per key and use a quarter of it). Same arithmetic, same dropout
// counters, so forward and backward (and the scalar kernels) agree on the mask.
__device__ __forceinline__ void rng8(uint64_t seed, uint64_t idx0, uint32_t (&r)[8]) {
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const uint64_t b0 = idx0 >> 2;  // idx0 is a multiple of 8
  const uint4 a = philox4x32(key, make_uint4((uint32_t)b0, (uint32_t)(b0 >> 32), 0x51u, 0u));
  const uint4 b = philox4x32(key, make_uint4((uint32_t)(b0 + 1), (uint32_t)((b0 + 1) >> 32), 0x51u, 0u));
  r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w; r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 p = __bfloat1622float2(h[q]);
    f[2 * q] = p.x;
    f[2 * q + 1] = p.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
  return u;
}

constexpr int kVecSteps = 2;  // 2 * 32 lanes * 8 keys = 512

__global__ void __launch_bounds__(128)
att_softmax_fwd_vec_kernel(const __nv_bfloat16* __restrict__ s_ac, const __nv_bfloat16* __restrict__ g, __nv_bfloat16* __restrict__ w,
                           __nv_bfloat16* __restrict__ wd, const int* __restrict__ lens, int batch, int heads, int lp, int rp, int center,
                           float p_drop, const long long* __restrict__ seed, const long long* __restrict__ offset) {
  rb_pdl_wait();
  rb_pdl_launch();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int z = blockIdx.y;
  const int b = z / heads, h = z % heads;
  const int len = lens[b];
  const int len64 = min(lp, (len + 63) & ~63);
  if (i >= len64) return;
  const long long srow = ((long long)z * lp + i) * lp;
  const bool drop = p_drop > 0.f;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  if (i >= len) {
    for (int j0 = lane * 8; j0 < len64; j0 += 256) {
      *reinterpret_cast<uint4*>(w + srow + j0) = zero4;
      if (drop) *reinterpret_cast<uint4*>(wd + srow + j0) = zero4;
    }
    return;
  }
  const long long grow = (((long long)h * batch + b) * lp + i) * rp + (center - i);
  float x[kVecSteps][8];
  float mx = -INFINITY;
#pragma unroll
  for (int t = 0; t < kVecSteps; ++t) {
    const int j0 = (t * 32 + lane) * 8;
    if (j0 < len) {
      float a[8];
      unpack8(*reinterpret_cast<const uint4*>(s_ac + srow + j0), a);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int j = j0 + e;
        x[t][e] = j < len ? a[e] + __bfloat162float(g[grow + j]) : -INFINITY;
        mx = fmaxf(mx, x[t][e]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[t][e] = -INFINITY;
    }
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int t = 0; t < kVecSteps; ++t)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      x[t][e] = x[t][e] > -INFINITY ? __expf(x[t][e] - mx) : 0.f;
      sum += x[t][e];
    }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
  const uint64_t sd = drop ? (uint64_t)seed[0] : 0;
  const uint64_t off = drop ? (uint64_t)offset[0] : 0;
  const uint32_t thresh = drop ? (uint32_t)(p_drop * 4294967296.0) : 0u;
  const float keep_scale = drop ? 1.f / (1.f - p_drop) : 1.f;
#pragma unroll
  for (int t = 0; t < kVecSteps; ++t) {
    const int j0 = (t * 32 + lane) * 8;
    if (j0 < len64) {
      float pr[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) pr[e] = x[t][e] * inv;  // zero beyond len
      *reinterpret_cast<uint4*>(w + srow + j0) = pack8(pr);
      if (drop) {
        uint32_t r[8];
        rng8(sd, off + (uint64_t)(srow + j0), r);
#pragma unroll
        for (int e = 0; e < 8; ++e) pr[e] = r[e] >= thresh ? pr[e] * keep_scale : 0.f;
        *reinterpret_cast<uint4*>(wd + srow + j0) = pack8(pr);
      }
    }
  }
}

__global__ void __launch_bounds__(128)
att_softmax_bwd_vec_kernel(const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ dwd, __nv_bfloat16* __restrict__ ds,
                           __nv_bfloat16* __restrict__ dg, const int* __restrict__ lens, int batch, int heads, int lp, int rp, int center,
                           float p_drop, const long long* __restrict__ seed, const long long* __restrict__ offset) {
  rb_pdl_wait();
  rb_pdl_launch();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int z = blockIdx.y;
  const int b = z / heads, h = z % heads;
  const int len = lens[b];
  const int len64 = min(lp, (len + 63) & ~63);
  if (i >= len64) return;
  const long long srow = ((long long)z * lp + i) * lp;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  if (i >= len) {
    for (int j0 = lane * 8; j0 < len64; j0 += 256) *reinterpret_cast<uint4*>(ds + srow + j0) = zero4;
    return;
  }
  const long long grow = (((long long)h * batch + b) * lp + i) * rp + (center - i);
  const bool drop = p_drop > 0.f;
  const uint64_t sd = drop ? (uint64_t)seed[0] : 0;
  const uint64_t off = drop ? (uint64_t)offset[0] : 0;
  const uint32_t thresh = drop ? (uint32_t)(p_drop * 4294967296.0) : 0u;
  const float keep_scale = drop ? 1.f / (1.f - p_drop) : 1.f;
  float pw[kVecSteps][8], dw[kVecSteps][8];
  float delta = 0.f;
#pragma unroll
  for (int t = 0; t < kVecSteps; ++t) {
    const int j0 = (t * 32 + lane) * 8;
    if (j0 < len) {
      unpack8(*reinterpret_cast<const uint4*>(w + srow + j0), pw[t]);
      unpack8(*reinterpret_cast<const uint4*>(dwd + srow + j0), dw[t]);
      uint32_t r[8];
      if (drop) rng8(sd, off + (uint64_t)(srow + j0), r);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (j0 + e >= len) {
          pw[t][e] = 0.f;
          dw[t][e] = 0.f;
        } else if (drop) {
          dw[t][e] = r[e] >= thresh ? dw[t][e] * keep_scale : 0.f;
        }
        delta += pw[t][e] * dw[t][e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) pw[t][e] = dw[t][e] = 0.f;
    }
  }
  delta = warp_sum(delta);
#pragma unroll
  for (int t = 0; t < kVecSteps; ++t) {
    const int j0 = (t * 32 + lane) * 8;
    if (j0 < len64) {
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = pw[t][e] * (dw[t][e] - delta);  // zero beyond len
      const uint4 packed = pack8(o);
      *reinterpret_cast<uint4*>(ds + srow + j0) = packed;
      const __nv_bfloat16* ob = reinterpret_cast<const __nv_bfloat16*>(&packed);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (j0 + e < len) dg[grow + j0 + e] = ob[e];
    }
  }
}

// wd = dropout(w) with the mask of the forward pass (same seed, same offset)
__global__ void __launch_bounds__(128)
att_redrop_kernel(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wd, const int* __restrict__ lens, int heads, int lp,
                  float p_drop, const long long* __restrict__ seed, const long long* __restrict__ offset) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int z = blockIdx.y;
  const int len = lens[z / heads];
  if (i >= len) return;
  const long long srow = ((long long)z * lp + i) * lp;
  const uint64_t sd = (uint64_t)seed[0], off = (uint64_t)offset[0];
  const uint32_t thresh = (uint32_t)(p_drop * 4294967296.0);
  const float keep_scale = 1.f / (1.f - p_drop);
  for (int j = lane; j < len; j += 32) {
    const bool keep = rng_u32(sd, off + (uint64_t)(srow + j)) >= thresh;
    wd[srow + j] = __float2bfloat16(keep ? __bfloat162float(w[srow + j]) * keep_scale : 0.f);
  }
}

// Padded dQu + dQv, dK, dV -> packed dqkv, with the column sums of what passes through: of dqkv (bias gradient of the projection), of dQu and
// dQv (gradients of the position biases). A CTA owns 64 columns of dqkv, 8 threads to a row, and a slice of the rows; each thread has the
// loads of two rows in flight. As a copy (15.6 us at 6740 x 1536) and three column-sum kernels (27 us) the gradients were read twice.
// ATOMIC: the sums are added to; else every slice leaves its own in sum_u / sum_v ([slices][2 * heads * dim], sum_v = sum_u + heads * dim).
// WHOLE: dim is a multiple of 64, so the CTA's columns are of one head and one part; else of 8, and a thread's columns are.
template <bool ATOMIC, bool WHOLE>
__global__ void __launch_bounds__(256)
att_pack_dqkv_kernel(const __nv_bfloat16* __restrict__ dqu, const __nv_bfloat16* __restrict__ dqv, const __nv_bfloat16* __restrict__ dk,
                     const __nv_bfloat16* __restrict__ dv, const int* __restrict__ row_batch, const int* __restrict__ row_pos,
                     __nv_bfloat16* __restrict__ dqkv, float* __restrict__ sum_qkv, float* __restrict__ sum_u, float* __restrict__ sum_v, int n_rows,
                     int heads, int dim, int lp, int rows_per_cta) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  __shared__ float red[32][65];
  const int lane8 = (threadIdx.x & 7) * 8, rl = threadIdx.x >> 3;
  const int hd = heads * dim;
  const int col0 = blockIdx.y * 64, col = col0 + lane8;  // of dqkv
  const int first = WHOLE ? col0 : col;
  const int h = first / (3 * dim);
  const int part = (first - h * 3 * dim) / dim;
  const int src_col = h * dim + (col - (h * 3 + part) * dim);
  const __nv_bfloat16* a_src = (part == 0 ? dqu : part == 1 ? dk : dv) + src_col;
  const __nv_bfloat16* b_src = dqv + src_col;
  const int r_end = WHOLE || col < 3 * hd ? min(n_rows, (int)(blockIdx.x + 1) * rows_per_cta) : 0;
  float s_x[8], s_u[8], s_v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s_x[i] = s_u[i] = s_v[i] = 0.f;
  for (int r0 = blockIdx.x * rows_per_cta + rl; r0 < r_end; r0 += 64) {
    uint4 a[2], c[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int r = r0 + 32 * k;
      if (r < r_end) {
        const long long at = ((long long)row_batch[r] * lp + row_pos[r]) * hd;
        a[k] = *reinterpret_cast<const uint4*>(a_src + at);
        if (part == 0) c[k] = *reinterpret_cast<const uint4*>(b_src + at);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int r = r0 + 32 * k;
      if (r >= r_end) break;
      F8 x = load8(&a[k], 0, 1);
      if (part == 0) {
        const F8 y = load8(&c[k], 0, 1);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          s_u[i] += x.v[i];
          s_v[i] += y.v[i];
          x.v[i] = __bfloat162float(__float2bfloat16(x.v[i] + y.v[i]));
        }
      }
      store8(dqkv, (long long)r * 3 * hd + col, x, 1);
#pragma unroll
      for (int i = 0; i < 8; ++i) s_x[i] += x.v[i];
    }
  }
  auto leave = [&](const float* s, float* dst, bool queries) {  // dst: of all columns of dqkv, or of those of the queries
    if (dst == nullptr) return;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) red[rl][lane8 + i] = s[i];
    __syncthreads();
    const int at = col0 + threadIdx.x, head = WHOLE ? h : at / (3 * dim), in_head = at - head * 3 * dim;
    if (threadIdx.x < 64 && (WHOLE || (at < 3 * hd && (!queries || in_head < dim)))) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < 32; ++k) t += red[k][threadIdx.x];
      dst += queries ? head * dim + in_head : at;
      if (ATOMIC) atomicAdd(dst, t);
      else *dst = t;
    }
  };
  leave(s_x, sum_qkv, false);
  if (WHOLE ? part == 0 : col0 % (3 * dim) < dim || col0 % (3 * dim) + 63 >= 3 * dim) {  // some of the 64 columns are a query's
    const long long slice = ATOMIC ? 0 : (long long)blockIdx.x * 2 * hd;
    leave(s_u, sum_u ? sum_u + slice : nullptr, true);
    leave(s_v, sum_v ? sum_v + slice : nullptr, true);
  }
}

// rows [B*Lp, HD] padded -> packed [N, HD]; F32: the source rows are fp32
template <typename I, bool F32>  // index type: 32 bits where the groups fit (the division is a large part of these copies)
__global__ void __launch_bounds__(256)
att_rows_gather_kernel(const void* __restrict__ src, __nv_bfloat16* __restrict__ dst, const int* __restrict__ row_batch,
                       const int* __restrict__ row_pos, int n_rows, int width, int lp) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const int groups = width / 8;
  const I gid = (I)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (I)n_rows * (I)groups) return;
  const int row = (int)(gid / (I)groups);
  const int c0 = (int)(gid % (I)groups) * 8;
  const long long padded = ((long long)row_batch[row] * lp + row_pos[row]) * width + c0;
  store8(dst, (long long)row * width + c0, load8(src, padded, !F32), 1);
}

}  // namespace

// CTAs per sequence of lp rows; 0: more than a launch holds
static int ctas_per_seq(int batch, int lp) {
  const long long n = (lp + kPadRows - 1) / kPadRows;
  return n * batch < (1LL << 31) ? (int)n : 0;
}

// packed qkv [N, H*3*D] -> qu = q + u, qv = q + v, k, v [B*Lp, H*D]; lens (device) of the sequences, back to back in qkv
RB_EXPORT int rb200_att_prepare(const void* qkv, const float* u, const float* v, const int* lens, void* qu, void* qv, void* k, void* vv, int batch,
                                int heads, int dim, int lp, cudaStream_t stream) {
  if (batch <= 0 || lp <= 0) return RB_OK;
  const int ctas = dim % 8 ? 0 : ctas_per_seq(batch, lp);
  if (!ctas) {
    rb_set_error("att_prepare: head dim %d must be a multiple of 8, batch %d x %d rows fit a launch", dim, batch, lp);
    return RB_ERR_ARG;
  }
  // as many threads as share the groups of 8 columns evenly
  const int groups = 3 * heads * dim / 8, passes = (groups + 255) / 256, threads = ((groups + passes - 1) / passes + 31) / 32 * 32;
  rb_launch_pdl(att_prepare_kernel, dim3((unsigned)ctas * batch), dim3(threads), 0, stream, (const __nv_bfloat16*)qkv, u, v, lens, (__nv_bfloat16*)qu,
                (__nv_bfloat16*)qv, (__nv_bfloat16*)k, (__nv_bfloat16*)vv, heads, dim, lp, ctas);
  return rb_check_launch("att_prepare");
}

// scores_bf16: s_ac and g are bf16 (what the batched GEMMs write on the training path) instead of fp32
RB_EXPORT int rb200_att_softmax_fwd_ex(const void* s_ac, const void* g, int scores_bf16, void* w, void* wd, const int* lens, int batch, int heads,
                                       int lp, int rp, int center, float p_drop, const long long* seed, const long long* offset, cudaStream_t stream) {
  if (lp > 32 * kMaxPerLane) {
    rb_set_error("att_softmax: padded length %d > %d", lp, 32 * kMaxPerLane);
    return RB_ERR_UNSUPPORTED;
  }
  dim3 grid((lp + 3) / 4, batch * heads);
  if (scores_bf16 && lp <= 512 && lp % 64 == 0 && rp % 8 == 0)
    rb_launch_pdl(att_softmax_fwd_vec_kernel, grid, dim3(128), 0, stream, (const __nv_bfloat16*)s_ac, (const __nv_bfloat16*)g, (__nv_bfloat16*)w,
                  (__nv_bfloat16*)wd, lens, batch, heads, lp, rp, center, p_drop, seed, offset);
  else if (scores_bf16)
    rb_launch_pdl(att_softmax_fwd_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, stream, (const __nv_bfloat16*)s_ac, (const __nv_bfloat16*)g, (__nv_bfloat16*)w,
                                                                    (__nv_bfloat16*)wd, lens, batch, heads, lp, rp, center, p_drop, seed, offset);
  else
  rb_launch_pdl(att_softmax_fwd_kernel<float>, dim3(grid), dim3(128), 0, stream, (const float*)s_ac, (const float*)g, (__nv_bfloat16*)w, (__nv_bfloat16*)wd, lens, batch, heads, lp, rp, center, p_drop,
                                                   seed, offset);
  return rb_check_launch("att_softmax_fwd");
}

RB_EXPORT int rb200_att_softmax_bwd_ex(const void* w, const void* dwd, int dwd_bf16, void* ds, void* dg, const int* lens, int batch, int heads, int lp,
                                       int rp, int center, float p_drop, const long long* seed, const long long* offset, cudaStream_t stream) {
  if (lp > 32 * kMaxPerLane) return RB_ERR_UNSUPPORTED;
  dim3 grid((lp + 3) / 4, batch * heads);
  if (dwd_bf16 && lp <= 512 && lp % 64 == 0 && rp % 8 == 0)
    rb_launch_pdl(att_softmax_bwd_vec_kernel, grid, dim3(128), 0, stream, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dwd, (__nv_bfloat16*)ds,
                  (__nv_bfloat16*)dg, lens, batch, heads, lp, rp, center, p_drop, seed, offset);
  else if (dwd_bf16)
    rb_launch_pdl(att_softmax_bwd_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, stream, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dwd, (__nv_bfloat16*)ds,
                                                                    (__nv_bfloat16*)dg, lens, batch, heads, lp, rp, center, p_drop, seed, offset);
  else
    rb_launch_pdl(att_softmax_bwd_kernel<float>, dim3(grid), dim3(128), 0, stream, (const __nv_bfloat16*)w, (const float*)dwd, (__nv_bfloat16*)ds, (__nv_bfloat16*)dg, lens,
                                                            batch, heads, lp, rp, center, p_drop, seed, offset);
  return rb_check_launch("att_softmax_bwd");
}

RB_EXPORT int rb200_att_softmax_fwd(const float* s_ac, const float* g, void* w, void* wd, const int* lens, int batch, int heads, int lp, int rp,
                                    int center, float p_drop, const long long* seed, const long long* offset, cudaStream_t stream) {
  return rb200_att_softmax_fwd_ex(s_ac, g, 0, w, wd, lens, batch, heads, lp, rp, center, p_drop, seed, offset, stream);
}

RB_EXPORT int rb200_att_softmax_bwd(const void* w, const float* dwd, void* ds, void* dg, const int* lens, int batch, int heads, int lp, int rp,
                                    int center, float p_drop, const long long* seed, const long long* offset, cudaStream_t stream) {
  return rb200_att_softmax_bwd_ex(w, dwd, 0, ds, dg, lens, batch, heads, lp, rp, center, p_drop, seed, offset, stream);
}

RB_EXPORT int rb200_att_redrop(const void* w, void* wd, const int* lens, int batch, int heads, int lp, float p_drop, const long long* seed,
                               const long long* offset, cudaStream_t stream) {
  dim3 grid((lp + 3) / 4, batch * heads);
  att_redrop_kernel<<<grid, 128, 0, stream>>>((const __nv_bfloat16*)w, (__nv_bfloat16*)wd, lens, heads, lp, p_drop, seed, offset);
  return rb_check_launch("att_redrop");
}

// rows of a slice: about three CTAs per SM, each with at least 64 rows
static int pack_rows_per_cta(int n_rows, int chunks) {
  int slices = (3 * 148 + chunks - 1) / chunks;
  if (slices > (n_rows + 63) / 64) slices = (n_rows + 63) / 64;
  return (n_rows + slices - 1) / slices;
}
RB_EXPORT int rb200_att_pack_slices(int n_rows, int heads, int dim) {
  if (n_rows <= 0) return 0;
  const int per = pack_rows_per_cta(n_rows, (3 * heads * dim + 63) / 64);
  return (n_rows + per - 1) / per;
}

// sums (fp32, each may be null): with accumulate added to: sum_qkv [3 * heads * dim], sum_u and sum_v [heads * dim]; else sum_u
// [rb200_att_pack_slices][2][heads * dim] receives the sums of dqu and dqv by slices of the rows (sum_qkv and sum_v null)
RB_EXPORT int rb200_att_pack_dqkv(const void* dqu, const void* dqv, const void* dk, const void* dv, const int* row_batch, const int* row_pos,
                                  void* dqkv, float* sum_qkv, float* sum_u, float* sum_v, int n_rows, int heads, int dim, int lp, int accumulate,
                                  cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (dim % 8 || dim <= 0 || heads <= 0 || 3LL * heads * dim / 64 >= 65535) {
    rb_set_error("att_pack_dqkv: head dim %d must be a multiple of 8 (%d heads)", dim, heads);
    return RB_ERR_ARG;
  }
  const int chunks = (3 * heads * dim + 63) / 64, per = pack_rows_per_cta(n_rows, chunks);
  if (!accumulate) sum_v = sum_u ? sum_u + (long long)heads * dim : nullptr;
  auto kernel = dim % 64 ? (accumulate ? att_pack_dqkv_kernel<true, false> : att_pack_dqkv_kernel<false, false>)
                         : (accumulate ? att_pack_dqkv_kernel<true, true> : att_pack_dqkv_kernel<false, true>);
  rb_launch_pdl(kernel, dim3((n_rows + per - 1) / per, chunks), dim3(256), 0, stream,
                (const __nv_bfloat16*)dqu, (const __nv_bfloat16*)dqv, (const __nv_bfloat16*)dk, (const __nv_bfloat16*)dv, row_batch, row_pos,
                (__nv_bfloat16*)dqkv, accumulate ? sum_qkv : nullptr, sum_u, sum_v, n_rows, heads, dim, lp, per);
  return rb_check_launch("att_pack_dqkv");
}

// bf16 rows [B*Lp, width] -> packed [N, width]
RB_EXPORT int rb200_att_rows_gather(const void* src, void* dst, const int* row_batch, const int* row_pos, int n_rows, int width, int lp, cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (width % 8) return RB_ERR_ARG;
  long long total = (long long)n_rows * (width / 8);
  rb_launch_pdl(total < (1LL << 31) ? att_rows_gather_kernel<uint32_t, false> : att_rows_gather_kernel<unsigned long long, false>,
                dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, src, (__nv_bfloat16*)dst, row_batch, row_pos, n_rows, width, lp);
  return rb_check_launch("att_rows_gather");
}

// packed bf16 rows [N, width] -> [B*Lp, width], zeros in the padding
RB_EXPORT int rb200_att_rows_pad(const void* src, void* dst, const int* lens, int batch, int width, int lp, cudaStream_t stream) {
  if (batch <= 0 || lp <= 0) return RB_OK;
  const int ctas = width % 8 ? 0 : ctas_per_seq(batch, lp);
  if (!ctas) {
    rb_set_error("att_rows_pad: width %d must be a multiple of 8, batch %d x %d rows fit a launch", width, batch, lp);
    return RB_ERR_ARG;
  }
  rb_launch_pdl(att_rows_pad_kernel, dim3((unsigned)ctas * batch), dim3(256), 0, stream, (const __nv_bfloat16*)src, (__nv_bfloat16*)dst, lens, width, lp, ctas);
  return rb_check_launch("att_rows_pad");
}

// padded fp32 rows -> packed bf16 rows
RB_EXPORT int rb200_att_rows_gather_f32(const float* src, void* dst, const int* row_batch, const int* row_pos, int n_rows, int width, int lp,
                                        cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (width % 8) return RB_ERR_ARG;
  long long total = (long long)n_rows * (width / 8);
  rb_launch_pdl(total < (1LL << 31) ? att_rows_gather_kernel<uint32_t, true> : att_rows_gather_kernel<unsigned long long, true>,
                dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, (const void*)src, (__nv_bfloat16*)dst, row_batch, row_pos, n_rows, width, lp);
  return rb_check_launch("att_rows_gather_f32");
}

// Conformer convolution module core on packed rows: GLU -> depthwise conv along time -> BatchNorm (statistics over the
// valid frames) -> SiLU, forward and backward.
//
// x [N, 2C] bf16 (output of the first pointwise GEMM), packed rows of B sequences (row_batch / row_pos / lens give the
// sequence, position and length of each row). Depthwise filter [C, K] taps, "same" padding with (K-1)/2 taps to the
// left, zero outside each sequence.
//
//   forward   glu_dwconv_fwd : h = a * sigmoid(g); y[r,c] = bias[c] + sum_k f[c,k] * h[r+k-left, c]
//             bn_part        : partial sums of y and y^2 per channel (scratch; more than 32 taps: in the kernel above)
//             bn_stats       : partials -> mean, rstd (and running statistics)
//             bn_silu_fwd    : z = silu((y - mean) * rstd * gamma + beta)
//   backward  bn_silu_bwd_a  : ds = dz * silu'(s); per-CTA partial sums of ds and ds * yhat
//             bn_bwd_reduce  : partials -> dgamma, dbeta (and the two means used below)
//             bn_silu_bwd_b  : dy = gamma * rstd * (ds - mean(ds) - yhat * mean(ds * yhat))
//             glu_dwconv_bwd : dh[r,c] = sum_k f[c,k] * dy[r-k+left, c]; dx = (dh * sigmoid(g), dh * a * sigmoid'(g));
//                              per-CTA partial sums for dfilter [C,K] and dbias
// All reductions go through per-CTA partials and a second pass: no atomics, deterministic.
#include <type_traits>
#include "common.cuh"

namespace {

constexpr int TT = 32;       // output rows per CTA
constexpr int CC = 64;       // channels per CTA
constexpr int KMAX = 64;     // maximum number of taps
constexpr int kThreads = 256;  // 64 channels x 4 row groups of 8 rows

__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + __expf(-x)); }

// ---------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
glu_dwconv_fwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ filt, const float* __restrict__ bias,
                      const int* __restrict__ row_batch, const int* __restrict__ row_pos, const int* __restrict__ lens,
                      __nv_bfloat16* __restrict__ y, float* __restrict__ part, int n_rows, int C, int K) {
  __shared__ float sh[(TT + KMAX - 1) * CC];
  __shared__ float red[2][4][CC];
  const int left = (K - 1) / 2;
  const int r0 = blockIdx.x * TT;
  const int c0 = blockIdx.y * CC;
  const int n_in = TT + K - 1;
  // stage h = a * sigmoid(g) for rows r0-left .. r0-left+n_in-1
  for (int idx = threadIdx.x; idx < n_in * CC; idx += kThreads) {
    const int s = idx / CC, c = idx % CC;
    const int r = r0 - left + s;
    float h = 0.f;
    if (r >= 0 && r < n_rows) {
      const float a = __bfloat162float(x[(size_t)r * 2 * C + c0 + c]);
      const float g = __bfloat162float(x[(size_t)r * 2 * C + C + c0 + c]);
      h = a * sigmoidf_(g);
    }
    sh[s * CC + c] = h;
  }
  __syncthreads();
  const int c = threadIdx.x % CC;
  const int rg = threadIdx.x / CC;
  float f[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; ++k) f[k] = k < K ? filt[(size_t)(c0 + c) * K + k] : 0.f;
  const float bv = bias ? bias[c0 + c] : 0.f;
  float s1 = 0.f, s2 = 0.f;
  for (int i = 0; i < TT / 4; ++i) {
    const int lr = rg * (TT / 4) + i;
    const int r = r0 + lr;
    if (r >= n_rows) break;
    const int t = row_pos[r];
    const int L = lens[row_batch[r]];
    const int k_lo = max(0, left - t);
    const int k_hi = min(K, L - t + left);
    float acc = bv;
#pragma unroll
    for (int k = 0; k < KMAX; ++k) {
      if (k >= k_lo && k < k_hi) acc += f[k] * sh[(lr + k) * CC + c];
    }
    const __nv_bfloat16 o = __float2bfloat16(acc);
    y[(size_t)r * C + c0 + c] = o;
    const float of = __bfloat162float(o);
    s1 += of;
    s2 += of * of;
  }
  red[0][rg][c] = s1;
  red[1][rg][c] = s2;
  __syncthreads();
  if (threadIdx.x < CC) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      a += red[0][g][threadIdx.x];
      b += red[1][g][threadIdx.x];
    }
    part[((size_t)blockIdx.x * 2 + 0) * C + c0 + threadIdx.x] = a;
    part[((size_t)blockIdx.x * 2 + 1) * C + c0 + threadIdx.x] = b;
  }
}

// eight bf16 values as they stand in memory (4 registers while they are in flight, 8 as floats)
__device__ __forceinline__ uint4 load_raw8(const __nv_bfloat16* __restrict__ p, int64_t at, bool on) {
  return on ? *reinterpret_cast<const uint4*>(p + at) : make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ F8 raw_to_f8(uint4 u) {
  F8 r;
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    r.v[2 * i] = f.x;
    r.v[2 * i + 1] = f.y;
  }
  return r;
}
// The eight channels of a thread: per-channel constants as two 16-byte loads each where the pointer allows them
__device__ __forceinline__ void load_chan8(const float* __restrict__ p, int c, float none, float (&v)[8]) {
  if (p == nullptr) {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = none;
  } else if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 a = *reinterpret_cast<const float4*>(p + c), b = *reinterpret_cast<const float4*>(p + c + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = p[c + k];
  }
}

// Rows of 8-channel groups: a thread keeps its channels and their constants (the grid is a whole number of rows) and takes every
// grid-th row, kRowsInFlight loads at a time. With the constants read once per group of eight values (40 scalar loads for two 16-byte
// ones) these kernels were bound by the L1: 22 (forward) and 28 us (backward, second pass) for 7900 x 512 in a pass, now 8 and 6.5.
constexpr int kRowsInFlight = 4;
__host__ __device__ inline int rows_grid(long long total8, int groups) {
  int a = groups, b = 256;  // CTAs in multiples of groups / gcd(groups, 256): grid * 256 threads are whole rows
  while (b) {
    const int t = a % b;
    a = b;
    b = t;
  }
  const long long unit = groups / a;
  long long want = (total8 + 256LL * kRowsInFlight - 1) / (256LL * kRowsInFlight);
  want = want < 148 * 6 ? want : 148 * 6;
  return (int)((want + unit - 1) / unit * unit);
}

__global__ void __launch_bounds__(256, 3)
bn_silu_fwd_kernel(const __nv_bfloat16* __restrict__ y, const float* __restrict__ mean, const float* __restrict__ rstd,
                   const float* __restrict__ gamma, const float* __restrict__ beta, __nv_bfloat16* __restrict__ z, long long total, int C) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8, stride = (long long)gridDim.x * blockDim.x * 8;
  const int c = (int)(first % C);
  float mu[8], rs[8], ga[8], be[8];
  load_chan8(mean, c, 0.f, mu);
  load_chan8(rstd, c, 1.f, rs);
  load_chan8(gamma, c, 1.f, ga);
  load_chan8(beta, c, 0.f, be);
  for (long long i0 = first; i0 < total; i0 += stride * kRowsInFlight) {
    uint4 raw[kRowsInFlight];
#pragma unroll
    for (int j = 0; j < kRowsInFlight; ++j) raw[j] = load_raw8(y, i0 + j * stride, i0 + j * stride < total);
#pragma unroll
    for (int j = 0; j < kRowsInFlight; ++j) {
      if (i0 + j * stride >= total) break;
      F8 v = raw_to_f8(raw[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float s = (v.v[k] - mu[k]) * rs[k] * ga[k] + be[k];
        v.v[k] = s * sigmoidf_(s);
      }
      store8(z, i0 + j * stride, v, 1);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// ds = dz * silu'(s) written to ds_out (bf16); per-CTA partials of sum(ds) and sum(ds*yhat) per channel.
// grid.x tiles of rows_per_cta rows; a thread handles 8 channels of one row at a time.
__global__ void __launch_bounds__(256, 2)
bn_silu_bwd_a_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ dz, const float* __restrict__ mean,
                     const float* __restrict__ rstd, const float* __restrict__ gamma, const float* __restrict__ beta,
                     __nv_bfloat16* __restrict__ ds_out, float* __restrict__ part, int n_rows, int C, int rows_per_cta) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  // threads: C/8 column groups x (256 / (C/8)) row lanes; requires C/8 <= 256 and 256 % (C/8) == 0
  extern __shared__ __align__(16) float shm[];  // [row_lanes][2][C]
  const int groups = C / 8;
  const int row_lanes = blockDim.x / groups;
  const int cg = threadIdx.x % groups;
  const int rl = threadIdx.x / groups;
  const int c = cg * 8;
  float a1[8], a2[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a1[k] = a2[k] = 0.f;
  const int r_begin = blockIdx.x * rows_per_cta;
  const int r_end = min(n_rows, r_begin + rows_per_cta);
  if (rl < row_lanes) {
    // per-channel constants once; then four rows per step with all of their loads issued before the first use (a thread owns few
    // rows: their load latency is the cost of this kernel)
    float mu[8], rs[8], ga[8], be[8];
    load_chan8(mean, c, 0.f, mu);
    load_chan8(rstd, c, 1.f, rs);
    load_chan8(gamma, c, 1.f, ga);
    load_chan8(beta, c, 0.f, be);
    for (int r0 = r_begin + rl; r0 < r_end; r0 += 4 * row_lanes) {
      uint4 yr[4], dr[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + j * row_lanes;
        yr[j] = load_raw8(y, (long long)r * C + c, r < r_end);
        dr[j] = load_raw8(dz, (long long)r * C + c, r < r_end);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + j * row_lanes;
        if (r < r_end) {
          const F8 yv = raw_to_f8(yr[j]), dv = raw_to_f8(dr[j]);
          F8 o;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float yh = (yv.v[k] - mu[k]) * rs[k];
            const float s = yh * ga[k] + be[k];
            const float sg = sigmoidf_(s);
            const float d = dv.v[k] * (sg * (1.f + s * (1.f - sg)));
            o.v[k] = d;
            a1[k] += d;
            a2[k] += d * yh;
          }
          store8(ds_out, (long long)r * C + c, o, 1);
        }
      }
    }
    float4* o1 = reinterpret_cast<float4*>(shm + (rl * 2 + 0) * C + c);
    float4* o2 = reinterpret_cast<float4*>(shm + (rl * 2 + 1) * C + c);
    o1[0] = make_float4(a1[0], a1[1], a1[2], a1[3]);
    o1[1] = make_float4(a1[4], a1[5], a1[6], a1[7]);
    o2[0] = make_float4(a2[0], a2[1], a2[2], a2[3]);
    o2[1] = make_float4(a2[4], a2[5], a2[6], a2[7]);
  }
  __syncthreads();
  for (int cc = threadIdx.x; cc < C; cc += blockDim.x) {
    float s1 = 0.f, s2 = 0.f;
    for (int l = 0; l < row_lanes; ++l) {
      s1 += shm[(l * 2 + 0) * C + cc];
      s2 += shm[(l * 2 + 1) * C + cc];
    }
    part[((size_t)blockIdx.x * 2 + 0) * C + cc] = s1;
    part[((size_t)blockIdx.x * 2 + 1) * C + cc] = s2;
  }
}

// dy = gamma * rstd * (ds - sum_ds/count - yhat * sum_ds_yh/count), in place over ds
__global__ void __launch_bounds__(256, 2)
bn_silu_bwd_b_kernel(const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ ds, const float* __restrict__ mean,
                     const float* __restrict__ rstd, const float* __restrict__ gamma, const float* __restrict__ sum_ds,
                     const float* __restrict__ sum_ds_yh, float inv_count, long long total, int C) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8, stride = (long long)gridDim.x * blockDim.x * 8;
  const int c = (int)(first % C);
  float mu[8], rs[8], ga[8], m1[8], m2[8];
  load_chan8(mean, c, 0.f, mu);
  load_chan8(rstd, c, 1.f, rs);
  load_chan8(gamma, c, 1.f, ga);
  load_chan8(sum_ds, c, 0.f, m1);
  load_chan8(sum_ds_yh, c, 0.f, m2);
  for (long long i0 = first; i0 < total; i0 += stride * kRowsInFlight) {
    uint4 yr[kRowsInFlight], dr[kRowsInFlight];
#pragma unroll
    for (int j = 0; j < kRowsInFlight; ++j) {
      yr[j] = load_raw8(y, i0 + j * stride, i0 + j * stride < total);
      dr[j] = load_raw8(ds, i0 + j * stride, i0 + j * stride < total);
    }
#pragma unroll
    for (int j = 0; j < kRowsInFlight; ++j) {
      if (i0 + j * stride >= total) break;
      const F8 yv = raw_to_f8(yr[j]);
      F8 dv = raw_to_f8(dr[j]);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float yh = (yv.v[k] - mu[k]) * rs[k];
        dv.v[k] = ga[k] * rs[k] * (dv.v[k] - m1[k] * inv_count - yh * m2[k] * inv_count);
      }
      store8(ds, i0 + j * stride, dv, 1);
    }
  }
}

// depthwise conv backward + GLU backward. Each CTA owns CC channels and walks over row tiles (tile = blockIdx.x, += gridDim.x),
// keeping its dfilter / dbias sums in registers; one partial per CTA at the end: part layout [gridDim.x][C][K+1].
template <int KM>
__global__ void __launch_bounds__(kThreads)
glu_dwconv_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const float* __restrict__ filt,
                      const int* __restrict__ row_batch, const int* __restrict__ row_pos, const int* __restrict__ lens,
                      __nv_bfloat16* __restrict__ dx, float* __restrict__ part, int n_rows, int C, int K) {
  __shared__ float sh_dy[(TT + KM - 1) * CC];   // dy rows r0-(K-1-left) .. : used for dh
  __shared__ float sh_h[(TT + KM - 1) * CC];    // h rows r0-left .. : used for dfilter
  __shared__ int sh_t[TT], sh_len[TT];
  const int left = (K - 1) / 2;
  const int right = K - 1 - left;
  const int c0 = blockIdx.y * CC;
  const int n_in = TT + K - 1;
  const int n_tiles = (n_rows + TT - 1) / TT;
  const int c = threadIdx.x % CC;
  const int rg = threadIdx.x / CC;
  float f[KM];
#pragma unroll
  for (int k = 0; k < KM; ++k) f[k] = k < K ? filt[(size_t)(c0 + c) * K + k] : 0.f;
  float df[KM];
#pragma unroll
  for (int k = 0; k < KM; ++k) df[k] = 0.f;
  float dbias = 0.f;
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int r0 = tile * TT;
    __syncthreads();  // the previous tile's readers are done with the shared arrays
    // stage dy and h = a * sigmoid(g), 8 channels per thread-iteration
    for (int idx = threadIdx.x; idx < n_in * (CC / 8); idx += kThreads) {
      const int s = idx / (CC / 8), cg = (idx % (CC / 8)) * 8;
      // dh[r] = sum_k f[k] * dy[r - k + left]  ->  needs dy rows r0 - right .. r0 + TT - 1 + left
      const int rd = r0 - right + s;
      F8 d;
      if (rd >= 0 && rd < n_rows) d = load8(dy, (int64_t)rd * C + c0 + cg, 1);
      else {
#pragma unroll
        for (int i = 0; i < 8; ++i) d.v[i] = 0.f;
      }
      const int rh = r0 - left + s;
      F8 h;
      if (rh >= 0 && rh < n_rows) {
        F8 a = load8(x, (int64_t)rh * 2 * C + c0 + cg, 1);
        F8 g = load8(x, (int64_t)rh * 2 * C + C + c0 + cg, 1);
#pragma unroll
        for (int i = 0; i < 8; ++i) h.v[i] = a.v[i] * sigmoidf_(g.v[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) h.v[i] = 0.f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sh_dy[s * CC + cg + i] = d.v[i];
        sh_h[s * CC + cg + i] = h.v[i];
      }
    }
    if (threadIdx.x < TT) {
      const int r = r0 + threadIdx.x;
      sh_t[threadIdx.x] = r < n_rows ? row_pos[r] : 0;
      sh_len[threadIdx.x] = r < n_rows ? lens[row_batch[r]] : 0;
    }
    __syncthreads();
    for (int i = 0; i < TT / 4; ++i) {
      const int lr = rg * (TT / 4) + i;
      const int r = r0 + lr;
      if (r >= n_rows) break;
      const int t = sh_t[lr];
      const int L = sh_len[lr];
      // dh: contributions from output rows r' = r - k + left (position t - k + left) that lie inside the sequence
      float dh = 0.f;
#pragma unroll
      for (int k = 0; k < KM; ++k) {
        const int tp = t - k + left;
        if (k < K && tp >= 0 && tp < L) dh += f[k] * sh_dy[(lr + right - k + left) * CC + c];
      }
      // a and g of this row: h = a * sig(g) is staged at row lr + left; recover a, g from global (coalesced over c)
      const float a = __bfloat162float(x[(size_t)r * 2 * C + c0 + c]);
      const float g = __bfloat162float(x[(size_t)r * 2 * C + C + c0 + c]);
      const float sg = sigmoidf_(g);
      dx[(size_t)r * 2 * C + c0 + c] = __float2bfloat16(dh * sg);
      dx[(size_t)r * 2 * C + C + c0 + c] = __float2bfloat16(dh * a * sg * (1.f - sg));
      // dfilter[k] += dy[r] * h[r + k - left] for taps inside the sequence
      const float dyr = sh_dy[(lr + right) * CC + c];
      dbias += dyr;
      const int k_lo = max(0, left - t);
      const int k_hi = min(K, L - t + left);
#pragma unroll
      for (int k = 0; k < KM; ++k) {
        if (k >= k_lo && k < k_hi) df[k] += dyr * sh_h[(lr + k) * CC + c];
      }
    }
  }
  // reduce the 4 row groups through shared memory (reuse sh_h as [K+1][CC] accumulators), then one partial per CTA
  __syncthreads();
  float* red = sh_h;
  for (int g = 0; g < 4; ++g) {
    if (rg == g) {
#pragma unroll
      for (int k = 0; k < KM; ++k)
        if (k < K) red[k * CC + c] = (g == 0 ? 0.f : red[k * CC + c]) + df[k];
      red[K * CC + c] = (g == 0 ? 0.f : red[K * CC + c]) + dbias;
    }
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < (K + 1) * CC; idx += kThreads) {
    const int k = idx / CC, cc = idx % CC;
    part[((size_t)blockIdx.x * C + c0 + cc) * (K + 1) + k] = red[k * CC + cc];
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Sliding-window versions for K <= 32 taps. A thread owns one channel and kRpt consecutive output rows: it walks once over
// the kRpt + KT - 1 staged rows of its window, and every staged value feeds up to kRpt accumulators through compile-time filter
// indices, so the filter and the accumulators stay in registers and each staged value is read from shared memory once
// (the kernels above read one value per tap and output).
//
// The rows are those of a wider layout: packed row r of sequence b stands at r + (KT - 1) b, and the KT - 1 rows between two sequences are
// zeros, so that no window needs a mask or sees another sequence, not even with the zeros that fill up its taps (with windows over the packed rows, a sequence boundary cost the five row groups around it three
// instructions for one product or a second pass, and the rest of the CTA waited). The price is KT - 1 rows of staging per sequence; groups
// of kRpt rows that hold no packed row are skipped. A CTA owns CC channels and walks over a piece of the rows in steps of kStep: the staged
// rows stand in a ring, a step brings in the kStep rows that the one before has not seen, and their loads are in flight during the products
// of that one. (A CTA per 64 rows that stages, synchronises, multiplies and stores: every chain of latencies stands alone.) 7900 x 512 in 36
// sequences, 32 taps: forward 28 -> 18 us, backward 47 -> 34; the products alone are 3 and 6 at full rate, 41 % of the issue slots are used.
constexpr int KM2 = 32;         // most taps (filters with fewer taps are zero-padded to 16 or 32)
constexpr int kRpt = 8;         // rows per thread
constexpr int kStep = 32;       // output rows per step: 64 channels x 4 row groups in 256 threads
constexpr int kHalo = 32;       // staged rows in front of the first step's new ones
constexpr int kRing = 64;       // staged rows held: the kHalo + kStep of a step
constexpr int kPieceMax = 2048; // rows of the wider layout per CTA
constexpr int kMap = kPieceMax + kHalo + kStep + 2;
constexpr int kWinThreads = 256;
constexpr int kFiltPitch = KM2 + 1;

// row j of the window that starts at staged row `at` (a multiple of 8, OFF = at & 8): ring[base[(j + OFF) >> 4] + ((j + OFF) & 15) * CC]
struct Window {
  int base[3];
};
__device__ __forceinline__ Window window_at(int at, int c) {
  Window w;
#pragma unroll
  for (int t = 0; t < 3; ++t) w.base[t] = (((at >> 4) + t) & (kRing / 16 - 1)) * 16 * CC + c;
  return w;
}
template <int OFF>
__device__ __forceinline__ float window_row(const float* ring, const Window& w, int j) {
  return ring[w.base[(j + OFF) >> 4] + ((j + OFF) & 15) * CC];
}

// acc[i] += sum_k w[k] row[i + k]
template <int KT, int OFF>
__device__ __forceinline__ void window_conv(const float* ring, const Window& col, const float (&w)[KT], float (&acc)[kRpt]) {
#pragma unroll
  for (int j = 0; j < kRpt + KT - 1; ++j) {
    const float v = window_row<OFF>(ring, col, j);
#pragma unroll
    for (int i = 0; i < kRpt; ++i)
      if (j - i >= 0 && j - i < KT) acc[i] = fmaf(w[j - i], v, acc[i]);
  }
}
// df[k] += sum_i d[i] row[i + k]
template <int KT, int OFF>
__device__ __forceinline__ void window_corr(const float* ring, const Window& col, const float (&d)[kRpt], float (&df)[KT]) {
#pragma unroll
  for (int j = 0; j < kRpt + KT - 1; ++j) {
    const float v = window_row<OFF>(ring, col, j);
#pragma unroll
    for (int i = 0; i < kRpt; ++i)
      if (j - i >= 0 && j - i < KT) df[j - i] = fmaf(d[i], v, df[j - i]);
  }
}

__device__ __forceinline__ void ring_store8(float* ring, int staged, int cg, const F8& h) {
  float4* dst = reinterpret_cast<float4*>(ring + (staged & (kRing - 1)) * CC + cg);
  dst[0] = make_float4(h.v[0], h.v[1], h.v[2], h.v[3]);
  dst[1] = make_float4(h.v[4], h.v[5], h.v[6], h.v[7]);
}

// The filters of the CTA's channels, [CC][K] contiguous in memory, into shared memory with an odd pitch. (Read from global memory by the
// thread that owns the channel, every load of a warp touches 32 lines: 32 taps took longer than the convolution of a 64-row tile.)
__device__ __forceinline__ void stage_filter(float* __restrict__ sf, const float* __restrict__ filt, int c0, int K) {
  int cc = threadIdx.x / K, k = threadIdx.x % K;
  const int dc = blockDim.x / K, dk = blockDim.x % K;
  for (int idx = threadIdx.x; idx < CC * K; idx += blockDim.x) {
    sf[cc * kFiltPitch + k] = filt[(size_t)c0 * K + idx];
    cc += dc;
    k += dk;
    if (k >= K) {
      k -= K;
      ++cc;
    }
  }
}

// map[i] = packed row at row first + i of the wider layout, -1 for the rows between sequences; i < n. Rows ascend in both layouts, the
// wider one adds `gap` per sequence: a look at every 32nd row that can lie in front of the piece finds where to start reading row_batch.
// Returns whether this thread has found a row of the piece.
__device__ __forceinline__ bool stage_map(int* __restrict__ map, int* __restrict__ start, const int* __restrict__ row_batch, int first, int n,
                                          int gap, int n_rows, int n_seqs) {
  const int lo = max(0, first - gap * (n_seqs - 1)), hi = min(n_rows, first);
  if (threadIdx.x == 0) *start = lo;
  for (int i = threadIdx.x; i < n; i += blockDim.x) map[i] = -1;
  __syncthreads();
  int at = lo;
  for (int r = lo + 32 * threadIdx.x; r < hi; r += 32 * blockDim.x)
    if (r + gap * row_batch[r] < first) at = r;
  if (at > lo) atomicMax(start, at);
  __syncthreads();
  bool any = false;
  for (int r = *start + threadIdx.x; r < n_rows; r += blockDim.x) {
    const int i = r + gap * row_batch[r] - first;
    if (i >= n) break;
    if (i >= 0) {
      map[i] = r;
      any = true;
    }
  }
  return any;
}

// pieces of the wider layout's rows, a whole number of row groups each: about `ctas` CTAs in all, at most one per 32 packed rows unless the map
// would not hold a piece. The rows of the wider layout grow with every sequence, empty ones too: with many of those there are more pieces than
// 32 packed rows, and the backward kernel's CTAs, `walkers` of them, take several (a partial sum each, in a scratch of one per 32 packed rows).
struct Pieces {
  int n, rows, walkers;
};
inline Pieces pieces_of(int n_rows, int n_seqs, int C, int K, int ctas) {
  const long long wide = n_rows + (long long)((K <= 16 ? 16 : KM2) - 1) * (n_seqs > 0 ? n_seqs - 1 : 0);
  long long most = ctas / (C / CC);
  if (most > (n_rows + 31) / 32) most = (n_rows + 31) / 32;
  if (most < 1) most = 1;
  long long rows = ((wide + most - 1) / most + kRpt - 1) / kRpt * kRpt;
  if (rows < kStep) rows = kStep;
  if (rows > kPieceMax) rows = kPieceMax;
  const long long n = (wide + rows - 1) / rows, slots = (n_rows + 31) / 32;
  return {(int)n, (int)rows, (int)(n < slots ? n : slots)};
}
constexpr int kFwdCtas = 3 * 148, kBwdCtas = 2 * 148;  // as many as are resident (80 and 128 registers)
constexpr size_t kFwd2Smem = (size_t)(kRing * CC + CC * kFiltPitch) * sizeof(float) + (kMap + 1) * sizeof(int);
constexpr size_t kBwd2Smem = (size_t)(3 * kRing * CC + CC * kFiltPitch) * sizeof(float) + (kMap + 1) * sizeof(int);

template <int KT>
__global__ void __launch_bounds__(kWinThreads, 3)
glu_dwconv_fwd2_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ filt, const float* __restrict__ bias,
                       const int* __restrict__ row_batch, __nv_bfloat16* __restrict__ y, int n_rows, int n_seqs, int C, int K, int piece) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  extern __shared__ __align__(16) float smem_f[];
  float* ring = smem_f;  // staged row i: GLU output of row begin - left + i
  float* sf = ring + kRing * CC;
  int* map = reinterpret_cast<int*>(sf + CC * kFiltPitch);  // of row begin - left + i
  const int tid = threadIdx.x;
  const int left = (K - 1) / 2;
  const int begin = blockIdx.x * piece;
  const int c0 = blockIdx.y * CC;
  const int cg = (tid & 7) * 8;
  stage_filter(sf, filt, c0, K);
  stage_map(map, map + kMap, row_batch, begin - left, piece + kHalo + kStep, KT - 1, n_rows, n_seqs);
  __syncthreads();
  uint4 pa, pg;
  auto fetch = [&](int staged) {  // rows staged .. staged + 31
    const int r = map[staged + (tid >> 3)];
    pa = load_raw8(x, (int64_t)r * 2 * C + c0 + cg, r >= 0);
    pg = load_raw8(x, (int64_t)r * 2 * C + C + c0 + cg, r >= 0);
  };
  auto place = [&](int staged) {
    F8 h = raw_to_f8(pa);
    const F8 g = raw_to_f8(pg);
#pragma unroll
    for (int i = 0; i < 8; ++i) h.v[i] *= sigmoidf_(g.v[i]);
    ring_store8(ring, staged + (tid >> 3), cg, h);
  };
  fetch(0);
  const int c = tid % CC;
  const int rg = tid / CC;
  float f[KT];
#pragma unroll
  for (int k = 0; k < KT; ++k) f[k] = k < K ? sf[c * kFiltPitch + k] : 0.f;
  const float bv = bias ? bias[c0 + c] : 0.f;
  place(0);
  fetch(kHalo);
  const int base = rg * kRpt;
  auto rows = [&](auto off, int at) {
    float acc[kRpt];
#pragma unroll
    for (int i = 0; i < kRpt; ++i) acc[i] = bv;
    window_conv<KT, decltype(off)::value>(ring, window_at(at, c), f, acc);
#pragma unroll
    for (int i = 0; i < kRpt; ++i) {
      const int r = map[at + left + i];
      if (r >= 0) y[(size_t)r * C + c0 + c] = __float2bfloat16(acc[i]);
    }
  };
  for (int step = 0; step * kStep < piece; ++step) {
    __syncthreads();  // the rows that are replaced have been read
    place(kHalo + step * kStep);
    if ((step + 1) * kStep < piece) fetch(kHalo + (step + 1) * kStep);
    __syncthreads();
    const int at = step * kStep + base;
    int any = -1;
#pragma unroll
    for (int i = 0; i < kRpt; ++i) any &= map[at + left + i];  // -1 where all are
    if (at >= piece || any == -1) continue;
    if (base & 8) rows(std::integral_constant<int, 8>(), at);
    else rows(std::integral_constant<int, 0>(), at);
  }
}

// part [ceil(N / 32)][2][C]: sums of y and y^2 per channel over 64 rows in every second slot, zeros in the others. A thread owns 8 channels
// of 16 rows, all of them in flight; four such groups are added in order. (Sums by the convolution over its own pieces of the rows would
// save a launch, but the statistics of a batch would then depend on how the rows were cut.)
constexpr int kPartRows = 64;
__global__ void __launch_bounds__(256)
bn_part_kernel(const __nv_bfloat16* __restrict__ y, float* __restrict__ part, int n_rows, int C) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  __shared__ float red[2][4][CC * 8];
  const int cl = threadIdx.x % CC, rg = threadIdx.x / CC;
  const int c = (blockIdx.y * CC + cl) * 8;
  const int r0 = blockIdx.x * kPartRows + rg * 16;
  float s1[8], s2[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) s1[k] = s2[k] = 0.f;
  if (c < C) {
    uint4 raw[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) raw[i] = load_raw8(y, (int64_t)(r0 + i) * C + c, r0 + i < n_rows);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (r0 + i >= n_rows) break;
      const F8 v = raw_to_f8(raw[i]);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s1[k] += v.v[k];
        s2[k] += v.v[k] * v.v[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    red[0][rg][k * CC + cl] = s1[k];
    red[1][rg][k * CC + cl] = s2[k];
  }
  __syncthreads();
  const int slot = blockIdx.x * (kPartRows / TT), n_slots = (n_rows + TT - 1) / TT;
  for (int i = threadIdx.x; i < 2 * CC * 8; i += blockDim.x) {
    const int which = i / (CC * 8), cc = i % (CC * 8), at = (cc & 7) * CC + (cc >> 3), ch = blockIdx.y * CC * 8 + cc;
    if (ch >= C) continue;
    float a = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) a += red[which][g][at];
    part[((size_t)slot * 2 + which) * C + ch] = a;
    if (slot + 1 < n_slots) part[((size_t)(slot + 1) * 2 + which) * C + ch] = 0.f;
  }
}

// dfilter / dbias sums stay in registers, over all pieces of a CTA; partial per CTA [gridDim.x][C][K+1]. MANY: more pieces than CTAs (the loop
// around a piece costs 2 % where there is but one)
template <int KT, bool MANY>
__global__ void __launch_bounds__(kWinThreads, 2)
glu_dwconv_bwd2_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const float* __restrict__ filt,
                       const int* __restrict__ row_batch, __nv_bfloat16* __restrict__ dx, float* __restrict__ part, int n_rows, int n_seqs, int C,
                       int K, int piece, int pieces) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  extern __shared__ __align__(16) float smem_f[];
  float* ring_dy = smem_f;                // staged row i: row begin - right + i
  float* ring_h = ring_dy + kRing * CC;   // staged row i: row begin - left + i
  float* ring_s = ring_h + kRing * CC;    // sigmoid of the gate of the same row
  float* sf = ring_s + kRing * CC;
  int* map = reinterpret_cast<int*>(sf + CC * kFiltPitch);  // of row begin - right + i
  const int tid = threadIdx.x;
  const int left = (K - 1) / 2;
  const int right = K - 1 - left;
  const int c0 = blockIdx.y * CC;
  const int cg = (tid & 7) * 8;
  int at_piece = blockIdx.x;
  auto piece_map = [&]() { return stage_map(map, map + kMap, row_batch, at_piece * piece - right, piece + kHalo + kStep + 1, KT - 1, n_rows, n_seqs); };
  stage_filter(sf, filt, c0, K);
  piece_map();
  __syncthreads();
  uint4 pd, pa, pg;
  auto fetch = [&](int staged) {  // rows staged .. staged + 31
    const int rd = map[staged + (tid >> 3)], rh = map[staged + (tid >> 3) + right - left];
    pd = load_raw8(dy, (int64_t)rd * C + c0 + cg, rd >= 0);
    pa = load_raw8(x, (int64_t)rh * 2 * C + c0 + cg, rh >= 0);
    pg = load_raw8(x, (int64_t)rh * 2 * C + C + c0 + cg, rh >= 0);
  };
  auto place = [&](int staged) {
    ring_store8(ring_dy, staged + (tid >> 3), cg, raw_to_f8(pd));
    F8 h = raw_to_f8(pa), s = raw_to_f8(pg);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      s.v[i] = sigmoidf_(s.v[i]);
      h.v[i] *= s.v[i];
    }
    ring_store8(ring_h, staged + (tid >> 3), cg, h);
    ring_store8(ring_s, staged + (tid >> 3), cg, s);
  };
  fetch(0);
  const int c = tid % CC;
  const int rg = tid / CC;
  float fr[KT];  // flipped filter: fr[m] = f[K-1-m]
#pragma unroll
  for (int m = 0; m < KT; ++m) fr[m] = m < K ? sf[c * kFiltPitch + (K - 1 - m)] : 0.f;
  float df[KT];
#pragma unroll
  for (int k = 0; k < KT; ++k) df[k] = 0.f;
  float dbias = 0.f;
  const int base = rg * kRpt;
  auto rows = [&](auto off, int at) {
    constexpr int OFF = decltype(off)::value;
    const Window col = window_at(at, c);
    float v[kRpt];
    // dh[r] = sum_k f[k] * dy[r - k + left]: staged index of that row is (r - begin) + (K-1) - k
#pragma unroll
    for (int i = 0; i < kRpt; ++i) v[i] = 0.f;
    window_conv<KT, OFF>(ring_dy, col, fr, v);
#pragma unroll
    for (int i = 0; i < kRpt; ++i) {
      const int r = map[at + right + i];
      if (r >= 0) {
        const int s = ((at + i + left) & (kRing - 1)) * CC + c;
        const float h = ring_h[s], sg = ring_s[s];
        __nv_bfloat16* o = dx + (size_t)r * 2 * C + c0 + c;
        o[0] = __float2bfloat16(v[i] * sg);
        o[C] = __float2bfloat16(v[i] * h * (1.f - sg));
      }
    }
    // dfilter[k] += dy[r] * h[r + k - left]: staged index of that h row is (r - begin) + k
#pragma unroll
    for (int i = 0; i < kRpt; ++i) dbias += v[i] = ring_dy[((at + i + right) & (kRing - 1)) * CC + c];
    window_corr<KT, OFF>(ring_h, col, v, df);
  };
  auto walk = [&]() {  // over the rows of the piece whose first ones have been fetched
    place(0);
    fetch(kHalo);
    for (int step = 0; step * kStep < piece; ++step) {
      __syncthreads();  // the rows that are replaced have been read
      place(kHalo + step * kStep);
      if ((step + 1) * kStep < piece) fetch(kHalo + (step + 1) * kStep);
      __syncthreads();
      const int at = step * kStep + base;
      int any = -1;
#pragma unroll
      for (int i = 0; i < kRpt; ++i) any &= map[at + right + i];  // -1 where all are
      if (at >= piece || any == -1) continue;
      if (base & 8) rows(std::integral_constant<int, 8>(), at);
      else rows(std::integral_constant<int, 0>(), at);
    }
  };
  walk();
  if (MANY) {
    for (at_piece += gridDim.x; at_piece < pieces; at_piece += gridDim.x) {
      __syncthreads();  // the map and the rows of the piece before have been read
      if (!__syncthreads_or(piece_map())) continue;  // empty sequences only
      fetch(0);
      walk();
    }
  }
  // sum the row groups in shared memory, one after the other (the same sum in every run), one partial per CTA
  float* red = ring_h;  // [KT + 1][CC]
  for (int g = 0; g < kWinThreads / CC; ++g) {
    __syncthreads();
    if (rg == g) {
#pragma unroll
      for (int k = 0; k < KT; ++k) red[k * CC + c] = g ? red[k * CC + c] + df[k] : df[k];
      red[KT * CC + c] = g ? red[KT * CC + c] + dbias : dbias;
    }
  }
  __syncthreads();
  for (int idx = tid; idx < (K + 1) * CC; idx += kWinThreads) {
    const int cc = idx / (K + 1), k = idx % (K + 1);
    part[((size_t)blockIdx.x * C + c0 + cc) * (K + 1) + k] = red[(k < K ? k : KT) * CC + cc];
  }
}

// Reductions of per-CTA partials with TL tile lanes per output and a shared-memory sum (coalesced over the outputs; one thread per output
// takes tens of microseconds for a few hundred tiles, 8 lanes 10 for 430).
template <int TL>
__device__ __forceinline__ float lane_sum(float s, float (*sh)[32], int tl, int lane) {
  sh[tl][lane] = s;
  __syncthreads();
  if (tl == 0) {
#pragma unroll
    for (int g = 1; g < TL; ++g) s += sh[g][lane];
  }
  __syncthreads();
  return s;
}

// part [n_tiles][C][K+1] -> dfilt [C][K], dbias [C]
__global__ void __launch_bounds__(256)
dwconv_bwd_reduce2_kernel(const float* __restrict__ part, int n_tiles, int C, int K, float* __restrict__ dfilt, float* __restrict__ dbias,
                          int accumulate) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  __shared__ float sh[8][32];
  const int lane = threadIdx.x % 32, tl = threadIdx.x / 32;
  const int idx = blockIdx.x * 32 + lane;
  const int n_out = C * (K + 1);
  float s = 0.f;
  if (idx < n_out)
    for (int t = tl; t < n_tiles; t += 8) s += part[(size_t)t * n_out + idx];
  s = lane_sum<8>(s, sh, tl, lane);
  if (tl == 0 && idx < n_out) {
    const int c = idx / (K + 1), k = idx % (K + 1);
    if (k < K) dfilt[(size_t)c * K + k] = accumulate ? dfilt[(size_t)c * K + k] + s : s;
    else if (dbias) dbias[c] = accumulate ? dbias[c] + s : s;
  }
}

// part [n_tiles][2][C] -> the two sums per channel (thread tl == 0 of each lane holds them)
template <int TL>
__device__ __forceinline__ void pair_sums(const float* __restrict__ part, int n_tiles, int C, int c, float (*sh)[32], int tl, int lane,
                                          float& s1, float& s2) {
  s1 = 0.f;
  s2 = 0.f;
  if (c < C) {
#pragma unroll 8
    for (int t = tl; t < n_tiles; t += TL) {
      s1 += part[((size_t)t * 2 + 0) * C + c];
      s2 += part[((size_t)t * 2 + 1) * C + c];
    }
  }
  s1 = lane_sum<TL>(s1, sh, tl, lane);
  s2 = lane_sum<TL>(s2, sh, tl, lane);
}

__global__ void __launch_bounds__(256)
bn_stats2_kernel(const float* __restrict__ part, int n_tiles, int C, float count, float eps, float momentum, float* __restrict__ mean,
                 float* __restrict__ rstd, float* __restrict__ running_mean, float* __restrict__ running_var) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  __shared__ float sh[8][32];
  const int lane = threadIdx.x % 32, tl = threadIdx.x / 32;
  const int c = blockIdx.x * 32 + lane;
  float s1, s2;
  pair_sums<8>(part, n_tiles, C, c, sh, tl, lane, s1, s2);
  if (tl == 0 && c < C) {
    const double m = (double)s1 / count;
    double var = (double)s2 / count - m * m;
    if (var < 0.0) var = 0.0;
    mean[c] = (float)m;
    rstd[c] = rsqrtf((float)var + eps);
    if (running_mean) {
      running_mean[c] += momentum * ((float)m - running_mean[c]);
      running_var[c] += momentum * ((float)var - running_var[c]);
    }
  }
}

__global__ void __launch_bounds__(1024)
bn_bwd_reduce2_kernel(const float* __restrict__ part, int n_tiles, int C, float* __restrict__ sum_ds, float* __restrict__ sum_ds_yh,
                      float* __restrict__ dgamma_acc, float* __restrict__ dbeta_acc) {
  rb_pdl_wait();  // may have been scheduled before the preceding kernel finished
  rb_pdl_launch();
  __shared__ float sh[32][32];
  const int lane = threadIdx.x % 32, tl = threadIdx.x / 32;
  const int c = blockIdx.x * 32 + lane;
  float s1, s2;
  pair_sums<32>(part, n_tiles, C, c, sh, tl, lane, s1, s2);
  if (tl == 0 && c < C) {
    sum_ds[c] = s1;
    sum_ds_yh[c] = s2;
    if (dgamma_acc) dgamma_acc[c] += s2;
    if (dbeta_acc) dbeta_acc[c] += s1;
  }
}

__global__ void dwconv_bwd_reduce_kernel(const float* __restrict__ part, int n_tiles, int C, int K, float* __restrict__ dfilt,
                                         float* __restrict__ dbias, int accumulate = 0) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= C * (K + 1)) return;
  const int c = idx / (K + 1), k = idx % (K + 1);
  double s = 0.0;
  for (int t = 0; t < n_tiles; ++t) s += part[((size_t)t * C + c) * (K + 1) + k];
  if (accumulate) {
    if (k < K) dfilt[(size_t)c * K + k] += (float)s;
    else if (dbias) dbias[c] += (float)s;
  } else {
    if (k < K) dfilt[(size_t)c * K + k] = (float)s;
    else if (dbias) dbias[c] = (float)s;
  }
}

}  // namespace

// scratch `part` sizes (floats): forward ceil(N/32)*2*C (null: no sums wanted; K <= 32 only); backward-a n_tiles_a*2*C; backward conv ceil(N/32)*C*(K+1)
RB_EXPORT int rb200_glu_dwconv_fwd(const void* x, const float* filt, const float* bias, const int* row_batch, const int* row_pos,
                                   const int* lens, void* y, float* part, int n_rows, int n_seqs, int C, int K, cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (C % CC || K > KMAX || K < 1) {
    rb_set_error("glu_dwconv: C=%d must be a multiple of %d and K=%d <= %d", C, CC, K, KMAX);
    return RB_ERR_ARG;
  }
  if (K <= KM2) {
    static RbPerDevice attr2;
    if (attr2.needed()) {
      cudaFuncSetAttribute(glu_dwconv_fwd2_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwd2Smem);
      cudaFuncSetAttribute(glu_dwconv_fwd2_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwd2Smem);
      attr2.done();
    }
    const Pieces pc = pieces_of(n_rows, n_seqs, C, K, kFwdCtas);
    rb_launch_pdl(K <= 16 ? glu_dwconv_fwd2_kernel<16> : glu_dwconv_fwd2_kernel<32>, dim3(pc.n, C / CC), dim3(kWinThreads), kFwd2Smem, stream,
                  (const __nv_bfloat16*)x, filt, bias, row_batch, (__nv_bfloat16*)y, n_rows, n_seqs, C, K, pc.rows);
    int st = rb_check_launch("glu_dwconv_fwd2");
    if (st || part == nullptr) return st;
    rb_launch_pdl(bn_part_kernel, dim3((n_rows + kPartRows - 1) / kPartRows, (C + CC * 8 - 1) / (CC * 8)), dim3(256), 0, stream,
                  (const __nv_bfloat16*)y, part, n_rows, C);
    return rb_check_launch("bn_part");
  }
  dim3 grid((n_rows + TT - 1) / TT, C / CC);
  glu_dwconv_fwd_kernel<<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, filt, bias, row_batch, row_pos, lens, (__nv_bfloat16*)y, part, n_rows, C, K);
  return rb_check_launch("glu_dwconv_fwd");
}

RB_EXPORT int rb200_bn_stats(const float* part, int n_tiles, int C, float count, float eps, float momentum, float* mean, float* rstd,
                             float* running_mean, float* running_var, cudaStream_t stream) {
  rb_launch_pdl(bn_stats2_kernel, dim3((C + 31) / 32), dim3(256), 0, stream, part, n_tiles, C, count, eps, momentum, mean, rstd, running_mean, running_var);
  return rb_check_launch("bn_stats");
}

RB_EXPORT int rb200_bn_silu_fwd(const void* y, const float* mean, const float* rstd, const float* gamma, const float* beta, void* z,
                                long long n_rows, int C, cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (C % 8) return RB_ERR_ARG;
  long long total = n_rows * C;
  rb_launch_pdl(bn_silu_fwd_kernel, dim3(rows_grid(total / 8, C / 8)), dim3(256), 0, stream, (const __nv_bfloat16*)y, mean, rstd, gamma, beta, (__nv_bfloat16*)z, total, C);
  return rb_check_launch("bn_silu_fwd");
}

// ds (bf16 [N,C]) receives ds, later overwritten in place by dy. part: n_tiles*2*C floats.
// dgamma_acc / dbeta_acc (optional): the parameter gradients are also added there
RB_EXPORT int rb200_bn_silu_bwd_ex(const void* y, const void* dz, const float* mean, const float* rstd, const float* gamma, const float* beta,
                                   void* ds, float* part, int n_tiles, float* sum_ds, float* sum_ds_yh, long long n_rows, int C,
                                   int training, float* dgamma_acc, float* dbeta_acc, cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  const int groups = C / 8;
  if (C % 8 || groups > 256 || 256 % groups) {
    rb_set_error("bn_silu_bwd: C=%d unsupported", C);
    return RB_ERR_ARG;
  }
  const int row_lanes = 256 / groups;
  const int rows_per_cta = (int)((n_rows + n_tiles - 1) / n_tiles);
  size_t smem = (size_t)row_lanes * 2 * C * sizeof(float);
  rb_launch_pdl(bn_silu_bwd_a_kernel, dim3(n_tiles), dim3(256), smem, stream, (const __nv_bfloat16*)y, (const __nv_bfloat16*)dz, mean, rstd, gamma, beta,
                                                       (__nv_bfloat16*)ds, part, (int)n_rows, C, rows_per_cta);
  int st = rb_check_launch("bn_silu_bwd_a");
  if (st) return st;
  rb_launch_pdl(bn_bwd_reduce2_kernel, dim3((C + 31) / 32), dim3(1024), 0, stream, part, n_tiles, C, sum_ds, sum_ds_yh, dgamma_acc, dbeta_acc);
  st = rb_check_launch("bn_bwd_reduce");
  if (st) return st;
  if (training) {
    long long total = n_rows * C;
    rb_launch_pdl(bn_silu_bwd_b_kernel, dim3(rows_grid(total / 8, C / 8)), dim3(256), 0, stream, (const __nv_bfloat16*)y, (__nv_bfloat16*)ds, mean, rstd, gamma,
                                                                                 sum_ds, sum_ds_yh, 1.f / (float)n_rows, total, C);
    st = rb_check_launch("bn_silu_bwd_b");
  }
  return st;
}

RB_EXPORT int rb200_bn_silu_bwd(const void* y, const void* dz, const float* mean, const float* rstd, const float* gamma, const float* beta,
                                void* ds, float* part, int n_tiles, float* sum_ds, float* sum_ds_yh, long long n_rows, int C,
                                int training, cudaStream_t stream) {
  return rb200_bn_silu_bwd_ex(y, dz, mean, rstd, gamma, beta, ds, part, n_tiles, sum_ds, sum_ds_yh, n_rows, C, training, nullptr, nullptr, stream);
}

// accumulate: dfilt / dbias += instead of =
RB_EXPORT int rb200_glu_dwconv_bwd_ex(const void* x, const void* dy, const float* filt, const int* row_batch, const int* row_pos,
                                      const int* lens, void* dx, float* part, float* dfilt, float* dbias, int n_rows, int n_seqs, int C, int K,
                                      int accumulate, cudaStream_t stream) {
  if (n_rows <= 0) return RB_OK;
  if (C % CC || K > KMAX || K < 1) return RB_ERR_ARG;
  const int n_tiles = (n_rows + TT - 1) / TT;
  // about four CTAs per SM in total; every CTA leaves one partial
  int row_ctas = (4 * 148 + C / CC - 1) / (C / CC);
  if (row_ctas > n_tiles) row_ctas = n_tiles;
  dim3 grid(row_ctas, C / CC);
  if (K <= KM2) {
    static RbPerDevice attr2;
    if (attr2.needed()) {
      for (auto kernel : {glu_dwconv_bwd2_kernel<16, false>, glu_dwconv_bwd2_kernel<32, false>, glu_dwconv_bwd2_kernel<16, true>, glu_dwconv_bwd2_kernel<32, true>})
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwd2Smem);
      attr2.done();
    }
    const Pieces pc = pieces_of(n_rows, n_seqs, C, K, kBwdCtas);
    row_ctas = pc.walkers;  // every CTA leaves one partial
    const bool many = pc.walkers < pc.n;
    auto kernel = K <= 16 ? (many ? glu_dwconv_bwd2_kernel<16, true> : glu_dwconv_bwd2_kernel<16, false>)
                          : (many ? glu_dwconv_bwd2_kernel<32, true> : glu_dwconv_bwd2_kernel<32, false>);
    rb_launch_pdl(kernel, dim3(pc.walkers, C / CC), dim3(kWinThreads), kBwd2Smem, stream,
                  (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, filt, row_batch, (__nv_bfloat16*)dx, part, n_rows, n_seqs, C, K, pc.rows, pc.n);
    int st2 = rb_check_launch("glu_dwconv_bwd2");
    if (st2) return st2;
    rb_launch_pdl(dwconv_bwd_reduce2_kernel, dim3((C * (K + 1) + 31) / 32), dim3(256), 0, stream, part, row_ctas, C, K, dfilt, dbias, accumulate);
    return rb_check_launch("dwconv_bwd_reduce2");
  } else {
    static RbPerDevice attr;
    if (attr.needed()) {
      cudaFuncSetAttribute(glu_dwconv_bwd_kernel<KMAX>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      attr.done();
    }
    glu_dwconv_bwd_kernel<KMAX><<<grid, kThreads, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, filt, row_batch, row_pos, lens,
                                                               (__nv_bfloat16*)dx, part, n_rows, C, K);
  }
  int st = rb_check_launch("glu_dwconv_bwd");
  if (st) return st;
  dwconv_bwd_reduce_kernel<<<(C * (K + 1) + 255) / 256, 256, 0, stream>>>(part, row_ctas, C, K, dfilt, dbias, accumulate);
  return rb_check_launch("dwconv_bwd_reduce");
}

RB_EXPORT int rb200_glu_dwconv_bwd(const void* x, const void* dy, const float* filt, const int* row_batch, const int* row_pos,
                                   const int* lens, void* dx, float* part, float* dfilt, float* dbias, int n_rows, int n_seqs, int C, int K,
                                   cudaStream_t stream) {
  return rb200_glu_dwconv_bwd_ex(x, dy, filt, row_batch, row_pos, lens, dx, part, dfilt, dbias, n_rows, n_seqs, C, K, 0, stream);
}

// One call per direction for programs that launch the module by itself, where the host sets the pace up to a few thousand rows: a training pass
// of one utterance takes 163 us of its time (three calls forward and two backward: 174, of which 6 for the launch of bn_part).
//
// x [n_rows, 2C] -> y (convolution) and z [n_rows, C]; part: as for rb200_glu_dwconv_fwd; stats [2][C]: mean and 1 / deviation, taken from y where
// own_stats is set (running_mean / running_var, if given, move towards them) and else given
RB_EXPORT int rb200_conv_module_fwd(const void* x, const float* filt, const float* bias, const float* gamma, const float* beta, const int* row_batch,
                                    const int* row_pos, const int* lens, void* y, void* z, float* part, float* stats, float* running_mean,
                                    float* running_var, int n_rows, int n_seqs, int C, int K, int own_stats, float eps, float momentum,
                                    cudaStream_t stream) {
  int st = rb200_glu_dwconv_fwd(x, filt, bias, row_batch, row_pos, lens, y, part, n_rows, n_seqs, C, K, stream);
  if (st == RB_OK && own_stats)
    st = rb200_bn_stats(part, (n_rows + TT - 1) / TT, C, (float)n_rows, eps, momentum, stats, stats + C, running_mean, running_var, stream);
  return st == RB_OK ? rb200_bn_silu_fwd(y, stats, stats + C, gamma, beta, z, n_rows, C, stream) : st;
}

// backward under batch statistics: ds [n_rows, C] and part (the larger of the two scratches, one after the other) are scratch
RB_EXPORT int rb200_conv_module_bwd(const void* x, const void* y, const void* dz, const float* stats, const float* filt, const float* gamma, const float* beta,
                                    const int* row_batch, const int* row_pos, const int* lens, void* ds, float* part, int n_tiles_a, float* sum_ds,
                                    float* sum_ds_yh, void* dx, float* dfilt, float* dbias, int n_rows, int n_seqs, int C, int K, cudaStream_t stream) {
  const int st = rb200_bn_silu_bwd(y, dz, stats, stats + C, gamma, beta, ds, part, n_tiles_a, sum_ds, sum_ds_yh, n_rows, C, 1, stream);
  if (st != RB_OK) return st;
  return rb200_glu_dwconv_bwd(x, ds, filt, row_batch, row_pos, lens, dx, part, dfilt, dbias, n_rows, n_seqs, C, K, stream);
}

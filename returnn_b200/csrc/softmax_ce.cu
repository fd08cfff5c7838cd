// Softmax cross entropy with label smoothing over a large vocabulary.
// One CTA per row; online softmax (running max and sum) in one pass over the logits; backward recomputes
// p = exp(x - lse) and writes dlogits = dloss * (p - q) with q the smoothed target distribution.
// mode 0: q = (1-s) one-hot + s/(V-1) on the other classes, the loss is the cross entropy against q.
// mode 1: the loss is the plain negative log likelihood and only the gradient is smoothed, uniformly over all V classes
//         (q = (1-s) one-hot + s/V): what an identity with a smoothing backward between log-softmax and the loss computes.
// The forward kernel optionally writes the arg max of each row (first index among equal maxima).
#include "common.cuh"
#include <type_traits>

namespace {

__device__ __forceinline__ float ld(const void* x, int64_t i, int is_bf16) {
  return is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i]) : reinterpret_cast<const float*>(x)[i];
}

// A row of an odd vocabulary starts anywhere: single elements up to the first 16-byte boundary of the logits, 16-byte accesses from there
// on, single elements at the end. (With single elements for every such row, 6000 x 10025 took as long as 6000 x 32000.)
__device__ __forceinline__ int row_head(const void* x, int64_t base, int v, int elem) {
  const int off = (int)((reinterpret_cast<uintptr_t>(x) + (uint64_t)base * elem) & 15);
  return min(off ? (16 - off) / elem : 0, v);
}

// kArg: the arg max is wanted, kTot: the plain sum of the row is (label smoothing in the loss). Every class costs an exponential, and the
// instructions around it are what kept the pass from the rate of its reads: with the position of the maximum searched and the sum taken for
// every caller, 6001 x 32000 bf16 took 89 us (4.3 TB/s). The maximum of a group comes from packed 16-bit comparisons, and its position is
// looked up only in batches that hold a new one; a batch of 32 classes changes the running maximum once.
//
// 16 bytes: 8 bf16 or 4 fp32 values
template <bool kBf16>
struct Chunk {
  static constexpr int kN = kBf16 ? 8 : 4;
  uint4 u;
  __device__ __forceinline__ void load(const void* x, int64_t at) {
    u = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(x) + at * (kBf16 ? 2 : 4));
  }
  __device__ __forceinline__ void fill_neg_inf() { u.x = u.y = u.z = u.w = kBf16 ? 0xff80ff80u : 0xff800000u; }
  __device__ __forceinline__ float at(int i) const {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
    if (kBf16) return __uint_as_float(i & 1 ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16);
    return __uint_as_float(w[i]);
  }
  __device__ __forceinline__ float max() const {
    if (kBf16) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
      const float2 m = __bfloat1622float2(__hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
      return fmaxf(m.x, m.y);
    }
    return fmaxf(fmaxf(at(0), at(1)), fmaxf(at(2), at(3)));
  }
};

// kBatch: chunks of a row that a thread has in flight. Two where four would leave half of the last batch of loads empty (up to little more than 4096
// classes, and from 9000 to 12288), and up to 16383 with the position of the maximum, whose search goes through all chunks; else four. us, bf16, out of memory, four / two:
// with the sum of the row 6000 x 1000 12.0 / 11.1, x 4000 18.4 / 17.0, x 6000 21.4 / 22.3, x 8000 24.6 / 25.3, x 10001 33.2 / 31.7, x 14000 37.5 / 38.4,
// x 32000 68.9 / 72.7; without 11.5 / 10.6, 16.9 / 15.2, 19.2 / 20.8, 22.2 / 23.4, 30.8 / 29.6, 34.2 / 35.7, 64.5 / 68.5; with the position 13.9 / 11.6,
// 22.6 / 17.9, 25.1 / 25.2, 28.3 / 27.8, 40.9 / 36.1, 44.6 / 44.2, 82.9 / 83.7. Both have eight CTAs on an SM (32 registers).
// kWide: as many registers as the loads of a batch like (up to 42, six CTAs), for fp32 rows of several batches; 32 registers / that: 6000 x 500 11.7 / 13.9,
// 6000 x 5000 27.3 / 27.9 (without the sum 27.1 / 25.1), 1500 x 16000 21.4 / 19.0, 6000 x 32000 119.4 / 114.1.
template <bool kBf16, bool kArg, bool kTot, int kBatch, bool kWide>
__global__ void __launch_bounds__(256, kWide ? 1 : 0)
ce_fwd_kernel(const void* __restrict__ logits, const int* __restrict__ tgt, float* __restrict__ loss, float* __restrict__ lse_out,
              int v, float smoothing, int* __restrict__ argmax_out) {
  constexpr int is_bf16 = kBf16 ? 1 : 0;
  const int64_t row = blockIdx.x;
  const int64_t base = row * (int64_t)v;
  float mx = -INFINITY, sum = 0.f, tot = 0.f;
  int bi = 0x7fffffff;  // index of this thread's first maximum
  const int head = row_head(logits, base, v, kBf16 ? 2 : 4);
  const int v8 = head + ((v - head) & ~7);
  for (int c = threadIdx.x; c < head; c += blockDim.x) {
    float a = ld(logits, base + c, is_bf16);
    if (kArg && a > mx) bi = c;
    float nm = fmaxf(mx, a);
    const float nu = nm == -INFINITY ? 0.f : nm;  // (only classes of score -inf so far)
    sum = sum * __expf(mx - nu) + __expf(a - nu);
    mx = nm;
    if (kTot) tot += a;
  }
  constexpr int kN = Chunk<kBf16>::kN;
  for (int c0 = head + threadIdx.x * kN; c0 < v8; c0 += kBatch * 256 * kN) {
    Chunk<kBf16> a[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      const int c = c0 + q * 256 * kN;
      if (c < v8) a[q].load(logits, base + c);
      else a[q].fill_neg_inf();
    }
    float lm = a[0].max();
#pragma unroll
    for (int q = 1; q < kBatch; ++q) lm = fmaxf(lm, a[q].max());
    if (kArg && lm > mx) {
#pragma unroll
      for (int q = kBatch - 1; q >= 0; --q)
#pragma unroll
        for (int k = kN - 1; k >= 0; --k)
          if (a[q].at(k) == lm) bi = c0 + q * 256 * kN + k;
    }
    const float nm = fmaxf(mx, lm);
    const float nu = nm == -INFINITY ? 0.f : nm;
    float s = 0.f;
    auto add = [&](int q) {
#pragma unroll
      for (int k = 0; k < kN; ++k) {
        s += __expf(a[q].at(k) - nu);
        if (kTot) tot += a[q].at(k);
      }
    };
    if (c0 + (kBatch - 1) * 256 * kN < v8) {
#pragma unroll
      for (int q = 0; q < kBatch; ++q) add(q);
    } else {  // no exponentials of padding (24 of 32 in a row of 1000 classes)
#pragma unroll
      for (int q = 0; q < kBatch - 1; ++q)
        if (c0 + q * 256 * kN < v8) add(q);
    }
    sum = sum * __expf(mx - nu) + s;
    mx = nm;
  }
  for (int c = v8 + threadIdx.x; c < v; c += blockDim.x) {
    float a = ld(logits, base + c, is_bf16);
    if (kArg && a > mx) bi = c;
    float nm = fmaxf(mx, a);
    const float nu = nm == -INFINITY ? 0.f : nm;  // (only classes of score -inf so far)
    sum = sum * __expf(mx - nu) + __expf(a - nu);
    mx = nm;
    if (kTot) tot += a;
  }
  __shared__ float sh_m[8], sh_s[8], sh_t[8];
  __shared__ int sh_i[8];
  float wm = warp_max(mx);
  int wi = (mx == wm) ? bi : 0x7fffffff;
  if (kArg)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wi = min(wi, __shfl_xor_sync(0xffffffffu, wi, o));
  float ws = warp_sum(mx == -INFINITY ? 0.f : sum * __expf(mx - wm));
  float wt = kTot ? warp_sum(tot) : 0.f;
  if ((threadIdx.x & 31) == 0) {
    sh_m[threadIdx.x >> 5] = wm;
    sh_s[threadIdx.x >> 5] = ws;
    sh_t[threadIdx.x >> 5] = wt;
    sh_i[threadIdx.x >> 5] = wi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = sh_m[0];
    for (int w = 1; w < 8; ++w) m = fmaxf(m, sh_m[w]);
    float s = 0.f, t = 0.f;
    int am = 0x7fffffff;
    for (int w = 0; w < 8; ++w) {
      if (sh_m[w] != -INFINITY) s += sh_s[w] * __expf(sh_m[w] - m);
      t += sh_t[w];
      if (sh_m[w] == m) am = min(am, sh_i[w]);
    }
    if (kArg) argmax_out[row] = am < v ? am : 0;
    float lse = m + logf(s);
    int y = tgt[row];
    float xy = (y >= 0 && y < v) ? ld(logits, base + y, is_bf16) : 0.f;
    float nll = lse - xy;
    float l = nll;
    if (kTot) {
      // other = mean over the v-1 non-target classes of (lse - x_c)
      float other = ((float)v * lse - t - nll) / (float)(v - 1);
      l = (1.f - smoothing) * nll + smoothing * other;
    }
    loss[row] = (y >= 0 && y < v) ? l : 0.f;
    lse_out[row] = lse;
  }
}

template <bool kBf16, bool kLastFirst>
__global__ void __launch_bounds__(256)
ce_bwd_kernel(const void* __restrict__ logits, const int* __restrict__ tgt, const float* __restrict__ lse_in,
              const float* __restrict__ dloss, void* __restrict__ dlogits, int v, float smoothing, int mode) {
  constexpr int is_bf16 = kBf16 ? 1 : 0;
  const int64_t row = kLastFirst ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const int64_t base = row * (int64_t)v;
  const float lse = lse_in[row];
  const int y = tgt[row];
  const bool valid = y >= 0 && y < v;
  const float dl = valid ? dloss[row] : 0.f;
  const float q_other = smoothing > 0.f ? smoothing / (float)(mode == 1 ? v : v - 1) : 0.f;
  const float q_tgt = 1.f - smoothing + (mode == 1 ? q_other : 0.f);
  const int head_in = row_head(logits, base, v, kBf16 ? 2 : 4), head_out = row_head(dlogits, base, v, kBf16 ? 2 : 4);
  const int head = head_in == head_out ? head_in : v;  // (buffers that are aligned differently: single elements)
  const int v8 = head + ((v - head) & ~7);
#pragma unroll 4
  for (int c = head + threadIdx.x * 8; c < v8; c += blockDim.x * 8) {
    F8 a = load8(logits, base + c, is_bf16);
    F8 o;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float p = __expf(a.v[k] - lse);
      float q = (c + k == y) ? q_tgt : q_other;
      o.v[k] = dl * (p - q);
    }
    store8(dlogits, base + c, o, is_bf16);
  }
  for (int i = threadIdx.x; i < v - (v8 - head); i += blockDim.x) {
    const int c = i < head ? i : i + (v8 - head);
    float p = __expf(ld(logits, base + c, is_bf16) - lse);
    float q = (c == y) ? q_tgt : q_other;
    float o = dl * (p - q);
    if (is_bf16) reinterpret_cast<__nv_bfloat16*>(dlogits)[base + c] = __float2bfloat16(o);
    else reinterpret_cast<float*>(dlogits)[base + c] = o;
  }
}

}  // namespace

RB_EXPORT int rb200_softmax_ce_fwd(const void* logits, const int* tgt, float* loss, float* lse, long long rows, int v, float smoothing,
                                   int is_bf16, int mode, int* argmax_out, cudaStream_t stream) {
  if (rows <= 0) return RB_OK;
  if (v < 2) return RB_ERR_ARG;
  const bool arg = argmax_out != nullptr, tot = smoothing > 0.f && mode == 0;
  auto pick = [&](auto bf16, auto batch, auto wide) {
    constexpr bool kB = decltype(bf16)::value, kW = decltype(wide)::value;
    constexpr int kN = decltype(batch)::value;
    return arg ? (tot ? ce_fwd_kernel<kB, true, true, kN, kW> : ce_fwd_kernel<kB, true, false, kN, kW>)
               : (tot ? ce_fwd_kernel<kB, false, true, kN, kW> : ce_fwd_kernel<kB, false, false, kN, kW>);
  };
  using Two = std::integral_constant<int, 2>;
  using Four = std::integral_constant<int, 4>;
  const std::true_type yes;
  const std::false_type no;
  const bool two = v <= 4352 || (v >= 9000 && v <= 12288) || (arg && v < 16384);
  auto kernel = is_bf16 ? (two ? pick(yes, Two(), no) : pick(yes, Four(), no)) : v < 4096 ? pick(no, Four(), no) : pick(no, Four(), yes);
  kernel<<<(unsigned)rows, 256, 0, stream>>>(logits, tgt, loss, lse, v, smoothing, argmax_out);
  return rb_check_launch("softmax_ce_fwd");
}

RB_EXPORT int rb200_softmax_ce_bwd(const void* logits, const int* tgt, const float* lse, const float* dloss, void* dlogits,
                                   long long rows, int v, float smoothing, int is_bf16, int mode, cudaStream_t stream) {
  if (rows <= 0) return RB_OK;
  // The last rows first where the logits and their gradient do not fit the L2 together (126 MB): what the forward pass read last is what it still holds.
  // Where they do, or all rows are resident at once, the order they are read in is the better one. us of both passes, bf16, first / last rows first, the
  // logits out of memory: 6000 x 32000 198.3 / 193.3, 1500 x 32000 60.6 / 57.1, 3000 x 16384 55.7 / 54.5; 1500 x 20000 (60 MB) 37.4 / 37.4, 1500 x 16384 29.2 / 29.9,
  // 800 x 8000 11.3 / 11.7, 1100 x 50000 65.8 / 67.3
  const bool last_first = rows > 8 * 148 && rows * v * (is_bf16 ? 2 : 4) >= (64LL << 20);
  auto kernel = is_bf16 ? (last_first ? ce_bwd_kernel<true, true> : ce_bwd_kernel<true, false>) : last_first ? ce_bwd_kernel<false, true> : ce_bwd_kernel<false, false>;
  kernel<<<(unsigned)rows, 256, 0, stream>>>(logits, tgt, lse, dloss, dlogits, v, smoothing, mode);
  return rb_check_launch("softmax_ce_bwd");
}

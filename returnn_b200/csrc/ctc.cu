// CTC loss with fused log-softmax on packed logits [N, V] (bf16 or fp32), forward and gradient in three launches:
//
//   ctc_softmax_gather   1 to 24 warps per frame: the row is read once and kept in registers, log-sum-exp over the vocabulary, the probabilities of
//                        the 2S+1 extended states (blank, l1, blank, l2, ..., blank), and the softmax straight to the gradient
//   ctc_alpha_beta       one CTA per sequence: the alpha and the beta recursion run at the same time in the two halves of the CTA, and the
//                        log-likelihood
//   ctc_occupancy        one warp per frame: the few gradient entries of the label classes, softmax minus the occupancies
//                        alpha * beta / P (several states share a class: all blanks, repeated labels)
//
// The [T, V] log-probabilities are never materialised. Scratch (global memory, given by the caller), SE = 2 * max_target_len + 1:
// lse [N], wide [N], prob, alpha, beta [N, SE + 1] numbers with an exponent of their own (8 bytes), and 4 + SE words per sequence.
// Infeasible alignments (fewer frames than needed) give loss 0 and zero gradient (zero_infinity semantics).
//
// 7900 frames x 10001 classes in 36 sequences of up to 333 frames, 67 labels (bf16): softmax 64 us (read and written once, 316 MB: 48 at the
// rate of a copy), recursions 52 (333 dependent frames), occupancies 20 (four dependent loads a frame), scaling in the backward pass 50 (316 MB, near
// the rate of a copy). Before: log-sum-exp 51, recursions in log space 92, gradient in a pass of its own 93, scaling 54.
#include <algorithm>
#include "common.cuh"

namespace {

constexpr float kNegInf = -INFINITY;

__device__ __forceinline__ float ldf(const void* x, size_t i, int is_bf16) {
  return is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(x)[i]) : reinterpret_cast<const float*>(x)[i];
}
__device__ __forceinline__ void stf(void* x, size_t i, float v, int is_bf16) {
  if (is_bf16) reinterpret_cast<__nv_bfloat16*>(x)[i] = __float2bfloat16(v);
  else reinterpret_cast<float*>(x)[i] = v;
}
// log(e^a + e^b + e^c); all three -inf give -inf
__device__ __forceinline__ float log_add3(float a, float b, float c) {
  const float lo = fminf(a, b), hi = max_nan(a, b), m = max_nan(hi, c);
  const float other = fminf(hi, c);  // the two that are not the largest: lo and this one
  const float sum = m + log1pf(__expf(lo - m) + __expf(other - m));
  return m == kNegInf ? m : sum;
}

// A non-negative number m * 2^e. The recursions over a sequence multiply a few hundred probabilities, far outside fp32's range; in log space
// every sum of three costs three exponentials and a logarithm, one after the other (0.28 us a frame), and values of a few thousand leave
// 2^-12 of relative precision. With the exponent beside the mantissa a sum takes shifts of exponents and two fused multiply-adds, and keeps 24 bits.
struct Wide {
  float m;
  int e;
};
constexpr int kFloor = -(1 << 29);      // exponent of zero; sums of two of them still fit
constexpr int kZeroBelow = -(1 << 28);  // exponents below stand for zero
// log-probabilities below this (in powers of two) would take a sequence of T frames out of the exponent's range: such a sequence (logits masked
// with a large negative number, say) takes the recursion in log space
__device__ __forceinline__ float wide_limit(int T) { return -(float)(1 << 28) / (float)(T + 1); }

// 2^(e - top), 0 below 2^-126; e - top <= 127
__device__ __forceinline__ float pow2i(int e, int top) {
  return __int_as_float(__viaddmax_s32(e, -top, -127) * (1 << 23) + 0x3f800000);
}

__device__ __forceinline__ Wide wide_exp(float lp) {  // e^lp for lp <= 0 (a little above: rounding)
  if (lp == kNegInf) return {0.f, kFloor};
  const float t = fmaxf(lp * 1.4426950408889634f, -1e9f);
  const float r = rintf(t);
  float f;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(t - r));
  return {lp != lp ? lp : f, lp != lp ? 0 : (int)r};
}

// x holds 16 bytes: 8 bf16 or 4 fp32 values
template <bool BF16>
struct Pack {
  static constexpr int N = BF16 ? 8 : 4;
  __device__ static __forceinline__ void get(uint4 u, float (&v)[N]) {
    if constexpr (BF16) {
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
      }
    } else {
      v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
    }
  }
  // the largest element of two vectors, element by element
  __device__ static __forceinline__ uint4 larger(uint4 a, uint4 b) {
    if constexpr (BF16) {
      __nv_bfloat162* x = reinterpret_cast<__nv_bfloat162*>(&a);
      const __nv_bfloat162* y = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = __hmax2(x[i], y[i]);
    } else {
      a = make_uint4(__float_as_uint(fmaxf(__uint_as_float(a.x), __uint_as_float(b.x))), __float_as_uint(fmaxf(__uint_as_float(a.y), __uint_as_float(b.y))),
                     __float_as_uint(fmaxf(__uint_as_float(a.z), __uint_as_float(b.z))), __float_as_uint(fmaxf(__uint_as_float(a.w), __uint_as_float(b.w))));
    }
    return a;
  }
  __device__ static __forceinline__ uint4 put(const float (&v)[N]) {
    uint4 u;
    if constexpr (BF16) {
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
      for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    } else {
      u = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
    }
    return u;
  }
};

// A row of V elements that starts anywhere: `head` elements up to a 16-byte boundary, `n_vec` vectors, the rest behind them. `other` (null:
// none) is a second buffer with rows of the same pitch: where its boundaries lie elsewhere, there are no vectors.
struct Row {
  int head, n_vec, scalars;  // scalars: elements outside the vectors
};
template <bool BF16>
__device__ __forceinline__ Row row_of(const void* x, const void* other, size_t base, int V) {
  constexpr int size = BF16 ? 2 : 4, per = 16 / size;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x) + base * size;
  Row r;
  if (other != nullptr && ((reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(other)) & 15)) {
    r.head = V;
  } else {
    r.head = min((int)((16 - (at & 15)) & 15) / size, V);
  }
  r.n_vec = (V - r.head) / per;
  r.scalars = V - r.n_vec * per;
  return r;
}
// position of scalar i
template <bool BF16>
__device__ __forceinline__ int scalar_at(const Row& r, int i) {
  return i < r.head ? i : i + r.n_vec * (BF16 ? 8 : 4);
}

template <int T>
__device__ __forceinline__ float cta_reduce(float v, float* sh, bool sum) {
  v = sum ? warp_sum(v) : warp_max(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  v = sh[0];
#pragma unroll
  for (int i = 1; i < T / 32; ++i) v = sum ? v + sh[i] : fmaxf(v, sh[i]);
  return v;
}

// Persistent CTAs of T threads, a frame at a time: T * NV vectors of the row stay in registers, as exponentials from the second pass over them
// on (the launch picks both by V); a longer row's rest is read three times. The next row is loaded as soon as the vectors are exponentials, and
// the chain sequence -> number of states -> class -> logit of the states is one step further with each phase of a row.
// grad (null: none wanted) receives the softmax.
// The exponentials are 2^(x log2(e) - c) with a whole number c near the maximum: one rounding each. (That of the constant, 1.3e-8 of it, moves all
// exponents of a row alike, by less than half a unit in the last place of the logit.) Where the maximum lies beyond
// 2^30, c is off by up to 64 and more, at last the product overflows (a frame that is filled with the type's lowest value): the log-sum-exp is not
// finite then, and the row is left to the next kernel. (A factor and an offset chosen by row, to have such rows right here: 75 us for 65.)
template <int T, int NV, bool BF16>
__global__ void __launch_bounds__(T, 768 / T)
ctc_softmax_gather_kernel(const void* __restrict__ logits, const int* __restrict__ row_batch, const int* __restrict__ cu, const int* __restrict__ targets,
                          const int* __restrict__ tgt_lens, float* __restrict__ lse, int* __restrict__ wide, Wide* __restrict__ prob,
                          void* __restrict__ grad, int n_rows, int V, int s_pitch, int pitch, int blank) {
  using P = Pack<BF16>;
  constexpr float kLog2e = 1.4426950408889634f;
  constexpr int kSize = BF16 ? 2 : 4;
  constexpr uint32_t kLow = BF16 ? 0xFF80FF80u : 0xFF800000u;  // -inf
  __shared__ float sh[2][T / 32];
  const int tid = threadIdx.x;
  uint4 raw[NV];
  auto load = [&](int r) {
    const size_t base = (size_t)r * V;
    const Row row = row_of<BF16>(logits, grad, base, V);
    const uint4* vec = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(logits) + (base + row.head) * kSize);
#pragma unroll
    for (int i = 0; i < NV; ++i) raw[i] = tid + i * T < row.n_vec ? vec[tid + i * T] : make_uint4(kLow, kLow, kLow, kLow);
  };
  auto cls_of = [&](int b, int s) { return (s & 1) ? targets[(size_t)b * s_pitch + (s >> 1)] : blank; };
  int r = blockIdx.x;
  load(r);
  int b = row_batch[r], se = 2 * tgt_lens[b] + 1;
  float limit = wide_limit(cu[b + 1] - cu[b]) * 0.6931471805599453f;
  int cls = tid < se ? cls_of(b, tid) : blank;
  for (; r < n_rows; r += gridDim.x) {
    const size_t base = (size_t)r * V;
    const Row row = row_of<BF16>(logits, grad, base, V);
    const uint4* vec = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(logits) + (base + row.head) * kSize);
    const int rn = min(r + (int)gridDim.x, n_rows - 1);
    const float mine = ldf(logits, base + cls, BF16);
    const int bn = row_batch[rn];
    float mx = kNegInf;
    for (int i = tid; i < row.scalars; i += T) mx = fmaxf(mx, ldf(logits, base + scalar_at<BF16>(row, i), BF16));
    uint4 top = raw[0];
#pragma unroll
    for (int i = 1; i < NV; ++i) top = P::larger(top, raw[i]);
    for (int i = tid + NV * T; i < row.n_vec; i += T) top = P::larger(top, vec[i]);
    {
      float v[P::N];
      P::get(top, v);
#pragma unroll
      for (int k = 0; k < P::N; ++k) mx = fmaxf(mx, v[k]);
    }
    mx = cta_reduce<T>(mx, sh[0], false);
    const float c = rintf(mx * kLog2e);
    auto ex = [&](float x) {
      float y;
      asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaf(x, kLog2e, -c)));
      return y;
    };
    float sum = 0.f;
    for (int i = tid; i < row.scalars; i += T) sum += ex(ldf(logits, base + scalar_at<BF16>(row, i), BF16));
    float e[NV][P::N];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      P::get(raw[i], e[i]);
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < P::N; ++k) t += e[i][k] = ex(e[i][k]);
      sum += i + 1 < NV || tid + i * T < row.n_vec ? t : 0.f;
    }
    for (int i = tid + NV * T; i < row.n_vec; i += T) {
      float v[P::N], t = 0.f;
      P::get(vec[i], v);
#pragma unroll
      for (int k = 0; k < P::N; ++k) t += ex(v[k]);
      sum += t;
    }
    const int sen = 2 * tgt_lens[bn] + 1, len = cu[bn + 1] - cu[bn];
    load(rn);
    sum = cta_reduce<T>(sum, sh[1], true);
    const float l = fmaf(c, 0.693147182464599609375f, fmaf(c, -1.904654323148236e-9f, logf(sum)));  // ln 2 in two parts
    const int clsn = tid < sen ? cls_of(bn, tid) : blank;
    bool far = !(fabsf(l) < INFINITY);
    for (int s = tid; s < se; s += T) {
      const float lp = (s == tid ? mine : ldf(logits, base + cls_of(b, s), BF16)) - l;
      far |= lp < limit && lp != kNegInf;
      prob[(size_t)r * pitch + s] = wide_exp(lp);
    }
    const int any = __syncthreads_or(far);
    if (tid == 0) {
      lse[r] = l;
      wide[r] = any;
    }
    if (grad != nullptr) {
      const float inv = 1.f / sum;
      uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<char*>(grad) + (base + row.head) * kSize);
      for (int i = tid; i < row.scalars; i += T) {
        const size_t at = base + scalar_at<BF16>(row, i);
        stf(grad, at, ex(ldf(logits, at, BF16)) * inv, BF16);
      }
#pragma unroll
      for (int i = 0; i < NV; ++i) {
#pragma unroll
        for (int k = 0; k < P::N; ++k) e[i][k] *= inv;
        if (tid + i * T < row.n_vec) out[tid + i * T] = P::put(e[i]);
      }
      for (int i = tid + NV * T; i < row.n_vec; i += T) {
        float v[P::N];
        P::get(vec[i], v);
#pragma unroll
        for (int k = 0; k < P::N; ++k) v[k] = ex(v[k]) * inv;
        out[i] = P::put(v);
      }
    }
    b = bn;
    se = sen;
    cls = clsn;
    limit = wide_limit(len) * 0.6931471805599453f;
  }
}

__device__ __forceinline__ void bar_sync_named(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// what the occupancies need of a sequence: P = m * 2^e, or (in_log) alpha and beta are logarithms and `logp` belongs to them
struct __align__(16) SeqInfo {
  float m;
  int e;
  float logp;  // -inf: infeasible
  int in_log;
};

// One recursion of a sequence. State i of T is the lattice state i for alpha, se - 1 - i for beta, which runs from the last frame to the first:
//   x'[i] = (x[i] + x[i-1] + skip[i] x[i-2]) * p[i],  skip: i is a label and differs from the label before it
// has the same form for both. A lane owns K (even) consecutive states, i.e. blank, label, blank, ..., and needs one value of the lane before.
// What a lane lacks moves up by two states per frame: a warp starts 2 D states early (the first warp at states that stay zero) and is right in
// the others for D frames, after which the warps exchange their states through shared memory. States past the last one need not be right
// either, so no load or product is guarded. The probabilities of the next two groups of D frames are on their way to shared memory (in
// registers they wait for each other's loads, of which a warp tells only six apart: 440 cycles a frame); K = 8, for the longest label
// sequences, has no room for that. alpha is stored with the frame's own probability, beta without. The rows of prob, alpha and beta have an even pitch, and beta stands one column further right: the K states of a
// lane are stored as 16-byte pairs. (One warp with 6 states per lane, guarded: 90 half-rate instructions and 590 cycles a frame.)
constexpr int kStages = 3;

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int K, int D>
struct Lattice {
  static constexpr bool kStaged = K < 8;
  static constexpr int kStage = D * K * 32;  // Wides of a warp's stage: [D][32 lanes][K]
  static constexpr int kHalo = (2 * D + K - 1) / K;  // lanes
  static constexpr int kOwn = (32 - kHalo) * K;      // states that a warp brings further
  static int warps(int SE) { return (SE + kOwn - 1) / kOwn; }
};

template <int K, int D, bool BACK>
__device__ __forceinline__ Wide ctc_recursion(const Wide* __restrict__ prob, Wide* __restrict__ out, const int* __restrict__ cls, int r0, int T, int se,
                                              int SE, int lane, int w, int n_warps, Wide* state, Wide* ring) {
  constexpr int kHalo = Lattice<K, D>::kHalo;
  const int pitch = SE + 1;
  const int i0 = w * Lattice<K, D>::kOwn + (lane - kHalo) * K;
  const bool own = lane >= kHalo;
  prob += (long long)r0 * pitch;
  out += (long long)r0 * pitch;
  const int step = BACK ? -pitch : pitch;
  const int first = BACK ? (T - 1) * pitch : 0, end = BACK ? 0 : (T - 1) * pitch;  // the first and the last frame's row
  int at[K];  // column of the lane's states in prob; outside the lattice any
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const int i = min(max(i0 + j, 0), se - 1);
    at[j] = BACK ? se - 1 - i : i;
  }
  const int n_out = own ? max(0, min(K, se - i0)) : 0;
  uint32_t skip = 0;
#pragma unroll
  for (int j = 1; j < K; j += 2) {
    const int i = i0 + j;
    if (i >= 2 && i < se && cls[BACK ? se - 1 - i : i] != cls[BACK ? se + 1 - i : i - 2]) skip |= 1u << j;
  }
  // states i0 + j, i0 + j + 1 (j even) of a frame's row `o`; what stands behind the last state lands in a column that nobody reads
  auto store = [&](int o, int j, Wide a, Wide z) {
    if (j >= n_out) return;
    if (BACK) *reinterpret_cast<float4*>(out + (o + se - 1 - i0 - j)) = make_float4(z.m, __int_as_float(z.e), a.m, __int_as_float(a.e));
    else *reinterpret_cast<float4*>(out + (o + i0 + j)) = make_float4(a.m, __int_as_float(a.e), z.m, __int_as_float(z.e));
  };
  float m[K];
  int e[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const bool on = i0 + j >= 0 && i0 + j < min(2, se);
    const Wide v = on ? prob[first + at[j]] : Wide{0.f, kFloor};
    m[j] = v.m;
    e[j] = v.e;
  }
#pragma unroll
  for (int j = 0; j < K; j += 2) {
    const bool on = i0 + j == 0, on2 = on && se > 1;
    if (BACK) store(first, j, on ? Wide{1.f, 0} : Wide{0.f, kFloor}, on2 ? Wide{1.f, 0} : Wide{0.f, kFloor});
    else store(first, j, {m[j], e[j]}, {m[j + 1], e[j + 1]});
  }
  constexpr bool kStaged = Lattice<K, D>::kStaged;
  int next = first;  // row of the frame fetched last; behind the last frame that one again
  auto advance = [&]() {
    next = BACK ? max(next + step, end) : min(next + step, end);
    return prob + next;
  };
  auto issue = [&](int stage) {  // the next D frames
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const Wide* p = advance();
#pragma unroll
      for (int j = 0; j < K; ++j) cp_async8(ring + stage * Lattice<K, D>::kStage + (d * 32 + lane) * K + j, p + at[j]);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if constexpr (kStaged) {
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) issue(i);
  }
  int o = first;
  auto frame = [&](const Wide (&x)[K]) {
    o += step;
    const float lm = __shfl_up_sync(0xffffffffu, m[K - 1], 1);
    const int le = __shfl_up_sync(0xffffffffu, e[K - 1], 1);
    Wide res[K];
#pragma unroll
    for (int j = K - 1; j >= 0; --j) {
      const float m1 = j ? m[j - 1] : lm;
      const int e1 = j ? e[j - 1] : le;
      float s;
      int top;
      if (j & 1) {
        const float m2 = j > 1 ? m[j - 2] : lm;
        const int e2 = (skip >> j & 1) ? (j > 1 ? e[j - 2] : le) : kFloor;
        top = __vimax3_s32(e[j], e1, e2);
        s = m[j] * pow2i(e[j], top);
        s = fmaf(m1, pow2i(e1, top), s);
        s = fmaf(m2, pow2i(e2, top), s);
      } else {
        top = max(e[j], e1);
        s = m[j] * pow2i(e[j], top);
        s = fmaf(m1, pow2i(e1, top), s);
      }
      m[j] = s * x[j].m;
      e[j] = __viaddmax_s32(top, x[j].e, kFloor);
      res[j] = BACK ? Wide{s, top} : Wide{m[j], e[j]};
    }
#pragma unroll
    for (int j = 0; j < K; j += 2) store(o, j, res[j], res[j + 1]);
  };
  const int bar = BACK ? 2 : 1;
  Wide* mine = state;  // the states of all warps, in two copies for exchanges in turn
  int stage = 0;
  for (int t0 = 1; t0 < T; t0 += D) {
    Wide q[D][K];
    if constexpr (kStaged) {
      issue(stage == 0 ? kStages - 1 : stage - 1);  // the stage that the group before has left
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");  // a lane reads only what it has fetched itself
      const Wide* x = ring + stage * Lattice<K, D>::kStage + lane * K;
#pragma unroll
      for (int d = 0; d < D; ++d) {
#pragma unroll
        for (int j = 0; j < K; j += 2) {
          const float4 v = *reinterpret_cast<const float4*>(x + d * 32 * K + j);
          q[d][j] = {v.x, __float_as_int(v.y)};
          q[d][j + 1] = {v.z, __float_as_int(v.w)};
        }
      }
      stage = stage == kStages - 1 ? 0 : stage + 1;
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const Wide* p = advance();
#pragma unroll
        for (int j = 0; j < K; ++j) q[d][j] = p[at[j]];
      }
    }
    if (t0 + D <= T) {
#pragma unroll
      for (int d = 0; d < D; ++d) frame(q[d]);
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d)
        if (t0 + d < T) frame(q[d]);
    }
    // a sum at most triples a mantissa and a probability's lies in [0.7, 1.42): D frames leave it far inside fp32's range
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int x = ((__float_as_int(m[j]) >> 23) & 255) - 127;
      if (m[j] > 0.f && m[j] < INFINITY) {
        m[j] = __int_as_float(__float_as_int(m[j]) - (x << 23));
        e[j] = max(e[j] + x, kFloor);
      }
    }
    if (n_warps > 1) {
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (j < n_out) mine[i0 + j] = {m[j], e[j]};
      bar_sync_named(bar, n_warps * 32);
      if (!own && w > 0) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const Wide v = mine[min(i0 + j, se - 1)];
          m[j] = v.m;
          e[j] = v.e;
        }
      }
      mine = mine == state ? state + SE : state;
    }
  }
  // the last two states, of all lanes
#pragma unroll
  for (int j = 0; j < K; ++j)
    if (j < n_out && i0 + j >= se - 2) mine[i0 + j] = {m[j], e[j]};
  if (n_warps > 1) bar_sync_named(bar, n_warps * 32);
  else __syncwarp();
  if constexpr (kStaged) asm volatile("cp.async.wait_all;" ::: "memory");
  const Wide a = mine[se - 1], z = se >= 2 ? mine[se - 2] : Wide{0.f, kFloor};
  const int top = max(a.e, z.e);
  return {a.m * pow2i(a.e, top) + z.m * pow2i(z.e, top), top};
}

// A row whose maximum lies beyond 2^30, by all threads of a CTA: two values there are equal or so far apart (2^7) that the maxima share the row.
// Rows with an infinite maximum, and rows that are not finite because they hold NaN, stay as the pass over the logits has left them.
__device__ void ctc_huge_row(const void* __restrict__ logits, int is_bf16, size_t base, int V, float* __restrict__ lse, void* __restrict__ grad, float* sh) {
  float mx = kNegInf, n = 0.f;
  for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, ldf(logits, base + i, is_bf16));
  auto all = [&](float v, bool sum) {
    __syncthreads();
    v = sum ? warp_sum(v) : warp_max(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sh[0];
    for (int i = 1; i < (int)blockDim.x / 32; ++i) v = sum ? v + sh[i] : fmaxf(v, sh[i]);
    return v;
  };
  mx = all(mx, false);
  if (fabsf(mx) <= 0x1p30f || fabsf(mx) == INFINITY) return;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float x = ldf(logits, base + i, is_bf16);
    n += x == mx ? 1.f : x != x ? x : 0.f;
  }
  n = all(n, true);
  if (threadIdx.x == 0) *lse = mx + logf(n);
  if (grad != nullptr)
    for (int i = threadIdx.x; i < V; i += blockDim.x) stf(grad, base + i, (ldf(logits, base + i, is_bf16) == mx ? 1.f : 0.f) / n, is_bf16);
}

// One CTA per sequence, the first half of its warps alpha, the second beta. Dynamic shared memory: SE classes, 4 * SE states, of which a
// sequence that goes through log space uses the first 4 * (SE + 4) floats, and the warps' rings. link [B, SE], for the labels: the next state of the same class, 0 if there
// is none, negative (minus one) where an earlier state has the class or the class is blank.
template <int K, int D>
__global__ void __launch_bounds__(K == 8 ? 832 : 512, 1)
ctc_alpha_beta_kernel(const void* __restrict__ logits, int is_bf16, float* __restrict__ lse, const int* __restrict__ wide, void* __restrict__ grad,
                      const Wide* __restrict__ prob, Wide* __restrict__ al, Wide* __restrict__ be, const int* __restrict__ cu,
                      const int* __restrict__ targets, const int* __restrict__ tgt_lens, SeqInfo* __restrict__ info, int* __restrict__ link,
                      float* __restrict__ loss, int V, int s_pitch, int SE, int blank) {
  extern __shared__ int smem_i[];
  const int warps = blockDim.x >> 6;  // per direction
  int* cls = smem_i;
  Wide* state = reinterpret_cast<Wide*>(smem_i + ((SE + 3) & ~3));  // [2 directions][2][SE]
  Wide* ring = state + 4 * SE + (threadIdx.x >> 5) * kStages * Lattice<K, D>::kStage;  // of this warp (K < 8)
  float* logs = reinterpret_cast<float*>(state);                    // [2 directions][2][2 + SE + 2]
  const int b = blockIdx.x;
  const int r0 = cu[b];
  const int T = cu[b + 1] - r0;
  const int S = tgt_lens[b];
  const int se = 2 * S + 1;
  for (int s = threadIdx.x; s < se; s += blockDim.x) cls[s] = (s & 1) ? targets[(size_t)b * s_pitch + (s >> 1)] : blank;
  int far = 0;
  for (int t = threadIdx.x; t < T; t += blockDim.x) far |= wide[r0 + t];
  far = __syncthreads_or(far);
  if (T <= 0) {
    if (threadIdx.x == 0) {
      info[b] = {0.f, 0, kNegInf, 0};
      loss[b] = 0.f;
    }
    return;
  }
  for (int i = threadIdx.x; i < S; i += blockDim.x) {
    const int s = 2 * i + 1, c = cls[s];
    bool first = c != blank;
#pragma unroll 4
    for (int q = 1; q < s; q += 2) first &= cls[q] != c;
    int next = 0;
#pragma unroll 4
    for (int q = se - 2; q > s; q -= 2) next = cls[q] == c ? q : next;
    link[(size_t)b * SE + s] = first ? next : -next - 1;
  }
  if (!far) {
    const int dir = (int)(threadIdx.x >> 5) >= warps ? 1 : 0;
    const int w = (threadIdx.x >> 5) - dir * warps;
    const Wide P = dir ? ctc_recursion<K, D, true>(prob, be, cls, r0, T, se, SE, threadIdx.x & 31, w, warps, state + 2 * SE, ring)
                       : ctc_recursion<K, D, false>(prob, al, cls, r0, T, se, SE, threadIdx.x & 31, w, warps, state, ring);
    if (threadIdx.x == 0) {
      const bool none = P.m == 0.f || P.e < kZeroBelow;
      const double logp = none ? -INFINITY : (double)P.e * 0.69314718055994530942 + (double)logf(P.m);
      info[b] = {P.m, P.e, (float)logp, 0};
      loss[b] = none ? 0.f : (float)-logp;
    }
    return;
  }
  for (int t0 = 0; t0 < T; t0 += blockDim.x) {
    const int t = t0 + threadIdx.x;
    if (!__syncthreads_or(t < T && !(fabsf(lse[r0 + t]) < INFINITY))) continue;
    for (int q = r0 + t0; q < r0 + min(T, t0 + (int)blockDim.x); ++q)
      if (!(fabsf(lse[q]) < INFINITY)) ctc_huge_row(logits, is_bf16, (size_t)q * V, V, lse + q, grad, reinterpret_cast<float*>(state));
  }
  __syncthreads();
  // ---- in log space, alpha and beta at the same time as above; al and be hold logarithms in place of mantissas. States i, i + G, ... per
  // thread, the log-probabilities of the next frames on their way during the sums of these, -inf around the states in place of conditions:
  // 8236 frames x 10001 classes in 36 sequences, one masked label each, without gradient: 685 -> 218 us (155 where no sequence comes here).
  constexpr int kAhead = K == 2 ? 4 : K == 4 ? 2 : 1;  // frames; a direction's threads hold K states each
  const int G = 32 * warps, dir = (int)threadIdx.x >= G ? 1 : 0, i = threadIdx.x - dir * G, pitch = SE + 4;
  for (int q = threadIdx.x; q < 4 * pitch; q += blockDim.x) logs[q] = kNegInf;
  __syncthreads();
  float* prev = logs + dir * 2 * pitch + 2;
  float* cur = prev + pitch;
  if (i == 0) prev[dir ? se - 1 : 0] = 0.f;  // a frame before the first
  if (dir) bar_sync_named(2, G);
  else bar_sync_named(1, G);
  const int near = dir ? 1 : -1, far_state = 2 * near;
  uint32_t skip = 0;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const int s = i + j * G, q = s + far_state;
    if (s < se && (s & 1) && q >= 0 && q < se && cls[s] != cls[q]) skip |= 1u << j;
  }
  auto fetch = [&](float (&x)[K], int f) {  // of the recursion's frame f
    const int t = r0 + (dir ? max(T - 1 - f, 0) : min(f, T - 1));
    const float l = lse[t];
#pragma unroll
    for (int j = 0; j < K; ++j) x[j] = ldf(logits, (size_t)t * V + cls[min(i + j * G, se - 1)], is_bf16) - l;
  };
  float lp[kAhead][K];
#pragma unroll
  for (int a = 0; a < kAhead; ++a) fetch(lp[a], a);
  Wide* out = dir ? be + (size_t)(r0 + T - 1) * (SE + 1) + 1 : al + (size_t)r0 * (SE + 1);
  const int step = dir ? -(SE + 1) : SE + 1;
  for (int f0 = 0; f0 < T; f0 += kAhead) {
    float next[kAhead][K];
#pragma unroll
    for (int a = 0; a < kAhead; ++a) fetch(next[a], f0 + kAhead + a);
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      if (f0 + a >= T) break;
      float x[K];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const float* p = prev + min(i + j * G, se - 1);
        x[j] = log_add3(p[0], p[near], (skip >> j & 1) ? p[far_state] : kNegInf);
      }
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int s = i + j * G;
        const float y = x[j] == kNegInf ? kNegInf : x[j] + lp[a][j];
        if (s < se) {
          cur[s] = y;
          out[s].m = dir ? x[j] : y;
        }
      }
      out += step;
      if (dir) bar_sync_named(2, G);
      else bar_sync_named(1, G);
      float* q = prev;
      prev = cur;
      cur = q;
    }
#pragma unroll
    for (int a = 0; a < kAhead; ++a)
#pragma unroll
      for (int j = 0; j < K; ++j) lp[a][j] = next[a][j];
  }
  if (threadIdx.x == 0) {
    const float z = log_add3(prev[se - 1], se >= 2 ? prev[se - 2] : kNegInf, kNegInf);
    info[b] = {0.f, 0, z, 1};
    loss[b] = z == kNegInf ? 0.f : -z;
  }
}

// Gradient w.r.t. the logits = softmax(logits) - (occupancy of each class): the softmax is there; one warp per frame rewrites the entries whose
// class occurs in the label sequence (at most S + 1 classes), or clears the rows of an infeasible sequence. The first state of a label adds up
// its equals along the links, blank (half of the states) is a warp sum. Dynamic shared memory: kGradFrames * 2 * SE floats.
constexpr int kGradFrames = 8;

__global__ void __launch_bounds__(32 * kGradFrames)
ctc_occupancy_kernel(const void* __restrict__ logits, int is_bf16, const int* __restrict__ row_batch, const int* __restrict__ targets,
                     const int* __restrict__ tgt_lens, const float* __restrict__ lse, const Wide* __restrict__ al, const Wide* __restrict__ be,
                     const SeqInfo* __restrict__ info, const int* __restrict__ link, void* __restrict__ grad, int n_rows, int V, int s_pitch, int SE,
                     int blank) {
  extern __shared__ float gsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * kGradFrames + warp;
  if (r >= n_rows) return;
  float* g_r = gsm + warp * 2 * SE;  // occupancies of the states
  float* x_r = g_r + SE;             // logits of the labels
  const int b = row_batch[r];
  const SeqInfo seq = info[b];
  const float l = lse[r];
  const int se = 2 * tgt_lens[b] + 1;
  const size_t base = (size_t)r * V;
  if (seq.logp == kNegInf) {
    const int size = is_bf16 ? 2 : 4;
    const Row row = is_bf16 ? row_of<true>(grad, nullptr, base, V) : row_of<false>(grad, nullptr, base, V);
    uint4* out = reinterpret_cast<uint4*>(reinterpret_cast<char*>(grad) + (base + row.head) * size);
#pragma unroll 4
    for (int i = lane; i < row.n_vec; i += 32) out[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = lane; i < row.scalars; i += 32) stf(grad, base + (is_bf16 ? scalar_at<true>(row, i) : scalar_at<false>(row, i)), 0.f, is_bf16);
    return;
  }
  const float inv = seq.in_log ? 0.f : 1.f / seq.m;
  const int* tg = targets + (size_t)b * s_pitch;
  const int* ln = link + (size_t)b * SE;
  const Wide* a = al + (size_t)r * (SE + 1);
  const Wide* z = be + (size_t)r * (SE + 1) + 1;
  auto occupancy = [&](Wide x, Wide y) {
    if (seq.in_log) return (x.m == kNegInf || y.m == kNegInf) ? 0.f : __expf(x.m + y.m - seq.logp);
    return (x.m * y.m) * inv * pow2i(min(x.e + y.e - seq.e, 127), 0);  // beta is without the frame's own probability
  };
  const float x_blank = lane == 0 ? ldf(logits, base + blank, is_bf16) : 0.f;
  float blank_sum = 0.f;
  // a blank and the label behind it per lane, kPairs of them in flight: the loads of a frame follow each other four deep
  constexpr int kPairs = 2;
  struct Label {
    int c;
    float x;
  };
  Label own[kPairs];
  for (int s0 = 2 * lane; s0 < se; s0 += 64 * kPairs) {
    Wide x[kPairs][2], y[kPairs][2];
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const int s = s0 + 64 * j;
      if (s + 1 < se) own[j] = {tg[s >> 1], 0.f};
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        x[j][k] = s + k < se ? a[s + k] : Wide{seq.in_log ? kNegInf : 0.f, kFloor};
        y[j][k] = s + k < se ? z[s + k] : Wide{0.f, kFloor};
      }
    }
#pragma unroll
    for (int j = 0; j < kPairs; ++j)
      if (s0 + 64 * j + 1 < se) own[j].x = ldf(logits, base + own[j].c, is_bf16);
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const int s = s0 + 64 * j;
      blank_sum += occupancy(x[j][0], y[j][0]);
      if (s + 1 < se) {
        const float g = occupancy(x[j][1], y[j][1]);
        if (own[j].c == blank) blank_sum += g;
        g_r[s + 1] = g;
        x_r[s >> 1] = own[j].x;
      }
    }
  }
  blank_sum = warp_sum(blank_sum);
  __syncwarp();
  const bool huge = fabsf(l) > 0x1p14f;  // the last digit of l is as coarse as those of the softmax that is there
  auto rewrite = [&](int c, float x, float total) {
    if (total != 0.f) stf(grad, base + c, (huge ? ldf(grad, base + c, is_bf16) : __expf(x - l)) - total, is_bf16);
  };
  for (int s = 2 * lane + 1; s < se; s += 64) {
    int q = ln[s];
    if (q < 0) continue;
    float total = g_r[s];
    while (q > 0) {
      total += g_r[q];
      q = ln[q];
      q = q < 0 ? -q - 1 : q;
    }
    rewrite(tg[s >> 1], x_r[s >> 1], total);
  }
  if (lane == 0) rewrite(blank, x_blank, blank_sum);
}

// threads and vectors per thread: the fewest whose registers hold a row (more rows per SM, fewer threads in a reduction, no idle vectors). With 128
// threads for the shortest rows too, 500 sequences of 30 frames, 80 classes, took 63 us a loss (now 50), 200 of 60, 1001 classes, 57 (44).
template <int T, int NV, bool BF16, typename... Args>
void launch_softmax(int vecs, int n_rows, cudaStream_t stream, Args... args) {
  if constexpr (NV < 5 || T < 768) {
    if (vecs > T * NV) {
      constexpr int wider = T == 256 ? 384 : T == 384 ? 768 : 2 * T;
      launch_softmax<NV == 5 ? wider : T, NV == 5 ? (T == 256 ? 4 : 3) : NV + 1, BF16>(vecs, n_rows, stream, args...);
      return;
    }
  }
  ctc_softmax_gather_kernel<T, NV, BF16><<<std::min(n_rows, 148 * (768 / T)), T, 0, stream>>>(args...);
}

}  // namespace

// scratch: at least n_rows * (2 + 6 * (SE + 1)) + batch * (4 + SE) floats, SE = 2 * max_s + 1, 16-byte aligned
RB_EXPORT int rb200_ctc_loss(const void* logits, int is_bf16, const int* cu, const int* row_batch, const int* targets, const int* tgt_lens,
                             float* loss, void* grad, float* scratch, int batch, int n_rows, int V, int s_pitch, int max_s, int blank,
                             long long scratch_floats, cudaStream_t stream) {
  if (batch <= 0) return RB_OK;
  const int SE = 2 * max_s + 1;
  const long long need = (long long)n_rows * (2 + 6LL * (SE + 1)) + (long long)batch * (4 + SE);
  if (scratch_floats < need || (reinterpret_cast<uintptr_t>(scratch) & 15)) {
    rb_set_error("ctc_loss: scratch of %lld floats given, %lld needed (16-byte aligned)", scratch_floats, need);
    return RB_ERR_ARG;
  }
  if (blank < 0 || blank >= V) {
    rb_set_error("ctc_loss: blank index %d outside [0, %d)", blank, V);
    return RB_ERR_ARG;
  }
  // the fewest states per lane whose lattice fits into eight warps per direction, for the longest label sequences 13 (a frame's time grows
  // with the states of a lane)
  using L2 = Lattice<2, 8>;
  using L4 = Lattice<4, 4>;
  using L8 = Lattice<8, 2>;
  const int per_lane = L2::warps(SE) <= 8 ? 2 : L4::warps(SE) <= 8 ? 4 : 8;
  const int warps = per_lane == 2 ? L2::warps(SE) : per_lane == 4 ? L4::warps(SE) : L8::warps(SE);
  auto recursion = per_lane == 2 ? ctc_alpha_beta_kernel<2, 8> : per_lane == 4 ? ctc_alpha_beta_kernel<4, 4> : ctc_alpha_beta_kernel<8, 2>;
  const size_t ring = per_lane == 2 ? L2::kStage : per_lane == 4 ? L4::kStage : 0;
  const size_t smem_ab = (size_t)((SE + 3) & ~3) * sizeof(int) + (4 * (size_t)SE + 2 * warps * kStages * ring) * sizeof(Wide);
  const size_t smem_grad = (size_t)kGradFrames * 2 * SE * sizeof(float);
  if (warps > 13 || smem_ab > 227 * 1024 || smem_grad > 200 * 1024) {
    rb_set_error("ctc_loss: target length %d too large", max_s);
    return RB_ERR_UNSUPPORTED;
  }
  SeqInfo* info = reinterpret_cast<SeqInfo*>(scratch);
  Wide* prob = reinterpret_cast<Wide*>(info + batch);
  Wide* al = prob + (size_t)n_rows * (SE + 1);
  Wide* be = al + (size_t)n_rows * (SE + 1);
  float* lse = reinterpret_cast<float*>(be + (size_t)n_rows * (SE + 1));
  int* wide = reinterpret_cast<int*>(lse + n_rows);
  int* link = wide + n_rows;
  int st;
  if (n_rows > 0) {
    if (is_bf16) launch_softmax<32, 1, true>(V / 8, n_rows, stream, logits, row_batch, cu, targets, tgt_lens, lse, wide, prob, grad, n_rows, V, s_pitch, SE + 1, blank);
    else launch_softmax<32, 1, false>(V / 4, n_rows, stream, logits, row_batch, cu, targets, tgt_lens, lse, wide, prob, grad, n_rows, V, s_pitch, SE + 1, blank);
    st = rb_check_launch("ctc_softmax_gather");
    if (st) return st;
  }
  if (smem_ab > 48 * 1024) cudaFuncSetAttribute(recursion, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_ab);
  recursion<<<batch, 64 * warps, smem_ab, stream>>>(logits, is_bf16, lse, wide, grad, prob, al, be, cu, targets, tgt_lens, info, link, loss, V, s_pitch, SE,
                                                      blank);
  st = rb_check_launch("ctc_alpha_beta");
  if (st) return st;
  if (n_rows > 0 && grad != nullptr) {
    if (smem_grad > 48 * 1024) cudaFuncSetAttribute(ctc_occupancy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_grad);
    ctc_occupancy_kernel<<<(n_rows + kGradFrames - 1) / kGradFrames, 32 * kGradFrames, smem_grad, stream>>>(
        logits, is_bf16, row_batch, targets, tgt_lens, lse, al, be, info, link, grad, n_rows, V, s_pitch, SE, blank);
    st = rb_check_launch("ctc_occupancy");
  }
  return st;
}

namespace {

// out[r, :] = grad[r, :] * dloss[row_batch[r]]: the backward of the loss function scales the gradient that the forward launches
// left behind (one pass instead of an fp32 copy, a multiply and a cast back). Four vectors per thread in flight.
template <bool BF16>
__global__ void __launch_bounds__(256)
ctc_scale_rows_kernel(const void* grad, const int* __restrict__ row_batch, const float* __restrict__ dloss, void* out, int V) {
  using P = Pack<BF16>;
  constexpr int kFlight = 4;
  const int r = blockIdx.x;
  const size_t base = (size_t)r * V;
  const Row row = row_of<BF16>(grad, out, base, V);
  const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(grad) + (base + row.head) * (BF16 ? 2 : 4));
  uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<char*>(out) + (base + row.head) * (BF16 ? 2 : 4));
  const float sc = dloss[row_batch[r]];
  for (int i0 = threadIdx.x; i0 < row.n_vec; i0 += kFlight * blockDim.x) {
    uint4 raw[kFlight];
#pragma unroll
    for (int j = 0; j < kFlight; ++j)
      if (i0 + j * blockDim.x < row.n_vec) raw[j] = src[i0 + j * blockDim.x];
#pragma unroll
    for (int j = 0; j < kFlight; ++j) {
      if (i0 + j * blockDim.x < row.n_vec) {
        float v[P::N];
        P::get(raw[j], v);
#pragma unroll
        for (int k = 0; k < P::N; ++k) v[k] *= sc;
        dst[i0 + j * blockDim.x] = P::put(v);
      }
    }
  }
  for (int i = threadIdx.x; i < row.scalars; i += blockDim.x) {
    const size_t c = base + scalar_at<BF16>(row, i);
    stf(out, c, ldf(grad, c, BF16) * sc, BF16);
  }
}

}  // namespace

// grad, out [n_rows, V] (bf16 or fp32, may be the same buffer), row_batch [n_rows], dloss [B] fp32
RB_EXPORT int rb200_ctc_scale_rows(const void* grad, const int* row_batch, const float* dloss, void* out, int n_rows, int V, int is_bf16,
                                   cudaStream_t stream) {
  if (n_rows <= 0 || V <= 0) return RB_OK;
  if (is_bf16) ctc_scale_rows_kernel<true><<<n_rows, 256, 0, stream>>>(grad, row_batch, dloss, out, V);
  else ctc_scale_rows_kernel<false><<<n_rows, 256, 0, stream>>>(grad, row_batch, dloss, out, V);
  return rb_check_launch("ctc_scale_rows");
}

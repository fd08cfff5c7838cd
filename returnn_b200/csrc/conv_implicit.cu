// 3x3 convolutions over (time, feature) of the subsampling frontend without patch matrices, on the tensor cores (sm_100a): forward pass, data gradient
// and filter gradient for 32 or 64 channels on either side.
//
// A frame is F rows (feature positions) of C channels. For one tap (kt, kf) the rows of the patch matrix that belong to an output frame are the rows
// of ONE input frame, shifted by kf - 1: a box of F rows that TMA reads in place, with zeros outside [0, F); a frame that does not exist
// (padding in time, past a sequence's length, between the steps of a stride) is a box past the last frame, which is zeros too.
//
//   conv_kernel    D[frames x F, N] = sum over taps A_tap[frames x F, C] W_tap[N, C]^T: a tile is as many frames as fit 128 rows, the filter stays
//                  in shared memory, the epilogue adds bias and ReLU, or multiplies with relu'(z). The data gradient is the same product with
//                  the flipped filter; a tile's frames then have the same phase of the stride, so that they share the taps that exist.
//   wgrad_kernel   D[9 C, N] += X_tap[F, 9 C]^T dY[F, N] frame by frame, all nine taps accumulate in tensor memory (3 or 5 tiles of 128 rows); a CTA
//                  adds its sum to the output once. Frames are padded to a multiple of 16 rows (zero rows of dY).
//
// With patch matrices the frontend of 36 x 2000 frames x 80 features (32, 64, 64 channels, strides 3 and 2) moved 870 MB five times: written,
// read by two products, and for the data gradients written by a product and read by the sum over patches. Times there (40 to 100 % of the frames
// valid), patch matrices -> here: second layer forward 260 -> 68 us, data gradient 300 -> 93, filter gradient 109 -> 73; third layer 195 -> 48,
// 232 -> 71, 71 -> 47; 8 x 1000 frames 36 -> 14, 39 -> 16, 17 -> 16; one sequence of 300: 9.0 -> 7.8, 10.5 -> 6.8, 9.7 -> 8.7. The forward pass is
// bound by the copies (about 1.9 cycles per row of 64 or 128 bytes, nine rows per position), the data gradient by the writes of the input's
// gradient (184 MB: 28 us) and the fixed time of a tile, the filter gradient by its copies (nine boxes of 48 rows a frame) and the final atomics.
#include "tcgen05.cuh"
#include <cstring>

using namespace rbt;

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kThreads = 320;  // producer, issuer, eight epilogue warps

struct Conv {
  const int *lens_in, *lens_out, *cu, *row_batch, *row_pos;
  const bf16* relu_z;
  const float* bias;
  bf16* y;
  float *dw, *sums;
  int* status;
  int T, To, F, stride, pad, n_frames, src_frames, tiles, nt, groups, fk;
};

// operand descriptors (upper word): rows of 128 or of 64 bytes, both swizzled over their length; groups of 8 rows follow each other
template <int C>
__host__ __device__ constexpr uint32_t desc_hi() {
  return C == 64 ? ((1024u >> 4) | (1u << 14) | (2u << 29)) : ((512u >> 4) | (1u << 14) | (4u << 29));
}
template <uint32_t HI_A, uint32_t HI_B>
__device__ __forceinline__ void umma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %6};\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
      ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(accumulate), "n"(HI_A), "n"(HI_B)
      : "memory");
}

// a tile of the data gradient: frames t0, t0 + stride, ... of a sequence
struct BackTile {
  int b, t0, taps;  // taps: bit kt is set where output frames can meet this phase
  __device__ __forceinline__ BackTile(const Conv& p, int tile) {
    const int per = p.stride * p.groups;
    b = tile / per;
    const int r = tile - b * per, ph = r / p.groups;
    t0 = ph + p.stride * p.nt * (r - ph * p.groups);
    taps = 0;
#pragma unroll
    for (int kt = 0; kt < 3; ++kt)
      if ((ph + p.pad - kt + 3 * p.stride) % p.stride == 0) taps |= 1 << kt;
  }
};

// frame of the operand that frame i of a tile meets at tap kt; src_frames (a box of zeros) where there is none
template <bool BACK>
__device__ __forceinline__ int source(const Conv& p, int tile, int i, int kt) {
  if (BACK) {
    const BackTile w(p, tile);
    const int t = w.t0 + i * p.stride, num = t + p.pad - kt;
    if (t >= min(p.lens_in[w.b], p.T) || num < 0 || num % p.stride) return p.src_frames;
    const int to = num / p.stride;
    if (to >= min(p.lens_out[w.b], p.To)) return p.src_frames;
    return p.cu ? p.cu[w.b] + to : w.b * p.To + to;
  }
  const int fr = tile * p.nt + i;
  if (fr >= p.n_frames) return p.src_frames;
  const int b = p.row_batch ? p.row_batch[fr] : fr / p.To, to = p.row_batch ? p.row_pos[fr] : fr % p.To;
  const int t = to * p.stride - p.pad + kt;
  return t >= 0 && t < min(p.lens_in[b], p.T) ? b * p.T + t : p.src_frames;
}

struct Bars {
  uint64_t *full, *empty, *acc_full, *acc_empty, *extra;
  uint32_t* slot;
  volatile int* abort_flag;
};
constexpr int kMaxStages = 6;

__device__ __forceinline__ Bars bars_at(uint8_t* at) {
  Bars s;
  s.full = reinterpret_cast<uint64_t*>(at);
  s.empty = s.full + kMaxStages;
  s.acc_full = s.empty + kMaxStages;
  s.acc_empty = s.acc_full + 2;
  s.extra = s.acc_empty + 2;
  s.slot = reinterpret_cast<uint32_t*>(s.extra + 1);
  s.abort_flag = reinterpret_cast<volatile int*>(s.slot + 1);
  return s;
}
template <uint32_t COLS>
__device__ __forceinline__ uint32_t begin(const Bars& s, int stages, int acc_arrivals) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.acc_full[i], 1);
      mbar_init(&s.acc_empty[i], acc_arrivals);
    }
    mbar_init(s.extra, 1);
    *s.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x >> 5 == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s.slot)), "r"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return *s.slot;
}
template <uint32_t COLS>
__device__ __forceinline__ void end(const Bars& s, uint32_t tmem) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*s.abort_flag && threadIdx.x == 0) {
    // let copies that are still in flight land before the shared memory goes away (bounded: about 1 ms)
    for (uint32_t i = 0; i < (1u << 12); ++i) __nanosleep(256);
  }
  __syncthreads();
  if (threadIdx.x >> 5 == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS) : "memory");
  }
}
// by a whole warp; raises the abort flag when it gives up
__device__ __forceinline__ bool wait_warp(const Conv& p, const Bars& s, uint64_t* bar, uint32_t parity, int code) {
  if (warp_wait(bar, parity, s.abort_flag)) return true;
  *s.abort_flag = 1;
  if (p.status && (threadIdx.x & 31) == 0) atomicCAS(p.status, 0, code << 24 | 1);
  return false;
}

// A stage holds the three taps of one kt: waiting for a stage, announcing its bytes and starting copies takes the loading warp about 500 cycles, a
// tap of 128 rows 230 (forward pass as below, a stage per tap: 155 us)
template <int C, int N>
struct ConvLayout {
  static constexpr int kBox = 128 * C * 2, kStage = 3 * kBox, kStages = C == 32 ? 4 : N == 32 ? 3 : 2, kRing = kStage * kStages;
  static_assert(kStages <= kMaxStages, "ring");
  static constexpr int kTable = 10240;  // bytes: tiles that are looked up at a time (see conv_kernel)
  static constexpr int kPitch = N * 2 + 16;  // of a row of the staging area (no bank conflicts)
  static constexpr int kSmem = kRing + N * 9 * C * 2 + 8 * 32 * kPitch + kTable + N * 4 + 256 + 1024;
};

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

template <int C, int N, bool BACK>
__global__ void __launch_bounds__(kThreads, 1)
conv_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_run, const __grid_constant__ CUtensorMap tm_w, const Conv p) {
  using L = ConvLayout<C, N>;
  constexpr int kTap = N * C * 2;  // bytes of the filter of a tap
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sw = ring + L::kRing;
  uint8_t* staging = sw + 9 * kTap;
  float* sbias = reinterpret_cast<float*>(staging + 8 * 32 * L::kPitch);
  int* table = reinterpret_cast<int*>(sbias + N);
  const Bars s = bars_at(reinterpret_cast<uint8_t*>(table) + L::kTable);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)threadIdx.x < N) sbias[threadIdx.x] = !BACK && p.bias ? p.bias[threadIdx.x] : 0.f;  // (data gradient: the column sums)
  const uint32_t tmem = begin<256>(s, L::kStages, 4);
  // What the roles have to know of a tile is looked up by all threads for as many tiles as the table holds: { taps with a frame (none: its rows are zeros), first
  // output frame, frames of it, frames of the operand [3][nt] }. One warp looking up eight tiles ahead waited for its loads and divisions longer
  // than a tile takes. Where the frames of a tap form a run (frame + i, or + i * stride in the forward pass), bit 3 + kt of the taps is set, and the run
  // is one copy: a box per frame takes the loading warp about 240 cycles to issue. 36 x 2000 frames (40 to 100 % valid), 32 -> 64 channels, stride 3,
  // forward pass and data gradient: 198 and 285 us, with the table 183 and 181, with runs 155 and 135, with three taps to a stage 68 and 93.
  const int entry = 3 + 3 * p.nt, batch = L::kTable / 4 / entry;
  const int mine = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles of this CTA
  const int bytes = p.nt * p.F * C * 2;
  const int q = warp & 3, set = (warp - 2) >> 2;  // epilogue: the two sets of four warps take the tiles in turn
  const int row = q * 32 + lane, fi = row / p.F, f = row - fi * p.F;
  uint8_t* box = staging + (warp - 2) * 32 * L::kPitch;
  uint32_t st = 0, ph = 0;  // (loading and issuing warp) stage of the ring
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // (epilogue of the data gradient) of the eight columns that this lane stores
  bool ok = true;
  if (warp == 0 && elect_one()) {
    mbar_expect_tx(s.extra, 9 * kTap);
    for (int j = 0; j < 9; ++j) tma_load_2d(sw + j * kTap, &tm_w, j * C, 0, s.extra);
  }
  if (warp == 1) ok = wait_warp(p, s, s.extra, 0, 42);
  for (int from = 0; from < mine; from += batch) {
    const int n = min(batch, mine - from);
    __syncthreads();
    for (int i = threadIdx.x; i < n * entry; i += kThreads) {
      const int k = i / entry, j = i - k * entry, tile = (int)blockIdx.x + (from + k) * (int)gridDim.x;
      int v;
      if (j >= 3) v = source<BACK>(p, tile, (j - 3) % p.nt, (j - 3) / p.nt);
      else if (BACK) {
        const BackTile w(p, tile);
        v = j == 0 ? w.taps : j == 1 ? w.b * p.T + w.t0 : min(p.nt, (p.T - w.t0 + p.stride - 1) / p.stride);
      } else {
        v = j == 0 ? 7 : j == 1 ? tile * p.nt : min(p.nt, p.n_frames - tile * p.nt);
      }
      table[i] = v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * 3; i += kThreads) {
      int* e = table + i / 3 * entry;
      int* fr = e + 3 + i % 3 * p.nt;
      const int f0 = fr[0], step = BACK ? 1 : p.stride;
      bool any = f0 < p.src_frames, run = any && p.nt > 1 && (BACK || f0 / p.stride + p.nt <= p.src_frames / p.stride);
      for (int j = 1; j < p.nt; ++j) {
        any = any || fr[j] < p.src_frames;
        run = run && fr[j] == f0 + j * step;
      }
      if (!any) atomicAnd(e, ~(1 << i % 3));
      if (run) {
        if (!BACK) {  // (the frames seen as [frames / stride][stride])
          fr[0] = f0 % p.stride;
          fr[1] = f0 / p.stride;
        }
        atomicOr(e, 8 << i % 3);
      }
    }
    __syncthreads();
    if (warp == 0) {
      for (int k = 0; k < n && ok; ++k) {
        const int* e = table + k * entry;
        const int taps = e[0];
        for (int kt = 0; kt < 3 && ok; ++kt) {
          if (!(taps >> kt & 1)) continue;
          const bool run = taps >> (3 + kt) & 1;
          const int f0 = e[3 + kt * p.nt], f1 = run ? e[4 + kt * p.nt] : 0;
          ok = wait_warp(p, s, &s.empty[st], ph ^ 1u, 41);
          if (!ok) break;
          if (elect_one()) {
            uint8_t* dst = ring + st * L::kStage;
            mbar_expect_tx(&s.full[st], 3 * bytes);
            if (run) {
#pragma unroll
              for (int kf = 0; kf < 3; ++kf) {
                if (BACK) tma_load_3d(dst + kf * L::kBox, &tm_run, 0, 1 - kf, f0, &s.full[st]);
                else tma_load_4d(dst + kf * L::kBox, &tm_run, 0, kf - 1, f0, f1, &s.full[st]);
              }
            } else {
              for (int i = 0; i < p.nt; ++i) {
                const int fr = e[3 + kt * p.nt + i];
#pragma unroll
                for (int kf = 0; kf < 3; ++kf) tma_load_3d(dst + kf * L::kBox + i * p.F * C * 2, &tm_x, 0, BACK ? 1 - kf : kf - 1, fr, &s.full[st]);
              }
            }
          }
          __syncwarp();
          if (++st == L::kStages) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    } else if (warp == 1) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      const uint32_t a0 = desc_lo(smem_u32(ring), 16), b0 = desc_lo(smem_u32(sw), 16);
      for (int k = 0; k < n && ok; ++k) {
        const int taps = table[k * entry];
        const uint32_t local = from + k, buf = local & 1u;
        ok = wait_warp(p, s, &s.acc_empty[buf], ((local >> 1) & 1u) ^ 1u, 43);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bool first = true;
        for (int kt = 0; kt < 3 && ok; ++kt) {
          if (!(taps >> kt & 1)) continue;
          ok = wait_warp(p, s, &s.full[st], ph, 44);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = a0 + st * (L::kStage >> 4), b = b0 + kt * 3 * (kTap >> 4);
#pragma unroll
          for (int kf = 0; kf < 3; ++kf)
#pragma unroll
            for (int kk = 0; kk < C / 16; ++kk)
              umma<desc_hi<C>(), desc_hi<C>()>(tmem + buf * 128, a + kf * (L::kBox >> 4) + 2 * kk, b + kf * (kTap >> 4) + 2 * kk, idesc,
                                               first && kf == 0 && kk == 0 ? 0u : 1u);
          first = false;
          umma_commit_warp(&s.empty[st]);
          if (++st == L::kStages) {
            st = 0;
            ph ^= 1u;
          }
        }
        if (ok) umma_commit_warp(&s.acc_full[buf]);  // (a tile without taps: nothing to wait for)
      }
    } else {
      for (int k = 0; k < n && ok; ++k) {
        const uint32_t local = from + k;
        if ((local & 1u) != (uint32_t)set) continue;
        const int* e = table + k * entry;
        const bool none = (e[0] & 7) == 0;
        const int out = fi < e[2] ? (e[1] + fi * (BACK ? p.stride : 1)) * p.F + f : -1;  // row of the output
        ok = wait_warp(p, s, &s.acc_full[set], (local >> 1) & 1u, 45);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t t_addr = tmem + set * 128 + ((uint32_t)(q * 32) << 16);
        uint32_t r[N];
#pragma unroll
        for (int c = 0; c < N; c += 32) tmem_ld32(t_addr + c, r + c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&s.acc_empty[set])) : "memory");
#pragma unroll
        for (int c = 0; c < N; c += 8) {
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            v[j] = none ? 0.f : __uint_as_float(r[c + j]);
            if (!BACK) v[j] = fmaxf(v[j] + sbias[c + j], 0.f);
          }
          uint4 o;
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          *reinterpret_cast<uint4*>(box + lane * L::kPitch + c * 2) = o;
        }
        __syncwarp();
        constexpr int kPer = N / 8;  // lanes to a row
        int to[kPer];
        uint4 z[kPer];
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
          to[i] = __shfl_sync(0xffffffffu, out, i * (32 / kPer) + lane / kPer);
          if (BACK && p.relu_z && to[i] >= 0) z[i] = *reinterpret_cast<const uint4*>(p.relu_z + (size_t)to[i] * N + lane % kPer * 8);
        }
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
          if (to[i] < 0) continue;
          uint4 o = *reinterpret_cast<const uint4*>(box + (i * (32 / kPer) + lane / kPer) * L::kPitch + lane % kPer * 16);
          if (BACK && p.relu_z) {
            const __nv_bfloat162* zh = reinterpret_cast<const __nv_bfloat162*>(&z[i]);
            uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 zf = __bfloat1622float2(zh[j]);
              ow[j] = (zf.x > 0.f ? ow[j] & 0xffffu : 0u) | (zf.y > 0.f ? ow[j] & 0xffff0000u : 0u);
            }
          }
          *reinterpret_cast<uint4*>(p.y + (size_t)to[i] * N + lane % kPer * 8) = o;
          if (BACK && p.sums) {
            const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[j] += __uint_as_float(j & 1 ? ow[j >> 1] & 0xffff0000u : ow[j >> 1] << 16);
          }
        }
        __syncwarp();
      }
    }
  }
  if (BACK && p.sums) {
    if (warp >= 2) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int o = 16; o >= N / 8; o >>= 1) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
        if (lane < N / 8) atomicAdd(&sbias[lane * 8 + j], sum[j]);
      }
    }
    __syncthreads();
    if ((int)threadIdx.x < N) atomicAdd(p.sums + threadIdx.x, sbias[threadIdx.x]);
  }
  end<256>(s, tmem);
}

// Bytes of a frame in the ring: nine taps and dY, padded to fk rows. Behind the last stage: what the groups of the last tile past the ninth tap read
__host__ __device__ constexpr int wgrad_stage(int c, int n, int fk) { return fk * 2 * (9 * c + n); }
__host__ __device__ constexpr int wgrad_tail(int c, int n, int fk) { return fk * 2 * (c == 32 ? 3 * c - n : c - n); }
constexpr int kWgradSmem = 227 * 1024;
__host__ __device__ constexpr int wgrad_stages(int c, int n, int fk) {
  const int k = (kWgradSmem - 2048 - wgrad_tail(c, n, fk)) / wgrad_stage(c, n, fk);
  return k > 6 ? 6 : k;
}

template <int C, int N>
__global__ void __launch_bounds__(kThreads, 1)
wgrad_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_dy, const Conv p) {
  constexpr int kPerTile = 128 / C, kTiles = (9 + kPerTile - 1) / kPerTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int tap = p.fk * C * 2, stage = wgrad_stage(C, N, p.fk), stages = wgrad_stages(C, N, p.fk);
  const Bars s = bars_at(ring + stages * stage + wgrad_tail(C, N, p.fk));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem = begin<512>(s, stages, 1);
  if (warp == 0) {
    uint32_t st = 0, ph = 0;
    bool ok = true;
    int src[3] = {0, 0, 0}, at = 32;
    for (int fr = blockIdx.x; fr < p.n_frames && ok; fr += gridDim.x) {
      if (at == 32) {  // a lane looks up a frame
        const long long mine = fr + (long long)lane * gridDim.x;
#pragma unroll
        for (int kt = 0; kt < 3; ++kt) src[kt] = mine < p.n_frames ? source<false>(p, (int)mine, 0, kt) : p.src_frames;
        at = 0;
      }
      int from[3];
#pragma unroll
      for (int kt = 0; kt < 3; ++kt) from[kt] = __shfl_sync(0xffffffffu, src[kt], at);
      ++at;
      ok = wait_warp(p, s, &s.empty[st], ph ^ 1u, 46);
      if (!ok) break;
      if (elect_one()) {
        uint8_t* dst = ring + st * stage;
        mbar_expect_tx(&s.full[st], stage);
        tma_load_3d(dst + 9 * tap, &tm_dy, 0, 0, fr, &s.full[st]);
#pragma unroll
        for (int j = 0; j < 9; ++j) tma_load_3d(dst + j * tap, &tm_x, 0, j % 3 - 1, from[j / 3], &s.full[st]);
      }
      __syncwarp();
      if (++st == (uint32_t)stages) {
        st = 0;
        ph ^= 1u;
      }
    }
  } else if (warp == 1) {
    // both operands have their rows (positions) along K
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    uint32_t st = 0, ph = 0;
    bool ok = true, first = true;
    for (int fr = blockIdx.x; fr < p.n_frames; fr += gridDim.x) {
      ok = wait_warp(p, s, &s.full[st], ph, 47);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t base = smem_u32(ring) + st * stage;
      const uint32_t b0 = desc_lo(base + 9 * tap, tap);
      for (int k = 0; k < p.fk / 16; ++k) {
#pragma unroll
        for (int m = 0; m < kTiles; ++m)
          umma<desc_hi<C>(), desc_hi<N>()>(tmem + m * N, desc_lo(base + m * kPerTile * tap, tap) + k * (16 * C * 2 >> 4), b0 + k * (16 * N * 2 >> 4), idesc,
                                           first ? 0u : 1u);
        first = false;
      }
      umma_commit_warp(&s.empty[st]);
      if (++st == (uint32_t)stages) {
        st = 0;
        ph ^= 1u;
      }
    }
    if (ok) umma_commit_warp(&s.acc_full[0]);
  } else if ((int)blockIdx.x < p.n_frames) {
    const int q = warp & 3, set = (warp - 2) >> 2;
    if (wait_warp(p, s, &s.acc_full[0], 0, 48)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int m = set; m < kTiles; m += 2) {
        uint32_t r[N];
#pragma unroll
        for (int c = 0; c < N; c += 32) tmem_ld32(tmem + m * N + c + ((uint32_t)(q * 32) << 16), r + c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int row = m * 128 + q * 32 + lane;  // tap * C + channel of x
        if (row < 9 * C) {
#pragma unroll
          for (int c = 0; c < N; ++c) atomicAdd(p.dw + c * 9 * C + row, __uint_as_float(r[c]));
        }
      }
    }
  }
  end<512>(s, tmem);
}

// frames of F rows of C channels; boxes of `rows` rows of a frame. run > 1: of as many frames, which are `stride` frames apart (stride > 1: a
// coordinate more, frames are [frames / stride][stride])
int frames_map(CUtensorMap* map, const void* base, int c, int f, long long frames, int rows, int run = 1, int stride = 1, bool split = false) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) {
    rb_set_error("conv3x3: cuTensorMapEncodeTiled not available");
    return RB_ERR_UNSUPPORTED;
  }
  const cuuint64_t frame = (cuuint64_t)c * f * 2;
  cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)f, (cuuint64_t)(split ? stride : frames), (cuuint64_t)(frames / stride)};
  cuuint64_t strides[3] = {(cuuint64_t)c * 2, frame, frame * stride};
  cuuint32_t box[4] = {(cuuint32_t)c, (cuuint32_t)rows, (cuuint32_t)(split ? 1 : run), (cuuint32_t)run};
  cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult r = encode_in_context([&]() {
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, split ? 4 : 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              c == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) {
    rb_set_error("conv3x3: cuTensorMapEncodeTiled failed (%d): base %p channels %d features %d frames %lld", (int)r, base, c, f, frames);
    return RB_ERR_ARG;
  }
  return RB_OK;
}

template <int C, int N, bool BACK>
int launch_conv(const CUtensorMap& tm_x, const CUtensorMap& tm_run, const void* w, const Conv& p, cudaStream_t stream) {
  CUtensorMap tm_w;
  int st = make_map(&tm_w, w, 9 * C, N, 9 * C, C, N, false, C == 32);
  if (st) return st;
  constexpr int smem = ConvLayout<C, N>::kSmem;
  static_assert(smem <= 227 * 1024, "shared memory");
  static RbPerDevice attr_set;
  if (attr_set.needed()) {
    cudaError_t e = cudaFuncSetAttribute(conv_kernel<C, N, BACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      rb_set_error("conv3x3: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return RB_ERR_LAUNCH;
    }
    attr_set.done();
  }
  const int grid = p.tiles < num_sms() ? p.tiles : num_sms();
  conv_kernel<C, N, BACK><<<grid, kThreads, smem, stream>>>(tm_x, tm_run, tm_w, p);
  return rb_check_launch("conv3x3");
}

template <int C, int N>
int launch_wgrad(const CUtensorMap& tm_x, const CUtensorMap& tm_dy, const Conv& p, cudaStream_t stream) {
  static RbPerDevice attr_set;
  if (attr_set.needed()) {
    cudaError_t e = cudaFuncSetAttribute(wgrad_kernel<C, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgradSmem);
    if (e != cudaSuccess) {
      rb_set_error("conv3x3_wgrad: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
      return RB_ERR_LAUNCH;
    }
    attr_set.done();
  }
  const int smem = wgrad_stages(C, N, p.fk) * wgrad_stage(C, N, p.fk) + wgrad_tail(C, N, p.fk) + 2048;
  const int grid = p.n_frames < num_sms() ? p.n_frames : num_sms();
  wgrad_kernel<C, N><<<grid, kThreads, smem, stream>>>(tm_x, tm_dy, p);
  return rb_check_launch("conv3x3_wgrad");
}

bool channels_ok(int c) { return c == 32 || c == 64; }

int check(const char* name, const void* a, const void* b, const void* c, long long rows, int f, int ci, int co, int stride, int pad) {
  auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!channels_ok(ci) || !channels_ok(co) || f <= 0 || f % 8 || f > 80) {
    rb_set_error("%s: %d and %d channels, %d features", name, ci, co, f);
    return RB_ERR_UNSUPPORTED;
  }
  if (!al(a) || !al(b) || !al(c) || rows >= 0x7fffffffLL || stride <= 0 || pad < 0 || pad > 2) {
    rb_set_error("%s: pointers %p %p %p (16-byte aligned?), %lld rows, stride %d, padding %d", name, a, b, c, rows, stride, pad);
    return RB_ERR_ARG;
  }
  return RB_OK;
}

}  // namespace

// channels of both sides (32 or 64) and features (a multiple of 8: boxes start on a group of 8 rows; at most 80: two frames of a filter gradient in
// shared memory) that the kernels below take
RB_EXPORT int rb200_conv3x3_supported(int f, int c, int n) { return channels_ok(c) && channels_ok(n) && f > 0 && f % 8 == 0 && f <= 80 ? 1 : 0; }

// back == 0: y [n_frames, F, n] = relu(conv(x [B, T, F, c], w [n, (kt, kf, c)]) + bias) at the output frames (row_batch, row_pos), or at all B x To
//            (row_batch null); input frames at or past lens_in[b] are zeros.
// back == 1: y [B, T, F, n] = data gradient of that convolution (n its input channels, c its output channels), x = dY, w [n, (kt, kf, c)] the filter with
//            its channels exchanged; dY [n_frames, F, c]: frame cu[b] + to, or b * To + to (cu null), frames at or past lens_out[b] give nothing;
//            zeros at or past lens_in[b]; times relu'(relu_z) if that is given.
//            sums (may be null) [n] += the column sums of y.
RB_EXPORT int rb200_conv3x3(const void* x, const void* w, const float* bias, const void* relu_z, void* y, float* sums, const int* lens_in, const int* lens_out, const int* cu,
                            const int* row_batch, const int* row_pos, int B, int T, int To, int F, int c, int n, int stride, int pad, long long n_frames,
                            int back, int* status, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || To <= 0 || (!back && n_frames <= 0)) return RB_OK;
  const long long out_frames = back ? (long long)B * T : n_frames, in_frames = back ? n_frames : (long long)B * T;
  int st = check("conv3x3", x, w, y, (out_frames > in_frames ? out_frames : in_frames) * F, F, c, n, stride, pad);
  if (st) return st;
  if (reinterpret_cast<uintptr_t>(relu_z) & 15) {
    rb_set_error("conv3x3: relu_z %p is not 16-byte aligned", relu_z);
    return RB_ERR_ARG;
  }
  if (in_frames <= 0) {
    cudaMemsetAsync(y, 0, (size_t)out_frames * F * n * 2, stream);
    return rb_check_launch("conv3x3");
  }
  Conv p;
  memset(&p, 0, sizeof(p));
  p.lens_in = lens_in; p.lens_out = lens_out; p.cu = cu; p.row_batch = row_batch; p.row_pos = row_pos;
  p.relu_z = (const bf16*)relu_z; p.bias = bias; p.y = (bf16*)y; p.sums = sums; p.status = status;
  p.T = T; p.To = To; p.F = F; p.stride = stride; p.pad = pad; p.n_frames = (int)out_frames; p.src_frames = (int)in_frames;
  p.nt = 128 / F < 10 ? 128 / F : 10;  // (three taps in time of a tile's frames fit a warp)
  p.groups = ((T + stride - 1) / stride + p.nt - 1) / p.nt;
  const long long tiles = back ? (long long)B * stride * p.groups : (n_frames + p.nt - 1) / p.nt;
  if (tiles >= 0x7fffffffLL) {
    rb_set_error("conv3x3: %lld tiles", tiles);
    return RB_ERR_ARG;
  }
  p.tiles = (int)tiles;
  CUtensorMap tm_x, tm_run;
  st = frames_map(&tm_x, x, c, F, in_frames, F);
  tm_run = tm_x;
  if (!st && p.nt > 1 && (back || in_frames >= stride)) st = frames_map(&tm_run, x, c, F, in_frames, F, p.nt, back ? 1 : stride, !back);
  if (st) return st;
#define RB_CONV(C, N) (back ? launch_conv<C, N, true>(tm_x, tm_run, w, p, stream) : launch_conv<C, N, false>(tm_x, tm_run, w, p, stream))
  if (c == 32) return n == 32 ? RB_CONV(32, 32) : RB_CONV(32, 64);
  return n == 32 ? RB_CONV(64, 32) : RB_CONV(64, 64);
#undef RB_CONV
}

// dw [n, (kt, kf, c)] (fp32) += filter gradient of the convolution above; dy [n_frames, F, n]
RB_EXPORT int rb200_conv3x3_wgrad(const void* x, const void* dy, float* dw, const int* lens_in, const int* row_batch, const int* row_pos, int B, int T, int To,
                                  int F, int c, int n, int stride, int pad, long long n_frames, int* status, cudaStream_t stream) {
  if (B <= 0 || T <= 0 || To <= 0 || n_frames <= 0) return RB_OK;
  const long long in_frames = (long long)B * T;
  int st = check("conv3x3_wgrad", x, dy, dw, (n_frames > in_frames ? n_frames : in_frames) * F, F, c, n, stride, pad);
  if (st) return st;
  Conv p;
  memset(&p, 0, sizeof(p));
  p.lens_in = lens_in; p.row_batch = row_batch; p.row_pos = row_pos; p.dw = dw; p.status = status;
  p.T = T; p.To = To; p.F = F; p.stride = stride; p.pad = pad; p.n_frames = (int)n_frames; p.src_frames = (int)in_frames;
  p.nt = 1;
  p.fk = (F + 15) / 16 * 16;
  CUtensorMap tm_x, tm_dy;
  st = frames_map(&tm_x, x, c, F, in_frames, p.fk);
  if (st) return st;
  st = frames_map(&tm_dy, dy, n, F, n_frames, p.fk);
  if (st) return st;
  if (c == 32) return n == 32 ? launch_wgrad<32, 32>(tm_x, tm_dy, p, stream) : launch_wgrad<32, 64>(tm_x, tm_dy, p, stream);
  return n == 32 ? launch_wgrad<64, 32>(tm_x, tm_dy, p, stream) : launch_wgrad<64, 64>(tm_x, tm_dy, p, stream);
}

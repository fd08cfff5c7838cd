// Log-mel filterbank features from raw audio in one kernel: framing, window, real FFT of 256, 512 or 1024 points in fp32, power spectrum, mel
// projection, log. Nothing but the audio is read and nothing but the features is written.
//
// Half a warp transforms one frame: the real frame of n_fft samples is a complex sequence z[n] = x[2n] + i x[2n+1] of M = n_fft / 2 = 16 E
// points, n = l + 16 i for lane l. Two passes with one exchange through shared memory between them: E-point transforms over i in the
// registers of every lane, twiddle W_M^(l j), 16-point transforms over l by the lane that owns residue j; k = j + E q. The spectrum of the
// real frame comes from Z[k] and Z[M-k], which for E = 16 lie in two lanes (two shuffles per pair) and else in the exchange buffer.
// A CTA of eight warps computes the power spectra of kTile = 32 consecutive frames into shared memory as [bin][frame]; then a lane is a
// frame, so the mel sums read one row of the array per bin without bank conflicts and the filter weights as broadcasts (with a lane per
// filter the lanes' ranges start anywhere: several conflicts per read). The features of a tile are one contiguous piece of the output.
//
// Bound by the instructions and the shared-memory accesses of the transform (36 us of 58 at 64 utterances of 10 s, 64 k frames; the mel sums
// take 14; DRAM 8 % busy, 61 MB); two or three CTAs per SM make no difference. The transform as a matrix product on the tensor cores (mel.cu)
// takes 79 GFLOP for fp32 precision there and moves the spectrum through memory twice: 147 us, error 6e-7 against 64 bits, here 1.7e-7.
#include <algorithm>
#include "common.cuh"

namespace {

constexpr int kWarps = 8;
constexpr int kTile = 32;   // frames per tile = lanes of the mel sums
constexpr int kPitch = 33;  // floats per bin of the power array: the lanes of the transform write a column of it, the mel sums read a row

struct __align__(8) C2 {
  float x, y;
};
// sum and difference of both parts in one instruction (the difference as a + b * -1, which rounds once, like a - b)
__device__ __forceinline__ unsigned long long bits(C2 a) { return ((unsigned long long)__float_as_uint(a.y) << 32) | __float_as_uint(a.x); }
__device__ __forceinline__ C2 value(unsigned long long u) { return {__uint_as_float((uint32_t)u), __uint_as_float((uint32_t)(u >> 32))}; }
__device__ __forceinline__ C2 operator+(C2 a, C2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits(a)), "l"(bits(b)));
  return value(r);
}
__device__ __forceinline__ C2 operator-(C2 a, C2 b) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(bits(b)), "l"(0xBF800000BF800000ull), "l"(bits(a)));
  return value(r);
}
__device__ __forceinline__ C2 cmul(C2 a, C2 b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }

// cos(2 pi k / 32), k = 0 .. 8
__host__ __device__ constexpr float cos32_octant(int k) {
  return k == 0 ? 1.f : k == 1 ? 0.980785280403230449f : k == 2 ? 0.923879532511286756f : k == 3 ? 0.831469612302545237f :
         k == 4 ? 0.707106781186547524f : k == 5 ? 0.555570233019602225f : k == 6 ? 0.382683432365089772f : k == 7 ? 0.195090322016128268f : 0.f;
}
__host__ __device__ constexpr float cos32(int k) {
  k &= 31;
  return k <= 8 ? cos32_octant(k) : k <= 16 ? -cos32_octant(16 - k) : k <= 24 ? -cos32_octant(k - 16) : cos32_octant(32 - k);
}
// a * exp(-2 pi i k / N), N a power of two up to 32; k is known when the loops are unrolled
template <int N>
__device__ __forceinline__ C2 rotate(C2 a, int k) {
  const int t = (k * (32 / N)) & 31;
  if (t == 0) return a;
  if (t == 8) return {a.y, -a.x};
  if (t == 16) return {-a.x, -a.y};
  if (t == 24) return {-a.y, a.x};
  const float c = cos32(t), s = cos32(t + 24);  // sin(t) = cos(t - 8)
  return {a.x * c + a.y * s, a.y * c - a.x * s};
}

// in-place transform of N values in registers, result in natural order: N = N1 * N2, N2-point transforms over every N1-th value, rotation,
// N1-point transforms
template <int N>
__device__ __forceinline__ void fft(C2 (&a)[N]) {
  if constexpr (N == 2) {
    const C2 t = a[0];
    a[0] = t + a[1];
    a[1] = t - a[1];
  } else if constexpr (N == 4) {
    const C2 s02 = a[0] + a[2], d02 = a[0] - a[2], s13 = a[1] + a[3], d13 = a[1] - a[3];
    a[0] = s02 + s13;
    a[2] = s02 - s13;
    a[1] = {d02.x + d13.y, d02.y - d13.x};
    a[3] = {d02.x - d13.y, d02.y + d13.x};
  } else {
    constexpr int N2 = 4, N1 = N / N2;
    C2 u[N1][N2];
#pragma unroll
    for (int c = 0; c < N1; ++c) {
      C2 b[N2];
#pragma unroll
      for (int r = 0; r < N2; ++r) b[r] = a[c + N1 * r];
      fft<N2>(b);
#pragma unroll
      for (int k = 0; k < N2; ++k) u[c][k] = rotate<N>(b[k], c * k);
    }
#pragma unroll
    for (int k = 0; k < N2; ++k) {
      C2 b[N1];
#pragma unroll
      for (int c = 0; c < N1; ++c) b[c] = u[c][k];
      fft<N1>(b);
#pragma unroll
      for (int q = 0; q < N1; ++q) a[k + N2 * q] = b[q];
    }
  }
}

struct Mel {
  const float* audio;
  const int* lens;
  long long T;  // samples from one row to the next
  int rows, n_frames_max, window, step, tiles;
  const float* win;      // [window]
  const float* weights;  // [max_len, n_mel]: entry i of filter m is the filterbank's [fb_start[m] + i, m]
  const int* fb_start;
  const int* fb_len;
  int max_len, len4, n_mel;
  float log_scale, eps;
  float* out;  // [rows, n_frames_max, n_mel]
  int quads;   // frames of features start on a 16-byte boundary
  int pairs;   // the window is even and every frame starts on an 8-byte boundary: two samples per load
};

template <int E>
struct Layout {
  static constexpr int M = 16 * E;             // complex points
  static constexpr int kBins = M + 1;
  // floats of one frame's exchange buffer: rows of 16 with a pitch of 17, and the buffers of the two half-warps 16 banks apart
  static constexpr int kXch = E == 16 ? 272 : E == 32 ? 560 : 144;
  static constexpr int kPower = 0;             // float offsets
  static constexpr int kRows = kBins + 3;      // three rows of zeros: the mel sums read whole groups of four bins
  static constexpr int kWin = kRows * kPitch / 4 * 4 + 4;
  static constexpr int kTw = kWin + 2 * M;     // [E][16] complex: W_M^(l j) at [j][l]
  static constexpr int kPost = kTw + 2 * M;    // [M / 2] complex: W_2M^k
  static constexpr int kVar = kPost + M;       // weights [n_mel][len4], filter ranges, then exchange buffers / features [kTile][n_mel | 1]
};

template <int E>
__global__ void __launch_bounds__(kWarps * 32, E == 32 ? 1 : 3)
log_mel_fft_kernel(const Mel p) {
  using L = Layout<E>;
  constexpr int M = L::M;
  extern __shared__ __align__(16) float sm[];
  float* power = sm + L::kPower;
  C2* tw = reinterpret_cast<C2*>(sm + L::kTw);
  C2* post = reinterpret_cast<C2*>(sm + L::kPost);
  float2* win = reinterpret_cast<float2*>(sm + L::kWin);
  float* wsm = sm + L::kVar;
  int2* ranges = reinterpret_cast<int2*>(wsm + p.n_mel * p.len4);
  float* feat = reinterpret_cast<float*>(ranges + p.n_mel);  // the features of a tile stand where its exchange buffers were
  const int feat_pitch = p.n_mel | 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane & 15, hw = lane >> 4;
  float* xch = feat + (warp * 2 + hw) * L::kXch;

  for (int i = L::kBins * kPitch + tid; i < L::kRows * kPitch; i += kWarps * 32) power[i] = 0.f;
  for (int i = tid; i < 2 * M; i += kWarps * 32) sm[L::kWin + i] = i < p.window ? p.win[i] : 0.f;
  for (int i = tid; i < M; i += kWarps * 32) {
    float s, c;
    sincospif(2.f * (float)((i >> 4) * (i & 15)) / (float)M, &s, &c);
    tw[i] = {c, -s};
  }
  for (int i = tid; i < M / 2; i += kWarps * 32) {
    float s, c;
    sincospif((float)i / (float)M, &s, &c);
    post[i] = {c, -s};
  }
  for (int i = tid; i < p.n_mel * p.len4; i += kWarps * 32) {
    const int m = i / p.len4, k = i - m * p.len4;
    wsm[i] = k < p.max_len ? 0.25f * p.weights[(size_t)k * p.n_mel + m] : 0.f;  // the halves of the sums below, squared
  }
  for (int i = tid; i < p.n_mel; i += kWarps * 32) ranges[i] = make_int2(p.fb_start[i], p.fb_len[i]);
  __syncthreads();

  for (int tile = blockIdx.x; tile < p.rows * p.tiles; tile += gridDim.x) {
    const int row = tile / p.tiles, f0 = (tile - row * p.tiles) * kTile;
    const long long len = p.lens ? (long long)p.lens[row] : p.T;
    const int n_frames = min(len >= p.window ? (int)((len - p.window) / p.step + 1) : 0, p.n_frames_max);
#pragma unroll 1
    for (int pass = 0; pass < kTile / (2 * kWarps); ++pass) {
      // frames 16 apart in the two half-warps: their columns of the power array lie in different banks
      const int f = warp + pass * kWarps + 16 * hw;
      const bool on = f0 + f < n_frames;
      if (!__any_sync(0xffffffffu, on)) continue;
      const float* x = p.audio + (size_t)row * p.T + (size_t)(f0 + f) * p.step;
      C2 a[E];
      const int left = on ? p.window - 2 * l : 0;  // sample 32 i of this lane lies inside the window where 32 i < left
      if (p.pairs) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
          float2 t = make_float2(0.f, 0.f);
          if (32 * i < left) t = __ldg(reinterpret_cast<const float2*>(x + 2 * l) + 16 * i);
          a[i] = {t.x, t.y};
        }
      } else {
#pragma unroll
        for (int i = 0; i < E; ++i) {
          a[i] = {0.f, 0.f};
          if (32 * i < left) a[i].x = __ldg(x + 2 * l + 32 * i);
          if (32 * i + 1 < left) a[i].y = __ldg(x + 2 * l + 32 * i + 1);
        }
      }
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const float2 w = win[l + 16 * i];
        a[i].x *= w.x;
        a[i].y *= w.y;
      }
      fft<E>(a);
#pragma unroll
      for (int j = 1; j < E; ++j) a[j] = cmul(a[j], tw[j * 16 + l]);
      // through shared memory real and imaginary parts one after the other: half the buffer, and the two half-warps share each access
      constexpr int R = E < 16 ? 1 : E / 16;  // residues per lane; with E = 8 the lanes of the upper half of 16 have none
      C2 z[R][16];
#pragma unroll
      for (int j = 0; j < E; ++j) xch[j * 17 + l] = a[j].x;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 16; ++i) z[r][i].x = l + 16 * r < E ? xch[(l + 16 * r) * 17 + i] : 0.f;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < E; ++j) xch[j * 17 + l] = a[j].y;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 16; ++i) z[r][i].y = l + 16 * r < E ? xch[(l + 16 * r) * 17 + i] : 0.f;
#pragma unroll
      for (int r = 0; r < R; ++r) fft<16>(z[r]);
      float* pw = power + f;
      if constexpr (E == 16) {
        // z[q] = Z[l + 16 q]; Z[M - k] is z[15 - q] of lane 16 - l, for l = 0 the lane's own z[16 - q]
        const int src = (lane & 16) | ((16 - l) & 15);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const C2 give = l ? z[0][15 - q] : z[0][(16 - q) & 15];
          const C2 b = {__shfl_sync(0xffffffffu, give.x, src), __shfl_sync(0xffffffffu, give.y, src)};
          const int k = l + 16 * q;
          const C2 e = {z[0][q].x + b.x, z[0][q].y - b.y}, o = {z[0][q].y + b.y, b.x - z[0][q].x};
          const C2 r = cmul(o, post[k]);
          const C2 s = e + r, d = e - r;
          pw[k * kPitch] = s.x * s.x + s.y * s.y;
          pw[(M - k) * kPitch] = d.x * d.x + d.y * d.y;
        }
        if (l == 0) pw[(M / 2) * kPitch] = 4.f * (z[0][8].x * z[0][8].x + z[0][8].y * z[0][8].y);
      } else {
        C2 c[E / 2], b[E / 2], mid;
        auto through = [&](auto get, auto put) {
          __syncwarp();
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (l + 16 * r < E) {
#pragma unroll
              for (int q = 0; q < 16; ++q) xch[l + 16 * r + E * q] = get(z[r][q]);
            }
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < E / 2; ++i) {
            put(c[i]) = xch[l + 16 * i];
            put(b[i]) = xch[(M - l - 16 * i) & (M - 1)];
          }
          put(mid) = xch[M / 2];
        };
        through([](C2 v) { return v.x; }, [](C2& v) -> float& { return v.x; });
        through([](C2 v) { return v.y; }, [](C2& v) -> float& { return v.y; });
#pragma unroll
        for (int i = 0; i < E / 2; ++i) {
          const int k = l + 16 * i;
          const C2 e = {c[i].x + b[i].x, c[i].y - b[i].y}, o = {c[i].y + b[i].y, b[i].x - c[i].x};
          const C2 r = cmul(o, post[k]);
          const C2 s = e + r, d = e - r;
          pw[k * kPitch] = s.x * s.x + s.y * s.y;
          pw[(M - k) * kPitch] = d.x * d.x + d.y * d.y;
        }
        if (l == 0) pw[(M / 2) * kPitch] = 4.f * (mid.x * mid.x + mid.y * mid.y);
      }
      __syncwarp();  // the exchange buffer is free for the next pass
    }
    __syncthreads();
    const bool on = f0 + lane < n_frames;
    for (int m = warp; m < p.n_mel; m += kWarps) {
      const int2 range = ranges[m];
      const float* pk = power + range.x * kPitch + lane;
      const float4* wm = reinterpret_cast<const float4*>(wsm + m * p.len4);
      float acc = 0.f, acc2 = 0.f;
      for (int k = 0; k < range.y; k += 4, pk += 4 * kPitch) {  // past the filter's last bin the weights are 0
        const float4 w = wm[k >> 2];
        acc += pk[0] * w.x;
        acc2 += pk[kPitch] * w.y;
        acc += pk[2 * kPitch] * w.z;
        acc2 += pk[3 * kPitch] * w.w;
      }
      feat[lane * feat_pitch + m] = on ? log_floor(acc + acc2, p.eps) * p.log_scale : 0.f;
    }
    __syncthreads();  // the features are complete, and the power array is free for the next tile
    const int n_here = min(kTile, p.n_frames_max - f0) * p.n_mel;
    float* o = p.out + ((size_t)row * p.n_frames_max + f0) * p.n_mel;
    const int per = p.quads ? 4 : 1, wide = p.n_mel / per;
    int fr = tid / wide, m = tid - fr * wide;
    const int df = (kWarps * 32) / wide, dm = kWarps * 32 - df * wide;
    for (int i = tid; i < n_here / per; i += kWarps * 32) {
      const float* s = feat + fr * feat_pitch + m * per;
      if (p.quads) reinterpret_cast<float4*>(o)[i] = make_float4(s[0], s[1], s[2], s[3]);
      else o[i] = s[0];
      fr += df;
      m += dm;
      if (m >= wide) {
        m -= wide;
        ++fr;
      }
    }
    __syncthreads();  // the features have left: their place takes the next tile's exchange
  }
}

template <int E>
size_t smem_bytes(int max_len, int n_mel) {
  const size_t len4 = (size_t)(max_len + 3) / 4 * 4;
  return ((size_t)Layout<E>::kVar + n_mel * (len4 + 2) + std::max<size_t>(kTile * (size_t)(n_mel | 1), 2 * kWarps * Layout<E>::kXch)) * sizeof(float);
}
size_t smem_for(int n_fft, int max_len, int n_mel) {
  return n_fft == 256 ? smem_bytes<8>(max_len, n_mel) : n_fft == 512 ? smem_bytes<16>(max_len, n_mel) : smem_bytes<32>(max_len, n_mel);
}
constexpr size_t kSmemMax = 220 * 1024;

template <int E>
int launch(const Mel& p, size_t smem, cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(log_mel_fft_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e != cudaSuccess) {
    rb_set_error("log_mel_fft: %s", cudaGetErrorString(e));
    return RB_ERR_LAUNCH;
  }
  const long long per_sm = std::max<long long>(1, std::min<long long>(E == 32 ? 1 : 3, (long long)(227 * 1024 / (smem + 1024))));
  const int grid = (int)std::min<long long>((long long)p.rows * p.tiles, 148 * per_sm);
  log_mel_fft_kernel<E><<<grid, kWarps * 32, smem, stream>>>(p);
  return rb_check_launch("log_mel_fft");
}

}  // namespace

// whether log_mel_fft takes this transform length with filters of up to max_len bins
RB_EXPORT int rb200_log_mel_fft_supported(int n_fft, int max_len, int n_mel) {
  return (n_fft == 256 || n_fft == 512 || n_fft == 1024) && max_len > 0 && n_mel > 0 && smem_for(n_fft, max_len, n_mel) <= kSmemMax;
}

// audio [rows, T] fp32; lens [rows] (samples; null: all rows full); win [window], window <= n_fft; weights [max_len, n_mel] with the filters'
// ranges fb_start, fb_len [n_mel] of the n_fft / 2 + 1 bins; out [rows, n_frames_max, n_mel], frames past a row's length are written as 0.
RB_EXPORT int rb200_log_mel_fft(const float* audio, const int* lens, int rows, long long T, int n_frames_max, int window, int step, int n_fft,
                                const float* win, const float* weights, int max_len, const int* fb_start, const int* fb_len, int n_mel, float log_scale,
                                float eps, float* out, cudaStream_t stream) {
  if (rows <= 0 || n_frames_max <= 0) return RB_OK;
  if (!rb200_log_mel_fft_supported(n_fft, max_len, n_mel) || window < 1 || window > n_fft || step < 1) {
    rb_set_error("log_mel_fft: n_fft=%d must be 256, 512 or 1024 and >= window=%d (%d filters of up to %d bins)", n_fft, window, n_mel, max_len);
    return RB_ERR_UNSUPPORTED;
  }
  Mel p;
  p.audio = audio;
  p.lens = lens;
  p.T = T;
  p.rows = rows;
  p.n_frames_max = n_frames_max;
  p.window = window;
  p.step = step;
  p.tiles = (n_frames_max + kTile - 1) / kTile;
  p.win = win;
  p.weights = weights;
  p.fb_start = fb_start;
  p.fb_len = fb_len;
  p.max_len = max_len;
  p.len4 = (max_len + 3) / 4 * 4;
  p.n_mel = n_mel;
  p.log_scale = log_scale;
  p.eps = eps;
  p.out = out;
  p.quads = n_mel % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  p.pairs = window % 2 == 0 && step % 2 == 0 && T % 2 == 0 && (reinterpret_cast<uintptr_t>(audio) & 7) == 0;
  if ((long long)rows * p.tiles > 2147483647LL) {
    rb_set_error("log_mel_fft: %d rows of %d frames", rows, n_frames_max);
    return RB_ERR_UNSUPPORTED;
  }
  const size_t smem = smem_for(n_fft, max_len, n_mel);
  return n_fft == 256 ? launch<8>(p, smem, stream) : n_fft == 512 ? launch<16>(p, smem, stream) : launch<32>(p, smem, stream);
}

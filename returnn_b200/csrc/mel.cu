// Log-mel filterbank features from raw audio in one kernel: framing, Hann window, DFT (zero-padded to n_fft), power spectrum,
// mel filterbank, log. fp32 throughout (the reference upcasts bf16 audio to fp32 for the STFT, returnn/torch/frontend/_backend.py:2695-2711;
// math of returnn/frontend/audio/mel.py:163-208). One CTA computes kFrames consecutive frames of one recording: the windowed
// frames and a cos / sin table live in shared memory, every thread owns one frequency bin for all frames, then the mel
// projection runs from the power spectrum in shared memory.
#include <algorithm>
#include <cuda_fp16.h>
#include "common.cuh"

namespace {

constexpr int kFrames = 8;
constexpr int kMaxFft = 1024;
constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads)
log_mel_kernel(const float* __restrict__ audio, const int* __restrict__ lens, long long row_pitch, int n_frames_max, int window, int step, int n_fft,
               const float* __restrict__ win, const float* __restrict__ fbank, int n_mel, float log_scale, float eps, float* __restrict__ out) {
  extern __shared__ float sh[];
  float* sx = sh;                          // [kFrames][window]
  float* scos = sx + kFrames * window;     // [n_fft]
  float* ssin = scos + n_fft;              // [n_fft]
  float* spow = ssin + n_fft;              // [kFrames][n_bins]
  const int n_bins = n_fft / 2 + 1;
  const int row = blockIdx.y;
  const int f0 = blockIdx.x * kFrames;
  const int len = lens ? lens[row] : (int)row_pitch;
  const int n_frames = len >= window ? (len - window) / step + 1 : 0;
  if (f0 >= n_frames_max) return;
  const float* a = audio + (size_t)row * row_pitch;
  for (int i = threadIdx.x; i < kFrames * window; i += kThreads) {
    const int f = i / window, n = i - f * window;
    const int fr = f0 + f;
    sx[i] = fr < n_frames ? a[(size_t)fr * step + n] * win[n] : 0.f;
  }
  for (int i = threadIdx.x; i < n_fft; i += kThreads) {
    float s, c;
    sincospif(2.0f * (float)i / (float)n_fft, &s, &c);
    scos[i] = c;
    ssin[i] = s;
  }
  __syncthreads();
  const int mask = n_fft - 1;
  for (int k = threadIdx.x; k < n_bins; k += kThreads) {
    float re[kFrames], im[kFrames];
#pragma unroll
    for (int f = 0; f < kFrames; ++f) re[f] = im[f] = 0.f;
    int idx = 0;
    for (int n = 0; n < window; ++n) {
      const float c = scos[idx], s = ssin[idx];
#pragma unroll
      for (int f = 0; f < kFrames; ++f) {
        const float x = sx[f * window + n];
        re[f] += x * c;
        im[f] -= x * s;
      }
      idx = (idx + k) & mask;
    }
#pragma unroll
    for (int f = 0; f < kFrames; ++f) spow[f * n_bins + k] = re[f] * re[f] + im[f] * im[f];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kFrames * n_mel; i += kThreads) {
    const int f = i / n_mel, m = i - f * n_mel;
    const int fr = f0 + f;
    if (fr >= n_frames_max) continue;
    float acc = 0.f;
    const float* p = spow + f * n_bins;
    for (int k = 0; k < n_bins; ++k) acc += p[k] * fbank[(size_t)k * n_mel + m];
    const float v = fr < n_frames ? log_floor(acc, eps) * log_scale : 0.f;
    out[((size_t)row * n_frames_max + fr) * n_mel + m] = v;
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// The tensor-core form: the DFT of all frames is ONE matrix product, frames [rows * slots, window] x table [window, n_fft], on the
// tcgen05 GEMM. The frames are never materialised: the A operand is a strided view of the audio (row pitch = step samples, so
// consecutive rows overlap by window - step samples), which a TMA tensor map expresses directly. fp32 audio and table are split into
// fp16 high and low parts and three products (hi*lo + lo*hi + hi*hi) accumulate in fp32, which keeps 22 mantissa bits per factor
// (bf16 parts would keep 16: an error floor 96 dB under a frame's strongest component, audible in the weakest mel bands).
// Audio is expected within fp16's range (|x| < 65504; samples scaled to [-1, 1] or raw 16-bit PCM values both are).
// The two kernels here are the ends of that pipeline: the split of the audio, and power spectrum -> mel -> log.

// audio [rows, T] fp32 -> hi, lo [rows * Tp + tail] fp16 with audio[r][c] at r * Tp + c, zeros elsewhere (Tp = slots * step)
// Eight samples per thread: two 16-byte loads where the row's start allows them, two 16-byte stores (Tp is a multiple of 8, so a group
// lies in one row). Bound by memory, 8 bytes per sample.
__global__ void __launch_bounds__(256)
split_hi_lo_kernel(const float* __restrict__ audio, int rows, long long T, long long Tp, long long total, __half* __restrict__ hi,
                   __half* __restrict__ lo) {
  const long long groups = total / 8, per_row = Tp / 8;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += stride) {
    const long long r = i / per_row, c = (i - r * per_row) * 8;
    const float* src = audio + r * T + c;
    float x[8];
    if (r < rows && c + 8 <= T && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      const float4 u = reinterpret_cast<const float4*>(src)[0], v = reinterpret_cast<const float4*>(src)[1];
      x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w;
      x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = r < rows && c + e < T ? src[e] : 0.f;
    }
    __align__(16) __half h[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      h[e] = __float2half_rn(x[e]);
      l[e] = __float2half_rn(x[e] - __half2float(h[e]));
    }
    *reinterpret_cast<uint4*>(hi + 8 * i) = *reinterpret_cast<const uint4*>(h);
    *reinterpret_cast<uint4*>(lo + 8 * i) = *reinterpret_cast<const uint4*>(l);
  }
}

// spec [rows * slots, ld] fp32: column 2j = Re X_j, 2j + 1 = Im X_j for 0 < j < n_fft / 2; column 0 = X_0 and column 1 = X_{n_fft/2}
// (both real). One warp per frame: power spectrum into shared memory, then every lane sums the bins of its mel filters, which are
// contiguous ranges [fb_start[m], fb_start[m] + fb_len[m]). The filter weights come as a table [max_len, n_mel], entry i of filter m at
// [i][m], held in shared memory for the kMelFrames frames of every warp: read from the filterbank matrix, where the lanes' filters lie in
// different rows, each load took 32 cache accesses, which was the time of the kernel.
constexpr int kMelWarps = 8;
constexpr int kMelFrames = 4;

__global__ void __launch_bounds__(kMelWarps * 32)
mel_from_spectrum_kernel(const float* __restrict__ spec, int ld, int slots, int n_frames_max, const int* __restrict__ lens, long long T, int window,
                         int step, int n_fft, const float* __restrict__ weights, int max_len, const int* __restrict__ fb_start,
                         const int* __restrict__ fb_len, int n_mel, float log_scale, float eps, float* __restrict__ out) {
  extern __shared__ float shm[];  // [kMelWarps][n_bins], then [max_len][n_mel]
  const int n_bins = n_fft / 2 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ws = shm + kMelWarps * n_bins;
  for (int i = threadIdx.x; i < max_len * n_mel; i += kMelWarps * 32) ws[i] = weights[i];
  __syncthreads();
  const int row = blockIdx.y;
  const long long len = lens ? (long long)lens[row] : T;
  const int n_frames = len >= window ? (int)((len - window) / step + 1) : 0;
  float* pw = shm + warp * n_bins;
  for (int f = 0; f < kMelFrames; ++f) {
    const int fr = (blockIdx.x * kMelFrames + f) * kMelWarps + warp;
    if (fr >= n_frames_max) return;
    float* o = out + ((size_t)row * n_frames_max + fr) * n_mel;
    if (fr >= n_frames) {
      for (int m = lane; m < n_mel; m += 32) o[m] = 0.f;
      continue;
    }
    const float2* sp = reinterpret_cast<const float2*>(spec + ((size_t)row * slots + fr) * ld);
    __syncwarp();  // all lanes have read the previous frame's power
#pragma unroll 8
    for (int j = lane; j < n_fft / 2; j += 32) {
      const float2 v = sp[j];
      if (j == 0) {
        pw[0] = v.x * v.x;
        pw[n_fft / 2] = v.y * v.y;
      } else {
        pw[j] = v.x * v.x + v.y * v.y;
      }
    }
    __syncwarp();
    for (int m = lane; m < n_mel; m += 32) {
      const int k0 = fb_start[m], n = fb_len[m];
      float acc = 0.f;
      for (int k = 0; k < n; ++k) acc += pw[k0 + k] * ws[k * n_mel + m];
      o[m] = log_floor(acc, eps) * log_scale;
    }
  }
}

}  // namespace

RB_EXPORT int rb200_split_hi_lo_fp16(const float* audio, int rows, long long T, long long Tp, long long total, void* hi, void* lo, cudaStream_t stream) {
  if (total <= 0) return RB_OK;
  if (Tp % 8 || total % 8 || ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15)) {
    rb_set_error("split_hi_lo: Tp=%lld and total=%lld must be multiples of 8, the outputs 16-byte aligned", Tp, total);
    return RB_ERR_ARG;
  }
  const int blocks = (int)std::min<long long>((total / 8 + 255) / 256, 148LL * 8);
  split_hi_lo_kernel<<<blocks, 256, 0, stream>>>(audio, rows, T, Tp, total, reinterpret_cast<__half*>(hi), reinterpret_cast<__half*>(lo));
  return rb_check_launch("split_hi_lo");
}

RB_EXPORT int rb200_mel_from_spectrum(const float* spec, int ld, int rows, int slots, int n_frames_max, const int* lens, long long T, int window, int step,
                                      int n_fft, const float* weights, int max_len, const int* fb_start, const int* fb_len, int n_mel, float log_scale,
                                      float eps, float* out, cudaStream_t stream) {
  if (rows <= 0 || n_frames_max <= 0) return RB_OK;
  if ((ld % 2) || n_fft < 2 || (reinterpret_cast<uintptr_t>(spec) & 7)) {
    rb_set_error("mel_from_spectrum: ld=%d must be even and the spectrum 8-byte aligned", ld);
    return RB_ERR_ARG;
  }
  const size_t smem = ((size_t)kMelWarps * (n_fft / 2 + 1) + (size_t)max_len * n_mel) * sizeof(float);
  if ((size_t)kMelWarps * (n_fft / 2 + 1) * sizeof(float) > 48 * 1024 || smem > 220 * 1024) {
    rb_set_error("mel_from_spectrum: n_fft=%d or the longest filter (%d bins, %d filters) too large", n_fft, max_len, n_mel);
    return RB_ERR_UNSUPPORTED;
  }
  const cudaError_t e = cudaFuncSetAttribute(mel_from_spectrum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  if (e != cudaSuccess) {
    rb_set_error("mel_from_spectrum: %s", cudaGetErrorString(e));
    return RB_ERR_LAUNCH;
  }
  dim3 grid((n_frames_max + kMelWarps * kMelFrames - 1) / (kMelWarps * kMelFrames), rows);
  mel_from_spectrum_kernel<<<grid, kMelWarps * 32, smem, stream>>>(spec, ld, slots, n_frames_max, lens, T, window, step, n_fft, weights, max_len, fb_start,
                                                                 fb_len, n_mel, log_scale, eps, out);
  return rb_check_launch("mel_from_spectrum");
}

// audio [rows, row_pitch] fp32; lens [rows] (samples; null: all rows full); win [window] window function; fbank [n_fft/2+1, n_mel];
// out [rows, n_frames_max, n_mel] with n_frames_max = (row_pitch - window) / step + 1; frames past a row's length are written as 0.
// n_fft must be a power of two <= 1024.
RB_EXPORT int rb200_log_mel(const float* audio, const int* lens, int rows, long long row_pitch, int window, int step, int n_fft, const float* win,
                            const float* fbank, int n_mel, float log_scale, float eps, float* out, cudaStream_t stream) {
  if (rows <= 0 || row_pitch < window) return RB_OK;
  if (n_fft > kMaxFft || (n_fft & (n_fft - 1)) || window > n_fft || n_mel < 1) {
    rb_set_error("log_mel: n_fft=%d must be a power of two <= %d and >= window=%d", n_fft, kMaxFft, window);
    return RB_ERR_UNSUPPORTED;
  }
  const int n_frames_max = (int)((row_pitch - window) / step + 1);
  const size_t smem = ((size_t)kFrames * window + 2 * n_fft + (size_t)kFrames * (n_fft / 2 + 1)) * sizeof(float);
  static size_t attr = 0;
  if (smem > 48 * 1024 && smem > attr) {
    cudaFuncSetAttribute(log_mel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = smem;
  }
  dim3 grid((n_frames_max + kFrames - 1) / kFrames, rows);
  log_mel_kernel<<<grid, kThreads, smem, stream>>>(audio, lens, row_pitch, n_frames_max, window, step, n_fft, win, fbank, n_mel, log_scale, eps, out);
  return rb_check_launch("log_mel");
}

// Element-wise kernels on bf16: dropout with a counter-based RNG whose seed and offset live in device memory
// (a CUDA-graph replay reads the current values, so every replay draws a fresh mask and backward re-creates the mask
// of its forward from the saved offset).
#include "common.cuh"

namespace {

__global__ void __launch_bounds__(256)
dropout_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int64_t n, float p,
               const int64_t* __restrict__ seed, const int64_t* __restrict__ offset) {
  const uint64_t sd = (uint64_t)seed[0];
  const uint64_t off = (uint64_t)offset[0];
  const float scale = 1.f / (1.f - p);
  const uint32_t thresh = rb_dropout_thresh16(p);
  const uint2 key = make_uint2((uint32_t)sd, (uint32_t)(sd >> 32));
  const int64_t n8 = n & ~(int64_t)7;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n8; i += (int64_t)gridDim.x * blockDim.x * 8) {
    F8 a = load8(x, i, 1);
    rb_dropout_apply8(key, off + (uint64_t)i, thresh, scale, a.v);
    store8(y, i, a, 1);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n - n8)) {
    // the last, incomplete group: the same 16-bit values as a complete group starting at n8 would use
    int64_t i = n8 + threadIdx.x;
    const uint4 r = rb_dropout_bits8(key, off + (uint64_t)n8);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    const uint32_t bits = (threadIdx.x & 1) ? (w[threadIdx.x >> 1] >> 16) : (w[threadIdx.x >> 1] & 0xFFFFu);
    float v = __bfloat162float(x[i]);
    y[i] = __float2bfloat16(bits >= thresh ? v * scale : 0.f);
  }
}

// The part of a linear layer's backward pass before its two products, in one pass over the rows: dz = dy * act'(z) (bf16; act 0: dz is
// dy and is not written) and the bias gradient db[c] += sum_r dz[r][c] of the rounded values. A CTA owns 64 columns (8 threads x 16
// bytes: whole 128-byte lines) and a slice of the rows; its 32 row lanes keep four loads in flight each. One fp32 atomic per column and CTA.
// Bound by memory: 6656 x 2048, silu: 82 MB.
template <int ACT>
__global__ void __launch_bounds__(256, 4)
act_grad_colsum_kernel(const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dz,
                       float* __restrict__ db, int rows, int cols, int rows_per_cta) {
  rb_pdl_wait();
  rb_pdl_launch();
  __shared__ float red[32][65];
  const int cg = threadIdx.x & 7, rl = threadIdx.x >> 3;
  const int col = blockIdx.y * 64 + cg * 8;
  const int r_begin = blockIdx.x * rows_per_cta;
  const int r_end = min(rows, r_begin + rows_per_cta);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < cols) {
    for (int r0 = r_begin + rl; r0 < r_end; r0 += 64) {
      F8 d[2], v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = r0 + u * 32;
        if (r < r_end) {
          d[u] = load8(dy, (int64_t)r * cols + col, 1);
          if (ACT) v[u] = load8(z, (int64_t)r * cols + col, 1);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = r0 + u * 32;
        if (r >= r_end) break;
        if (ACT) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float x = v[u].v[i];
            float g;
            if (ACT == 1) {
              g = x > 0.f ? 1.f : 0.f;
            } else if (ACT == 2) {
              const float s = 1.f / (1.f + __expf(-x));
              g = s * (1.f + x * (1.f - s));
            } else {
              g = 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * __expf(-0.5f * x * x) * 0.39894228040143268f;
            }
            d[u].v[i] = __bfloat162float(__float2bfloat16(d[u].v[i] * g));
          }
          store8(dz, (int64_t)r * cols + col, d[u], 1);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += d[u].v[i];
      }
    }
  }
  if (!db) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) red[rl][cg * 8 + i] = acc[i];
  __syncthreads();
  if (threadIdx.x < 64 && blockIdx.y * 64 + threadIdx.x < cols) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) sum += red[k][threadIdx.x];
    atomicAdd(db + blockIdx.y * 64 + threadIdx.x, sum);
  }
}

}  // namespace

// act: 0 none (dz unused), 1 relu, 2 silu, 3 gelu; db (may be null) is added to; cols a multiple of 8, 16-byte aligned rows
RB_EXPORT int rb200_act_grad_colsum(const void* z, const void* dy, void* dz, float* db, int rows, int cols, int act, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0 || (!db && act == 0)) return RB_OK;
  if (cols % 8 || act < 0 || act > 3) {
    rb_set_error("act_grad_colsum: cols=%d act=%d", cols, act);
    return RB_ERR_ARG;
  }
  const int chunks = (cols + 63) / 64;
  // four CTAs per SM; at least one row per row lane
  int splits = (4 * 148 + chunks - 1) / chunks;
  splits = min(splits, (rows + 31) / 32);
  const int per = (rows + splits - 1) / splits;
  splits = (rows + per - 1) / per;
  auto kernel = act == 0 ? act_grad_colsum_kernel<0> : act == 1 ? act_grad_colsum_kernel<1> : act == 2 ? act_grad_colsum_kernel<2> : act_grad_colsum_kernel<3>;
  rb_launch_pdl(kernel, dim3(splits, chunks), dim3(256), 0, stream, (const __nv_bfloat16*)z, (const __nv_bfloat16*)dy, (__nv_bfloat16*)dz, db, rows, cols, per);
  return rb_check_launch("act_grad_colsum");
}

RB_EXPORT int rb200_dropout_bf16(const __nv_bfloat16* x, __nv_bfloat16* y, long long n, float p, const long long* seed,
                                 const long long* offset, cudaStream_t stream) {
  if (n <= 0) return RB_OK;
  if (!(p >= 0.f && p < 1.f)) {
    rb_set_error("dropout: p=%f out of [0,1)", p);
    return RB_ERR_ARG;
  }
  int grid = (int)((n / 8 + 255) / 256);
  if (grid < 1) grid = 1;
  if (grid > 148 * 8) grid = 148 * 8;
  dropout_kernel<<<grid, 256, 0, stream>>>(x, y, n, p, (const int64_t*)seed, (const int64_t*)offset);
  return rb_check_launch("dropout");
}

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
// dy and is not written) and the bias gradient db[c] += sum_r dz[r][c] of the rounded values. A CTA owns 8 CG columns (CG threads x 16
// bytes: lines of 128 or pieces of 512 bytes) and a slice of the rows; its 32 row lanes take U rows at a time (2 U loads in flight, U without an
// activation). Column sums: with `part` every slice leaves its own there, and colsum_slices_kernel adds them up in the order of the slices, so
// that the gradient of the same inputs is the same in every run; without, one atomic per column and CTA adds them to what is in db (6656 x 2048,
// silu: 19.3 us ordered, 18.2 by atomics; 6656 x 512, no activation: 5.1 and 2.6).
// Bound by memory: 6656 x 2048, silu: 82 MB.
template <int ACT, int CG, int U>
__global__ void __launch_bounds__(32 * CG, CG == 8 ? 4 : 1)
act_grad_colsum_kernel(const __nv_bfloat16* __restrict__ z, const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dz,
                       float* __restrict__ db, float* __restrict__ part, int rows, int cols, int rows_per_cta) {
  rb_pdl_wait();
  rb_pdl_launch();
  __shared__ float red[32][8 * CG + 1];
  const int cg = threadIdx.x % CG, rl = threadIdx.x / CG;
  const int col = (blockIdx.y * CG + cg) * 8;
  const int r_begin = blockIdx.x * rows_per_cta;
  const int r_end = min(rows, r_begin + rows_per_cta);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < cols) {
    for (int r0 = r_begin + rl; r0 < r_end; r0 += 32 * U) {
      uint4 dr[U], vr[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = r0 + u * 32;
        if (r < r_end) {
          dr[u] = *reinterpret_cast<const uint4*>(dy + (int64_t)r * cols + col);
          if (ACT) vr[u] = *reinterpret_cast<const uint4*>(z + (int64_t)r * cols + col);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = r0 + u * 32;
        if (r >= r_end) break;
        F8 d[1], v[1];
        d[0] = load8(&dr[u], 0, 1);
        if (ACT) v[0] = load8(&vr[u], 0, 1);
        if (ACT) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float x = v[0].v[i];
            float g;
            if (ACT == 1) {
              if (!(x > 0.f)) d[0].v[i] = 0.f;  // (also where the gradient is not finite)
              continue;
            } else if (ACT == 2) {
              const float s = 1.f / (1.f + __expf(-x));
              g = s * (1.f + x * (1.f - s));
            } else {
              g = 0.5f * (1.f + erff(x * 0.70710678118654752f)) + x * __expf(-0.5f * x * x) * 0.39894228040143268f;
            }
            d[0].v[i] = __bfloat162float(__float2bfloat16(d[0].v[i] * g));
          }
          store8(dz, (int64_t)r * cols + col, d[0], 1);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += d[0].v[i];
      }
    }
  }
  if (!db) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) red[rl][cg * 8 + i] = acc[i];
  __syncthreads();
  const int c = blockIdx.y * 8 * CG + threadIdx.x;
  if (threadIdx.x < 8 * CG && c < cols) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) sum += red[k][threadIdx.x];
    if (part) part[(int64_t)blockIdx.x * cols + c] = sum;
    else atomicAdd(db + c, sum);
  }
}

__global__ void __launch_bounds__(256)
colsum_slices_kernel(const float* __restrict__ part, float* __restrict__ db, int splits, int cols) {
  rb_pdl_wait();
  rb_pdl_launch();
  __shared__ float red[4][64];
  const int c = threadIdx.x & 63, lane = threadIdx.x >> 6, col = blockIdx.x * 64 + c;
  float sum = 0.f;
  if (col < cols)
    for (int i = lane; i < splits; i += 4) sum += part[(int64_t)i * cols + col];
  red[lane][c] = sum;
  __syncthreads();
  if (lane == 0 && col < cols) db[col] = (red[0][c] + red[1][c]) + (red[2][c] + red[3][c]);
}

// slices of the rows: four CTAs per SM, at least one row per row lane
int colsum_splits(int rows, int cols) {
  const int chunks = (cols + 63) / 64;
  return max(1, min((4 * 148 + chunks - 1) / chunks, (rows + 31) / 32));
}

}  // namespace

// act: 0 none (dz unused), 1 relu, 2 silu, 3 gelu; cols a multiple of 8, 16-byte aligned rows. db (may be null): with work
// (4 * 148 * 64 + cols words, the most that colsum_splits * cols comes to) written, the sums in order; without added to, by atomics
RB_EXPORT int rb200_act_grad_colsum(const void* z, const void* dy, void* dz, float* db, float* work, int rows, int cols, int act, cudaStream_t stream) {
  if (cols <= 0 || (!db && act == 0) || (rows <= 0 && !(db && work))) return RB_OK;
  if (cols % 8 || act < 0 || act > 3) {
    rb_set_error("act_grad_colsum: cols=%d act=%d", cols, act);
    return RB_ERR_ARG;
  }
  if (!db) work = nullptr;
  const int chunks = (cols + 63) / 64;
  if (rows <= 0) {
    rb_launch_pdl(colsum_slices_kernel, dim3(chunks), dim3(256), 0, stream, (const float*)work, db, 0, cols);
    return rb_check_launch("colsum_slices");
  }
  // Wide where the matrices do not stay in the L2 (dz, z and dy of 12 M elements: 72 MB). us out of memory, narrow / wide, silu: 6656 x 2048 28.4 / 20.9,
  // 25000 x 1024 36.6 / 31.9, 25000 x 512 21.5 / 21.1, 50000 x 256 21.4 / 21.5, 1000 x 36000 50.1 / 40.6, 400 x 60000 37.2 / 36.3; below the launch and the start of
  // a CTA of 1024 threads cost more: 2000 x 4096 11.5 / 12.0, 6656 x 512 7.5 / 8.7, 50 x 512 3.1 / 4.6. Without an activation one matrix is read, and the wide
  // form needs rows of several CTAs, all of them resident at once: 6656 x 2048 10.7 / 8.8, 8000 x 1536 9.9 / 9.0, 1000 x 16000 11.1 / 9.5, 700 x 22000 10.9 / 10.6,
  // 350 x 36000 8.8 / 8.1, but 50000 x 512 13.0 / 13.2, 100000 x 256 13.3 / 13.7, 400 x 40000 9.6 / 13.1
  const bool wide = (long long)rows * cols >= 12000000 && (act ? cols >= 256 : cols >= 1536 && cols <= 148 * 256);
  const int cta_chunks = wide ? (cols + 255) / 256 : chunks;
  int splits = wide ? max(1, min(148 / cta_chunks, (rows + 31) / 32)) : colsum_splits(rows, cols);
  const int per = (rows + splits - 1) / splits;
  splits = (rows + per - 1) / per;
  using Kernel = void (*)(const __nv_bfloat16*, const __nv_bfloat16*, __nv_bfloat16*, float*, float*, int, int, int);
  // Without an activation the narrow form has four rows of a thread in flight where columns are few and each CTA has many rows, or where the CTAs are
  // more than fit at once anyway; else two, with which five CTAs fit an SM: 6656 x 512 6.4 us with two, 5.7 with four; 20000 x 512 8.8 / 8.3, 25000 x 1024 13.7 / 12.4,
  // 400 x 60000 14.9 / 12.7; 600 x 2048 4.0 / 4.8, 800 x 8000 6.3 / 7.3, 400 x 40000 9.6 / 11.4
  const bool ahead = act == 0 && (cols <= 1024 || chunks > 5 * 148);
  static const Kernel narrow[] = {act_grad_colsum_kernel<0, 8, 2>, act_grad_colsum_kernel<1, 8, 2>, act_grad_colsum_kernel<2, 8, 2>, act_grad_colsum_kernel<3, 8, 2>};
  static const Kernel wides[] = {act_grad_colsum_kernel<0, 32, 4>, act_grad_colsum_kernel<1, 32, 4>, act_grad_colsum_kernel<2, 32, 4>, act_grad_colsum_kernel<3, 32, 2>};
  const Kernel kernel = wide ? wides[act] : ahead ? act_grad_colsum_kernel<0, 8, 4> : narrow[act];
  const dim3 grid(splits, cta_chunks), block(wide ? 1024 : 256);
  const __nv_bfloat16 *zp = (const __nv_bfloat16*)z, *dyp = (const __nv_bfloat16*)dy;
  if (!work) {
    rb_launch_pdl(kernel, grid, block, 0, stream, zp, dyp, (__nv_bfloat16*)dz, db, work, rows, cols, per);
    return rb_check_launch("act_grad_colsum");
  }
  // Not launched early: CTAs that come onto the SMs one by one while a product ends do not walk through the rows side by side, and the 64-column
  // pieces of a row are then read far apart in time (6656 x 10000 after a product: 61 us, launched in order 37)
  kernel<<<grid, block, 0, stream>>>(zp, dyp, (__nv_bfloat16*)dz, db, work, rows, cols, per);
  const int st = rb_check_launch("act_grad_colsum");
  if (st) return st;
  rb_launch_pdl(colsum_slices_kernel, dim3(chunks), dim3(256), 0, stream, (const float*)work, db, splits, cols);
  return rb_check_launch("colsum_slices");
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

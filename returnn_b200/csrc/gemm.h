// Internal C++ interface of the persistent tcgen05 GEMM (gemm_persist.cu), used by the C entry points and by the native
// encoder executor. D[m,n] = epilogue(alpha * op(A)·op(B)).
#pragma once
#include <cuda_runtime.h>

struct RbGemm {
  const void* a = nullptr;   // bf16; stored [m][k] (a_mn_major = 0) or [k][m] (1), row pitch lda elements
  const void* b = nullptr;   // bf16; stored [n][k] (b_mn_major = 0) or [k][n] (1), row pitch ldb elements
  void* c = nullptr;         // bf16 or fp32 [m][ldc]
  void* c2 = nullptr;        // optional bf16 [m][ldc]: receives the final value while c receives the pre-activation
  const void* bias = nullptr;
  int bias_bf16 = 0;
  int m = 0, n = 0, k = 0, lda = 0, ldb = 0, ldc = 0;
  int a_mn_major = 0, b_mn_major = 0;
  int ab_fp16 = 0;           // A and B hold IEEE fp16 instead of bf16 (same size, so the copies and layouts are the same; only the MMA reads them differently)
  int act = 0;               // 0 none, 1 relu, 2 silu, 3 gelu(erf)
  int out_fp32 = 0;
  int accumulate = 0;        // fp32 output only: 0 store, 1 c += value, 2 atomic c += value (needed with split_k > 1)
  float alpha = 1.f;
  // epilogue, applied in this order to v = alpha * acc + bias:
  const void* dact_z = nullptr;  // bf16 [m][ldc]: v *= act'(z)  (act names the function; the value itself is not activated then)
  float drop_p = 0.f;            // dropout on the (activated) value; mask of element (r, c) = philox(seed, offset + drop_site + r*ldc + c)
  const long long* seed = nullptr;
  const long long* offset = nullptr;
  unsigned long long drop_site = 0;
  const void* resid = nullptr;   // bf16 [m][ldc]: final = resid + res_scale * v
  float res_scale = 1.f;
  float* colsum = nullptr;       // [n] += the column sums of the stored bf16 values; only where rb_gemm_column_sums says so
  int split_k = 0;               // 0: chosen by the launcher (> 1 only with accumulate == 2)
  int slice_k = 0;               // CTA-pair kernel, fp32 output without the rest of the epilogue, m a multiple of 32: the contraction is cut into slices
                                 // of this many (a multiple of 64), whose products lie one behind the other in c, [ceil(k / slice_k)][m][ldc]
  // batched form (batch > 0): problem z = b * heads + h reads A from the stored origin (b*a_rb + h*a_rh, b*a_cb + h*a_ch),
  // B likewise, and writes at element offset b*c_sb + h*c_sh. m / n / k are fixed or lens[b] where the *_from_lens flag is set;
  // a problem with an empty extent is skipped. a_rows .. b_cols are the extents of the stored matrices.
  int batch = 0, heads = 1;
  long long a_rb = 0, a_rh = 0, a_cb = 0, a_ch = 0, b_rb = 0, b_rh = 0, b_cb = 0, b_ch = 0, c_sb = 0, c_sh = 0;
  long long a_rows = 0, a_cols = 0, b_rows = 0, b_cols = 0;
  const int* lens = nullptr;
  int m_from_lens = 0, n_from_lens = 0, k_from_lens = 0;
  // batched form, bf16 output without bias or activation: each problem owns whole rows of c, of ldc columns, and its rows up to the next multiple of 32.
  // c_rows > 0 (rows of the matrix that holds all problems' outputs): the output leaves in boxes of 32 x 64, what lies in them past m and n is unspecified
  long long c_rows = 0;
  // batched form, at most 64 columns, no more of the epilogue than alpha: as many problems again, of the same shape and origins, with other operands, another
  // output and another alpha (one launch, and the units of both share the SMs)
  const void *a_next = nullptr, *b_next = nullptr;
  void* c_next = nullptr;
  float alpha_next = 1.f;
  // windows of a relative-position band (batched form): row i of a sequence of length len concerns the columns [win_center - i, win_center - i + len).
  // win = 1: the output is the band, m_from_lens; tiles of it without such a column are not computed (and not written).
  // win = 2: A, stored [k][m], is the band of sequences of win_lp rows each (a multiple of 64) with lengths win_lens, zero outside the windows;
  // the contraction leaves out blocks of 64 rows that have no such column among those of the tile, and does not read them. k a multiple of 64.
  int win = 0, win_center = 0, win_lp = 0;
  const int* win_lens = nullptr;
  // split operands (CTA-pair kernel only): A and B are sums hi + lo whose parts lie in ONE stored matrix each, the rows of lo seg_a / seg_b
  // rows after those of hi (seg_a > 0). The contraction runs over hi*lo, lo*hi and hi*hi into one accumulator. B is stored [k][n].
  int seg_a = 0, seg_b = 0;
  int* status = nullptr;         // device word: 0 fine, else (role << 24 | detail) of the wait that gave up
};

// returns an RB_* status code; the launch is asynchronous on `stream`
int rb_gemm(const RbGemm& g, cudaStream_t stream);

// whether the epilogue of this problem's kernel can leave column sums (`colsum`): the full epilogue of the CTA-pair kernel with one bf16 output
// that leaves through bulk stores
bool rb_gemm_column_sums(const RbGemm& g);

// whether the CTA-pair kernel takes this problem with slice_k
bool rb_gemm_slices(const RbGemm& g);

// CTA-pair kernel (gemm_2cta.cu): rb_gemm routes to it when rb_gemm_pair_wanted says so
bool rb_gemm_pair_wanted(const RbGemm& g);
int rb_gemm_pair(const RbGemm& g, cudaStream_t stream);

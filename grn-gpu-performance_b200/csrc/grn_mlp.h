// grn_mlp.h -- launch interface of the surrogate MLP kernels (grn_mlp.cu,
// grn_umma.cu).
#ifndef GRN_MLP_H_
#define GRN_MLP_H_

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace grn {

// Programmatic dependent launch: a chain's kernel is launched while the one
// before it still runs, sets itself up, and waits (pdl_wait) before it
// touches anything an earlier kernel of the chain writes or reads; the weights
// are older than the chain.  pdl_trigger lets the next kernel start doing so.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#endif

enum MlpEpilogue {
  kEpiF32 = 0,       // C = acc (FP32)
  kEpiBiasRelu = 1,  // C = relu(acc + bias[n]) (BF16)
  kEpiMask = 2       // C = mask > 0 ? acc : 0 (BF16; ReLU backward)
};

// C[m][n] = sum_k A[m][k] B[n][k], both operands K-major (row m of A at
// A + m*lda, row n of B at B + n*ldb); BF16 operands, FP32 accumulation.
// The BF16 epilogues can also store the transposed result,
// Ct[n*ldt + m] = C[m][n].
struct MlpGemm {
  int M, N, K;
  const __nv_bfloat16 *A;
  int64_t lda;
  const __nv_bfloat16 *B;
  int64_t ldb;
  int epi;
  float *Cf;                  // FP32 output (kEpiF32)
  __nv_bfloat16 *Cb;          // BF16 output (kEpiBiasRelu, kEpiMask)
  int64_t ldc;
  __nv_bfloat16 *Ct;          // optional transposed BF16 output
  int64_t ldt;
  const float *bias;          // [N] (kEpiBiasRelu)
  const __nv_bfloat16 *mask;  // [M][ldc] (kEpiMask): keep where mask > 0
};

// The GEMM on warp-level mma.sync (the legacy tensor-core path).
cudaError_t mlp_gemm(const MlpGemm &p, cudaStream_t st);
// The GEMM on the tcgen05 tensor cores with TMA loads (grn_umma.cu).  An
// FP32 GEMM with few output tiles and a long K is split over K into ranges
// whose partial tiles go to `work` (up to work_elems floats) and are then
// added in range order.  Sets *error_flag (device) to 1 if a wait for the
// tensor core or a load timed out.  Operand rows must start on 16 bytes
// (lda, ldb multiples of 8, 16-byte aligned bases): cudaErrorInvalidValue
// otherwise.
cudaError_t mlp_gemm_tc(const MlpGemm &p, float *work, size_t work_elems, int *error_flag,
                        cudaStream_t st);

// K ranges that mlp_gemm_tc splits a kEpiF32 GEMM into, given a workspace of
// work_elems floats (1: no split).
int mlp_split_k(int M, int N, int K, size_t work_elems);
// The GEMM without the final addition: with more than one range, range z's
// tile is left at work + z*M*N (row-major M x N) and C is not written.
cudaError_t mlp_gemm_tc_partial(const MlpGemm &p, float *work, size_t work_elems, int *error_flag,
                                cudaStream_t st);

// The output layer of a training step and its gradient, one pass over h:
// y[b] = h[b] . w + b0, dy[b] = 2 (y[b] - t[b]) / B, dz[b][k] = h[b][k] > 0 ?
// dy[b] w[k] : 0 (BF16) and its transpose dzT[k][b].  K a multiple of 32.
cudaError_t mlp_output_step(int B, int K, const __nv_bfloat16 *h, const float *w, const float *b0,
                            const float *t, float *y, float *dy, __nv_bfloat16 *dz,
                            __nv_bfloat16 *dzT, int64_t ldt, cudaStream_t st);
// y[b] = h[b] . w + b0 (the output layer).
cudaError_t mlp_output_forward(int B, int K, const __nv_bfloat16 *h, const float *w,
                               const float *b0, float *y, cudaStream_t st);
// loss[0] = mean (y - t)^2, loss[1] += loss[0]; db[0] = sum of dy (2 (y - t)
// / B; the output bias gradient); *adam_step += 1 and *row += B unless null (a
// training step's count of Adam steps, read by mlp_adam, and the first row of
// the next minibatch's indices, read by mlp_gather_rows).
cudaError_t mlp_loss(int B, const float *y, const float *t, double *loss, float *db,
                     int *adam_step, int *row, cudaStream_t st);
// Up to four row reductions in one launch: out_j[r] = sum_c X_j[r][c] (x w[c]
// when w_j is set) for r < rows, c < cols; a fixed summation order.
struct MlpRowSum {
  const __nv_bfloat16 *X;
  const float *w;
  float *out;
};
cudaError_t mlp_row_sums(int n_jobs, const MlpRowSum *jobs, int rows, int cols, int64_t ldx,
                         cudaStream_t st);
// Square n x n blocks of the parameter vector, starting at offset[j], whose
// BF16 transpose Adam also writes to dst[j] (skipped where dst[j] is null).
struct MlpTransposed {
  int64_t offset[2];
  __nv_bfloat16 *dst[2];
  int n;
};
// Gradients left as split-K partial tiles (mlp_gemm_tc_partial): parameters
// offset .. offset + n - 1 have the gradient sum over z < split of
// work[z*n + i], added in order; split 1: the gradient array's own value.
struct MlpPartials {
  int64_t offset[3];
  int n[3];
  int split[3];
  const float *work[3];
};
// One Adam step on the FP32 parameters w (moments m, v; step number
// *adam_step, in device memory; gradients g or, where split, the partial
// sums), refreshing their BF16 copy wb and the transposed copies of tr.
cudaError_t mlp_adam(int n, float *w, const float *g, const MlpPartials &part, float *m, float *v,
                     float lr, float b1, float b2, float eps, const int *adam_step,
                     __nv_bfloat16 *wb, const MlpTransposed &tr, cudaStream_t st);
cudaError_t mlp_to_bf16(int n, const float *x, __nv_bfloat16 *y, cudaStream_t st);
// dst[c][r] = src[r][c] for a rows x cols BF16 matrix.
cudaError_t mlp_transpose(int rows, int cols, const __nv_bfloat16 *src, int64_t lds,
                          __nv_bfloat16 *dst, int64_t ldd, cudaStream_t st);
// Row r of dst (width columns) = row idx[*first + r] of src, tdst[r] =
// tsrc[idx[*first + r]] (*first in device memory, so that a captured
// training step gathers the next minibatch each time); dstT (optional)
// receives the transpose, dstT[c*ldt + r].
cudaError_t mlp_gather_rows(int rows, int width, const int32_t *idx, const int *first,
                            const __nv_bfloat16 *src,
                            const float *tsrc, __nv_bfloat16 *dst, float *tdst,
                            __nv_bfloat16 *dstT, int64_t ldt, cudaStream_t st);
// FP32 rows to BF16 (dst) and optionally their transpose (dstT).
cudaError_t mlp_convert_rows(int rows, int width, const float *src, __nv_bfloat16 *dst,
                             __nv_bfloat16 *dstT, int64_t ldt, cudaStream_t st);

}  // namespace grn

#endif  // GRN_MLP_H_

// zbuild.cuh — host entry points of the Z-build and genotype kernels (zbuild.cu).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace soda {

cudaError_t zb_decode_bed(const uint8_t *bed, int n, int p, int8_t *G, int ldx, cudaStream_t st);
cudaError_t zb_freq(int8_t *G, int n, int p, int ldx, double *freq, int *bad, cudaStream_t st);
cudaError_t zb_gather(const int8_t *Gsnp, int8_t *Gpos, const int32_t *perm, int p, int ldx, cudaStream_t st);
cudaError_t zb_xv(const double *freq, const int32_t *perm, int p, double *xv, cudaStream_t st);
cudaError_t zb_xv32(const double *xv, int p, float *xv32, cudaStream_t st);
// tm_g: the codes G as [p][ldx] bytes in 128 x 128 boxes, 128-byte swizzle.  W32 (or nullptr): an FP32 copy of each
// subset of the batch, columns ld32 apart, subsets ld32 * maxN.  *err is set when a device wait gave up.
cudaError_t zb_gram(const CUtensorMap *tm_g, const int8_t *G, int ldx, const int32_t *blk_ls,
                    const int32_t *batch_blocks, int nbatch, int maxN, const int64_t *wofs, const double *freq,
                    const int32_t *perm, int n, double *W, float *W32, int ld32, int *err, cudaStream_t st);
// Lanczos runs of a batch of subsets (lanczos.cuh).  V: [batch][mmax][N], subsets vstride apart; wpart:
// zb_lz_wpart() elements.  zb_lz_start fills v_0 from an FP32 run on W32 (V32: batch * zb_lz_pre() * maxN, ab32:
// 2 * batch * zb_lz_pre()); zb_lz_step is step j of the FP64 run.
int zb_lz_pre();
size_t zb_lz_wpart(int maxN, int nbatch);
cudaError_t zb_lz_prepare(int maxN, int mmax);
cudaError_t zb_lz_start(const float *W32, int ld32, const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch,
                        int maxN, size_t vstride, double *V, float *V32, float *wpart32, float *ab32, uint64_t seed,
                        cudaStream_t st);
cudaError_t zb_lz_step(const double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks,
                       int nbatch, int maxN, size_t vstride, double *V, double *wpart, double *alpha, double *beta,
                       int mmax, int j, const uint8_t *done, cudaStream_t st);
cudaError_t zb_form_m(double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch,
                      const double *xxd, cudaStream_t st);
// Cholesky of d I - A of a batch of subsets (chol_tc.cuh), A in W on entry, U's upper triangle there on return.
// dig: nbatch * zb_chol_digits() digits, seen by tm_a and tm_b as rows of zb_chol_ldt() bf16 in boxes of 32 x 128 and
// 32 x 64, 64-byte swizzle; work: zb_chol_work() doubles.
int zb_chol_np(int maxN);
int zb_chol_ldt(int maxN);
size_t zb_chol_digits(int maxN);
size_t zb_chol_work(int maxN, int nbatch);
cudaError_t zb_cholesky(const CUtensorMap *tm_a, const CUtensorMap *tm_b, double *W, const int64_t *wofs,
                        const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch, int maxN, const double *xxd,
                        int32_t *status, uint16_t *dig, double *work, int *err, cudaStream_t st);
cudaError_t zb_pd_lengths(const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch, const int32_t *status,
                          int32_t *ulen, uint8_t *skip, cudaStream_t st);
cudaError_t zb_psd_block(double *Wb, double *M, int N, int ls, int32_t *ulen, uint8_t *skip, int32_t *piv,
                         int32_t *rank, int32_t *status, double *work, cudaStream_t st);
cudaError_t zb_pack(const double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks,
                    int nbatch, const int64_t *uoff, const int32_t *ulen, double *U64, float *U32,
                    __nv_bfloat16 *Uhi, __nv_bfloat16 *Ulo, cudaStream_t st);
cudaError_t zb_unpack_dense(const double *U64, const int64_t *uoff, const int32_t *ulen, int p, int bs, double *xa,
                            cudaStream_t st);
// Genomic values (dgv.cuh): part holds zb_dgv_splits(n, p) * n doubles.  The codes of a context are centred by
// xv (nullptr: by freq), a .bed payload by freq.
int zb_dgv_splits(int n, int p);
cudaError_t zb_dgv(const int8_t *G, int ldx, const double *xv, const double *freq, const int32_t *perm,
                   const double *eff, int n, int p, double mu, double *part, double *pred, cudaStream_t st);
// The splits' sums of p SNPs of a .bed payload (their records, frequencies and effects): returns how many were
// written, at most nsplit, or -1; then mu + the sum of all of them.
int zb_dgv_bed(const uint8_t *bed, const double *freq, const double *eff, int n, int p, double *part, int nsplit,
               cudaStream_t st);
cudaError_t zb_dgv_sum(const double *part, int n, int nsplit, double mu, double *pred, cudaStream_t st);

}  // namespace soda

// The C ABI with two device calls of the Z build replaced, for tests of what follows their failure: the Gram of a single
// subset (the pivoted fallback's) can report that a wait gave up, and one subset's d can be lowered before the
// factorisation, which makes that subset alone indefinite; the free device memory is noted where the factors are packed.
// Linked with the library's other objects.
#include "../sodabayes_gb300/csrc/zbuild.cuh"

namespace {

int g_fallback_err = 0, g_subset = -1;
double g_shift = 0.0;
size_t g_free = 0;

__global__ void k_shift(double *x, double s) { *x -= s; }

cudaError_t hook_gram(const CUtensorMap *tm_g, const int8_t *G, int ldx, const int32_t *blk_ls,
                      const int32_t *batch_blocks, int nbatch, int maxN, const int64_t *wofs, const double *freq,
                      const int32_t *perm, int n, double *W, float *W32, int ld32, int *err, cudaStream_t st)
{
    cudaError_t e = soda::zb_gram(tm_g, G, ldx, blk_ls, batch_blocks, nbatch, maxN, wofs, freq, perm, n, W, W32, ld32,
                                  err, st);
    if (e == cudaSuccess && !W32 && g_fallback_err) e = cudaMemsetAsync(err, 1, sizeof(int), st);
    return e;
}

cudaError_t hook_cholesky(const CUtensorMap *tm_a, const CUtensorMap *tm_b, double *W, const int64_t *wofs,
                          const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch, int maxN, const double *xxd,
                          int32_t *status, uint16_t *dig, double *work, int *err, cudaStream_t st)
{
    if (g_subset >= 0 && g_subset < nbatch) k_shift<<<1, 1, 0, st>>>(const_cast<double *>(xxd) + g_subset, g_shift);
    return soda::zb_cholesky(tm_a, tm_b, W, wofs, blk_ls, batch_blocks, nbatch, maxN, xxd, status, dig, work, err, st);
}

cudaError_t hook_pack(const double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks,
                      int nbatch, const int64_t *uoff, const int32_t *ulen, double *U64, float *U32,
                      __nv_bfloat16 *Uhi, __nv_bfloat16 *Ulo, cudaStream_t st)
{
    size_t total = 0;
    cudaMemGetInfo(&g_free, &total);
    return soda::zb_pack(W, wofs, blk_ls, batch_blocks, nbatch, uoff, ulen, U64, U32, Uhi, Ulo, st);
}

}  // namespace

#define zb_gram hook_gram
#define zb_cholesky hook_cholesky
#define zb_pack hook_pack
#include "../sodabayes_gb300/csrc/api.cu"

extern "C" void zbuild_hooks(int fallback_err, int subset, double shift)
{
    g_fallback_err = fallback_err;
    g_subset = subset;
    g_shift = shift;
}

// Free device memory when the factors of the last build were packed (now: at this moment).
extern "C" uint64_t zbuild_free(int now)
{
    size_t f = g_free, total = 0;
    if (now) cudaMemGetInfo(&f, &total);
    return f;
}

// Kernels and device functions of the Z build behind plain C functions, for tests of what no entry point shows: the
// Gram of given codes, and the quotients and roots that stand in for FP64's own.
#include <cudaTypedefs.h>
#include <vector>
#include "../sodabayes_gb300/csrc/zbuild.cu"

namespace {

__global__ void k_quotients(int n, const double *a, const double *b, double *root, double *inv, double *quot, double *ref)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    soda::ch_rsqrt(b[i], inv[i], root[i]);
    quot[i] = soda::ch_div(a[i], root[i], inv[i]);
    ref[i] = sqrt(b[i]);
    ref[n + i] = 1.0 / ref[i];
    ref[2 * n + i] = a[i] / root[i];
}

__global__ void k_gram_scaled(int n, const double *num, const double *f, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const soda::GramCol a = soda::gram_col(f[i], 1), b = soda::gram_col(f[n + i], 1);
    out[i] = soda::gram_scale(num[i], a.inv, a.lo, b.inv, b.lo);
}

}  // namespace

// X'X of the p SNPs of G (device memory, [p][ldx] codes, zero past the n individuals), centred and scaled by the allele
// frequencies freq; W: p x p on the device.  0, or what failed; *err: a device wait gave up.
extern "C" int hook_gram(const int8_t *G, int n, int p, int ldx, const double *freq, double *W, int *err)
{
    using namespace soda;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        return 1;
    CUtensorMap tm;
    const cuuint64_t dims[2] = {(cuuint64_t)ldx, (cuuint64_t)p}, strides[1] = {(cuuint64_t)ldx};
    const cuuint32_t box[2] = {128, 128}, es[2] = {1, 1};
    if (reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)(
            &tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t *>(G), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return 2;
    struct Small {   // subset bounds, the batch, the subset's offset, the order
        int32_t ls[2], batch, err;
        int64_t wofs;
    } h = {{0, p}, 0, 0, 0}, *d = nullptr;
    std::vector<int32_t> ident(p);
    for (int k = 0; k < p; ++k) ident[k] = k;
    int32_t *perm = nullptr;
    int rc = 3;
    if (cudaMalloc(&d, sizeof h) == cudaSuccess && cudaMalloc(&perm, sizeof(int32_t) * p) == cudaSuccess &&
        cudaMemcpy(d, &h, sizeof h, cudaMemcpyHostToDevice) == cudaSuccess &&
        cudaMemcpy(perm, ident.data(), sizeof(int32_t) * p, cudaMemcpyHostToDevice) == cudaSuccess &&
        zb_gram(&tm, G, ldx, d->ls, &d->batch, 1, p, &d->wofs, freq, perm, n, W, nullptr, 0, &d->err, 0) == cudaSuccess &&
        cudaDeviceSynchronize() == cudaSuccess &&
        cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) == cudaSuccess) {
        *err = h.err;
        rc = 0;
    }
    cudaFree(d);
    cudaFree(perm);
    return rc;
}

// root = sqrt(b), inv = 1 / root, quot = a / root, and CUDA's own values of the three in ref; all on the device.
extern "C" int hook_quotients(int n, const double *a, const double *b, double *root, double *inv, double *quot, double *ref)
{
    k_quotients<<<(n + 255) / 256, 256>>>(n, a, b, root, inv, quot, ref);
    return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}

// out = num / sqrt(pa qa pb qb) for the allele frequencies f[0 .. n-1] and f[n .. 2n-1].
extern "C" int hook_gram_scaled(int n, const double *num, const double *f, double *out)
{
    k_gram_scaled<<<(n + 255) / 256, 256>>>(n, num, f, out);
    return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}

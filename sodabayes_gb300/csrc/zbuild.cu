// zbuild.cu — construction of the SODA augmenting matrix on the GPU.
//
// Per subset b of N SNPs (get_aug_matrix, soda.f90:445-518):
//   A   = X_b'X_b from the exact integer Gram of the 0/1/2 codes, centred and
//         scaled like xxproduct (soda.f90:520-556)              k_gram_tc
//   d   = lambda_max(A) + 0.001 (soda.f90:484-486); lambda_max from a
//         fully reorthogonalised Lanczos run (lanczos.cuh) instead of the
//         reference's power iteration (soda.f90:378-401): both converge to
//         the same eigenvalue, Lanczos in far fewer products with A.
//   U   = chol(d I - A), upper (choleskyPD, soda.f90:8-47)     chol_tc.cuh
//   fallback for a failed factorisation: the reference's own sequence —
//         the unpivoted attempt up to the failing row, then the pivoted
//         factorisation (choleskyPSD, soda.f90:49-124) — in k_psd_block.
// All kernels work on a batch of subsets at once; each subset's FP64 work
// matrix W_b (N x N, column-major, ld N) lives at wofs[b].
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include "chol_tc.cuh"
#include "dgv.cuh"
#include "gram_tc.cuh"
#include "lanczos.cuh"
#include "rng.cuh"
#include "state.cuh"
#include "zbuild.cuh"

namespace soda {

// ---------------------------------------------------------------------------
// genotype ingest: bed decode, allele frequencies, centring tables
// ---------------------------------------------------------------------------

// load_geno's decode (utilities.f90:438-454): b - ((b>>1)&0x55) maps the
// 2-bit codes 00,01,10,11 to 0,1,1,2.  One thread per output byte quad.
__global__ void k_decode_bed(const uint8_t *bed, int n, int p, size_t rec_bytes, int8_t *G, int ldx)
{
    const size_t tot = (size_t)p * rec_bytes;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / rec_bytes);
        const int q = (int)(t % rec_bytes);
        uint8_t b = bed[t];
        b = (uint8_t)(b - ((b >> 1) & 0x55));
        for (int s = 0; s < 4; ++s) {
            const int i = q * 4 + s;
            if (i < n) G[(size_t)j * ldx + i] = (int8_t)((b >> (2 * s)) & 3);
        }
    }
}

// freq_j = sum(codes)/(2n) (xscale, utilities.f90:527).  One warp per SNP.
// Codes outside 0..2 are counted in *bad and replaced by 1 (a missing call).
__global__ void k_freq(int8_t *G, int n, int p, int ldx, double *freq, int *bad)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= p) return;
    int8_t *col = G + (size_t)warp * ldx;
    long long s = 0;
    int nbad = 0;
    for (int i = lane; i < n; i += 32) {
        int v = col[i];
        if (v < 0 || v > 2) {
            ++nbad;
            v = 1;
            col[i] = 1;
        }
        s += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        nbad += __shfl_xor_sync(0xffffffffu, nbad, o);
    }
    if (lane == 0) {
        freq[warp] = (double)s / (2.0 * (double)n);
        if (nbad) atomicAdd(bad, nbad);
    }
}

// Gather SNP columns into subset order and build the centring table.
__global__ void k_gather(const int8_t *Gsnp, int8_t *Gpos, const int32_t *perm, int p, int ldx)
{
    const size_t tot = (size_t)p * (ldx / 16);
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / (ldx / 16));
        const int q = (int)(t % (ldx / 16));
        reinterpret_cast<uint4 *>(Gpos + (size_t)k * ldx)[q] =
            reinterpret_cast<const uint4 *>(Gsnp + (size_t)perm[k] * ldx)[q];
    }
}

__global__ void k_xv32(const double *xv, int p, float *xv32)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 4 * p) xv32[t] = (float)xv[t];
}

__global__ void k_xv(const double *freq, const int32_t *perm, int p, double *xv)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= p) return;
    const double eps = 2.220446049250313e-16;
    const double f = freq[perm[k]];
    double *o = xv + (size_t)k * 4;
    if (f < eps || (1.0 - f) < eps) {
        o[0] = o[1] = o[2] = o[3] = 0.0;
        return;
    }
    const double sd = sqrt(__dmul_rn(__dmul_rn(2.0, f), __dsub_rn(1.0, f)));
    const double twop = __dmul_rn(2.0, f);
    o[0] = __ddiv_rn(__dsub_rn(0.0, twop), sd);
    o[1] = __ddiv_rn(__dsub_rn(1.0, twop), sd);
    o[2] = __ddiv_rn(__dsub_rn(2.0, twop), sd);
    o[3] = __ddiv_rn(1.0, sd);
}

// ---------------------------------------------------------------------------
// Gram: S = G_b'G_b and the xxproduct scaling, on the tensor cores (gram_tc.cuh);
// with dp4a on 64x64 tiles for more than GR_NMAX individuals, whose counts
// FP32 sums do not hold
// ---------------------------------------------------------------------------
constexpr int GT = 64;   // output tile
constexpr int GK = 64;   // bytes of K per stage

__global__ void __launch_bounds__(256) k_gram(const int8_t *G, int ldx, const int32_t *blk_ls,
                                              const int32_t *batch_blocks, const int64_t *wofs,
                                              const double *freq, const int32_t *perm, int n,
                                              double *W, float *W32, int ld32, size_t stride32)
{
    __shared__ int sA[GT][GK / 4 + 1];
    __shared__ int sB[GT][GK / 4 + 1];
    const int b = batch_blocks[blockIdx.y];
    const int ls = blk_ls[b], N = blk_ls[b + 1] - ls;
    const int nt = (N + GT - 1) / GT;
    // decode the upper-triangular tile index
    int t = blockIdx.x, ti = 0;
    while (ti < nt && t >= nt - ti) { t -= nt - ti; ++ti; }
    if (ti >= nt) return;
    const int tj = ti + t;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int acc[4][4] = {};
    const int lr = threadIdx.x >> 2;          // column of the tile this thread loads
    const int lq = (threadIdx.x & 3) * 4;     // first word of the 16-byte chunk
    const int ca = ti * GT + lr, cb = tj * GT + lr;
    for (int k0 = 0; k0 < ldx; k0 += GK) {
        uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
        if (ca < N) va = *reinterpret_cast<const uint4 *>(G + (size_t)(ls + ca) * ldx + k0 + lq * 4);
        if (cb < N) vb = *reinterpret_cast<const uint4 *>(G + (size_t)(ls + cb) * ldx + k0 + lq * 4);
        __syncthreads();
        sA[lr][lq + 0] = (int)va.x; sA[lr][lq + 1] = (int)va.y; sA[lr][lq + 2] = (int)va.z; sA[lr][lq + 3] = (int)va.w;
        sB[lr][lq + 0] = (int)vb.x; sB[lr][lq + 1] = (int)vb.y; sB[lr][lq + 2] = (int)vb.z; sB[lr][lq + 3] = (int)vb.w;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < GK / 4; ++w) {
            int a[4], bb[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { a[q] = sA[ty * 4 + q][w]; bb[q] = sB[tx * 4 + q][w]; }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[q][r] = __dp4a(a[q], bb[r], acc[q][r]);
        }
    }
    const double ep = 2.220446049250313e-16;
    double *Wb = W + wofs[b];
    float *Fb = W32 ? W32 + blockIdx.y * stride32 : nullptr;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int j = ti * GT + ty * 4 + q;
        if (j >= N) continue;
        const double fj = freq[perm[ls + j]];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = tj * GT + tx * 4 + r;
            if (k >= N) continue;
            const double fk = freq[perm[ls + k]];
            // the scaling takes the frequency of the later position first, like xxproduct's
            // (jj, kk) with kk <= jj (soda.f90:474-481, 553-554): products of doubles are not
            // associative, and in a diagonal tile the two threads holding (j, k) and (k, j) both
            // write both entries, so they must compute the same value
            const double fa = k > j ? fk : fj, fb = k > j ? fj : fk;
            const double qa = __dsub_rn(1.0, fa), qb = __dsub_rn(1.0, fb);
            double res;
            if (fa <= ep || qa <= ep || fb <= ep || qb <= ep) {
                res = 0.0;
            } else {
                const double pa = __dmul_rn(fa, 2.0), pb = __dmul_rn(fb, 2.0);
                const double t1 = __dmul_rn(__dmul_rn((double)n, pa), pb);
                const double den = sqrt(__dmul_rn(__dmul_rn(__dmul_rn(pa, pb), qa), qb));
                res = __ddiv_rn(__dsub_rn((double)acc[q][r], t1), den);
            }
            Wb[(size_t)j + (size_t)k * N] = res;
            Wb[(size_t)k + (size_t)j * N] = res;
            if (Fb) {
                Fb[(size_t)j + (size_t)k * ld32] = (float)res;
                Fb[(size_t)k + (size_t)j * ld32] = (float)res;
            }
        }
    }
}

__device__ double blk_sum(double v, double *sh)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        double t = lane < nw ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

// M = d I - A in place (soda.f90:487-490)
__global__ void k_form_m(double *W, const int64_t *wofs, const int32_t *blk_ls,
                         const int32_t *batch_blocks, const double *xxd)
{
    const int b = batch_blocks[blockIdx.y];
    const int N = blk_ls[b + 1] - blk_ls[b];
    double *A = W + wofs[b];
    const double d = xxd[b];
    const size_t tot = (size_t)N * N;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(t % N), j = (int)(t / N);
        const double v = -A[t];
        A[t] = i == j ? d + v : v;
    }
}

// column lengths of PD subsets: column jj of the subset holds rows 0..jj
__global__ void k_pd_lengths(const int32_t *blk_ls, const int32_t *batch_blocks, const int32_t *status,
                             int32_t *ulen, uint8_t *skip)
{
    const int b = batch_blocks[blockIdx.y];
    if (status[b] != 0) return;
    const int ls = blk_ls[b], N = blk_ls[b + 1] - ls;
    for (int jj = blockIdx.x * blockDim.x + threadIdx.x; jj < N; jj += gridDim.x * blockDim.x) {
        ulen[ls + jj] = jj + 1;
        skip[ls + jj] = 0;
    }
}

// ---------------------------------------------------------------------------
// failed factorisation: the reference's sequence on one subset, one CTA.
// M (N x N) holds d I - A on entry (scratch, destroyed).  W_b receives the
// columns the reference leaves in XA(1:N, ls:le): rows of the unpivoted
// attempt before the failing row, overwritten by the pivoted factor.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_psd_block(double *Wb, double *M, int N, int ls,
                                                    int32_t *ulen, uint8_t *skip, int32_t *piv_out,
                                                    int32_t *rank_out, int32_t *status_out, double *work)
{
    __shared__ double sh[33];
    __shared__ int s_fail, s_pvt, s_stop;
    __shared__ double s_ajj;
    const int tid = threadIdx.x;
    // (1) choleskyPD attempt (soda.f90:8-47), up-looking, into Wb
    if (tid == 0) s_fail = 0;
    __syncthreads();
    for (int i = tid; i < N; i += blockDim.x)
        if (M[(size_t)i * N + i] <= 0.0) s_fail = -1;
    __syncthreads();
    int ifail = 0;   // rows [0, ifail) of the attempt are written
    if (s_fail == 0) {
        for (size_t t = tid; t < (size_t)N * N; t += blockDim.x) Wb[t] = 0.0;
        __syncthreads();
        for (int i = 0; i < N; ++i) {
            double part = 0.0;
            for (int k = tid; k < i; k += blockDim.x) part += Wb[k + (size_t)i * N] * Wb[k + (size_t)i * N];
            const double dd = blk_sum(part, sh);
            const double tmp = M[i + (size_t)i * N] - dd;
            if (tmp <= 0.0 || isnan(tmp)) { ifail = i; break; }
            const double uii = sqrt(tmp);
            if (tid == 0) Wb[i + (size_t)i * N] = uii;
            for (int j = i + 1 + tid; j < N; j += blockDim.x) {
                double dj = 0.0;
                for (int k = 0; k < i; ++k) dj += Wb[k + (size_t)j * N] * Wb[k + (size_t)i * N];
                Wb[i + (size_t)j * N] = (M[j + (size_t)i * N] - dj) / uii;
            }
            __syncthreads();
            ifail = i + 1;
        }
    } else {
        for (size_t t = tid; t < (size_t)N * N; t += blockDim.x) Wb[t] = 0.0;
    }
    __syncthreads();
    // (2) choleskyPSD (soda.f90:49-124) on M in place
    double *wk = work;   // [2N]
    const double EPS = 2.220446049250313e-16;
    if (tid == 0) {
        int pvt = 0;
        double best = M[0];
        for (int t = 1; t < N; ++t)
            if (M[(size_t)t * N + t] > best) { best = M[(size_t)t * N + t]; pvt = t; }
        s_pvt = pvt;
        s_ajj = best;
        s_stop = 0;
    }
    for (int t = tid; t < N; t += blockDim.x) { piv_out[t] = t + 1; wk[t] = 0.0; }
    __syncthreads();
    if (s_ajj <= EPS) {
        if (tid == 0) { *status_out = -1; *rank_out = 0; }
        return;
    }
    const double DSTOP = N * EPS * s_ajj;
    int rank = N;
    for (int j = 0; j < N; ++j) {
        for (int p = j + tid; p < N; p += blockDim.x) {
            if (j > 0) wk[p] = wk[p] + M[(j - 1) + (size_t)p * N] * M[(j - 1) + (size_t)p * N];
            wk[N + p] = M[p + (size_t)p * N] - wk[p];
        }
        __syncthreads();
        if (tid == 0) {
            if (j > 0) {
                int pv = j;
                double best = wk[N + j];
                for (int p = j + 1; p < N; ++p)
                    if (wk[N + p] > best) { best = wk[N + p]; pv = p; }
                s_pvt = pv;
                s_ajj = best;
                if (best <= DSTOP) {
                    M[j + (size_t)j * N] = best;
                    s_stop = 1;
                }
            }
        }
        __syncthreads();
        if (s_stop) { rank = j; break; }
        const int pvt = s_pvt;
        if (j != pvt) {
            if (tid == 0) M[pvt + (size_t)pvt * N] = M[j + (size_t)j * N];
            __syncthreads();
            for (int t = tid; t < j; t += blockDim.x) {   // rows 0..j-1 of columns j and pvt
                const double a = M[t + (size_t)j * N];
                M[t + (size_t)j * N] = M[t + (size_t)pvt * N];
                M[t + (size_t)pvt * N] = a;
            }
            for (int t = tid; t < pvt - j - 1; t += blockDim.x) {   // row j (cols j+1..) <-> col pvt (rows j+1..)
                const double a = M[j + (size_t)(j + 1 + t) * N];
                M[j + (size_t)(j + 1 + t) * N] = M[(j + 1 + t) + (size_t)pvt * N];
                M[(j + 1 + t) + (size_t)pvt * N] = a;
            }
            for (int t = tid; t < N - pvt - 1; t += blockDim.x) {   // rows j and pvt, cols pvt+1..
                const double a = M[j + (size_t)(pvt + 1 + t) * N];
                M[j + (size_t)(pvt + 1 + t) * N] = M[pvt + (size_t)(pvt + 1 + t) * N];
                M[pvt + (size_t)(pvt + 1 + t) * N] = a;
            }
            if (tid == 0) {
                const double dt = wk[j];
                wk[j] = wk[pvt];
                wk[pvt] = dt;
                const int it = piv_out[pvt];
                piv_out[pvt] = piv_out[j];
                piv_out[j] = it;
            }
            __syncthreads();
        }
        const double ajj = sqrt(s_ajj);
        if (tid == 0) M[j + (size_t)j * N] = ajj;
        __syncthreads();
        if (j < N - 1) {
            const double sc = 1.0 / ajj;
            for (int jc = j + 1 + tid; jc < N; jc += blockDim.x) {
                double temp = 0.0;
                for (int i = 0; i < j; ++i) temp = temp + M[i + (size_t)jc * N] * M[i + (size_t)j * N];
                const double v = M[j + (size_t)jc * N] + (-1.0) * temp;
                M[j + (size_t)jc * N] = sc * v;
            }
        }
        __syncthreads();
    }
    __syncthreads();
    // (3) scatter: XA(1:j, ls+jj-1) = factor(1:j, j) for j <= rank, else skip
    for (int j = tid; j < N; j += blockDim.x) {
        const int jj = piv_out[j] - 1;   // 0-based subset column
        const int jj_stale = ifail < (jj + 1) ? ifail : (jj + 1);   // rows written by the attempt
        if (j < rank) {
            for (int i = 0; i <= j; ++i) Wb[i + (size_t)jj * N] = M[i + (size_t)j * N];
            ulen[ls + jj] = (j + 1) > jj_stale ? (j + 1) : jj_stale;
            skip[ls + jj] = 0;
        } else {
            // skipped column: XA keeps the rows of the unpivoted attempt
            ulen[ls + jj] = jj_stale;
            skip[ls + jj] = 1;
        }
    }
    if (tid == 0) { *rank_out = rank; *status_out = 0; }
}

// ---------------------------------------------------------------------------
// pack the factors into ragged columns in the sweep's precision
// ---------------------------------------------------------------------------
__global__ void k_pack(const double *W, const int64_t *wofs, const int32_t *blk_ls,
                       const int32_t *batch_blocks, const int64_t *uoff, const int32_t *ulen,
                       double *U64, float *U32, __nv_bfloat16 *Uhi, __nv_bfloat16 *Ulo)
{
    const int b = batch_blocks[blockIdx.y];
    const int ls = blk_ls[b], N = blk_ls[b + 1] - ls;
    const double *Wb = W + wofs[b];
    for (int jj = blockIdx.x; jj < N; jj += gridDim.x) {
        const int len = ulen[ls + jj];
        const int64_t off = uoff[ls + jj];
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            const double v = Wb[(size_t)i + (size_t)jj * N];
            if (U64) U64[off + i] = v;
            if (U32) U32[off + i] = (float)v;
            if (Uhi) {
                const __nv_bfloat16 hi = __double2bfloat16(v);
                const double rem = v - (double)__bfloat162float(hi);
                Uhi[off + i] = hi;
                Ulo[off + i] = __double2bfloat16(rem);
            }
        }
    }
}

// dense XA(bs, nloci) from the ragged columns (for inspection)
__global__ void k_unpack_dense(const double *U64, const int64_t *uoff, const int32_t *ulen, int p, int bs,
                               double *xa)
{
    const size_t tot = (size_t)p * bs;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < tot; t += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(t / bs), i = (int)(t % bs);
        xa[t] = i < ulen[k] ? U64[uoff[k] + i] : 0.0;
    }
}

// ---------------------------------------------------------------------------
// host wrappers
// ---------------------------------------------------------------------------
cudaError_t zb_decode_bed(const uint8_t *bed, int n, int p, int8_t *G, int ldx, cudaStream_t st)
{
    const size_t rec = ((size_t)n + 3) / 4;
    k_decode_bed<<<1024, 256, 0, st>>>(bed, n, p, rec, G, ldx);
    return cudaGetLastError();
}

cudaError_t zb_freq(int8_t *G, int n, int p, int ldx, double *freq, int *bad, cudaStream_t st)
{
    k_freq<<<(int)(((size_t)p * 32 + 255) / 256), 256, 0, st>>>(G, n, p, ldx, freq, bad);
    return cudaGetLastError();
}

cudaError_t zb_gather(const int8_t *Gsnp, int8_t *Gpos, const int32_t *perm, int p, int ldx, cudaStream_t st)
{
    k_gather<<<2048, 256, 0, st>>>(Gsnp, Gpos, perm, p, ldx);
    return cudaGetLastError();
}

cudaError_t zb_xv(const double *freq, const int32_t *perm, int p, double *xv, cudaStream_t st)
{
    k_xv<<<(p + 255) / 256, 256, 0, st>>>(freq, perm, p, xv);
    return cudaGetLastError();
}

cudaError_t zb_xv32(const double *xv, int p, float *xv32, cudaStream_t st)
{
    k_xv32<<<(4 * p + 255) / 256, 256, 0, st>>>(xv, p, xv32);
    return cudaGetLastError();
}

cudaError_t zb_gram(const CUtensorMap *tm_g, const int8_t *G, int ldx, const int32_t *blk_ls,
                    const int32_t *batch_blocks, int nbatch, int maxN, const int64_t *wofs, const double *freq,
                    const int32_t *perm, int n, double *W, float *W32, int ld32, int *err, cudaStream_t st)
{
    const size_t stride32 = (size_t)ld32 * maxN;
    if (n <= GR_NMAX) {
        cudaError_t e = cudaFuncSetAttribute(k_gram_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GR_SMEM);
        if (e != cudaSuccess) return e;
        const int nt = (maxN + GR_T - 1) / GR_T;
        k_gram_tc<<<dim3(nt * (nt + 1) / 2, nbatch), GR_THREADS, GR_SMEM, st>>>(
            *tm_g, ldx, blk_ls, batch_blocks, wofs, freq, perm, n, W, W32, ld32, stride32, err);
        return cudaGetLastError();
    }
    const int nt = (maxN + GT - 1) / GT;
    k_gram<<<dim3(nt * (nt + 1) / 2, nbatch), 256, 0, st>>>(G, ldx, blk_ls, batch_blocks, wofs, freq, perm, n, W, W32,
                                                            ld32, stride32);
    return cudaGetLastError();
}

// Launch with programmatic stream serialization (the kernels wait for the one before them by themselves).
template <typename... KArgs, typename... Args>
static cudaError_t launch_after(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                Args... args)
{
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
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <typename T>
static size_t lz_smem(int maxN, int mmax)
{
    return sizeof(T) * (size_t)(3 * mmax + (maxN + LZ_CTAS - 1) / LZ_CTAS);
}

int zb_lz_pre() { return LZ_PRE; }

// Column splits of a product: about four CTAs an SM (152 of them), at most LZ_VCOLS columns each.
template <typename T>
static int lz_splits(int maxN, int nbatch)
{
    const int tiles = (maxN + LzTile<T>::v - 1) / LzTile<T>::v * nbatch;
    return std::max((maxN + LZ_VCOLS - 1) / LZ_VCOLS, std::min(LZ_SPLITS, (608 + tiles - 1) / tiles));
}

size_t zb_lz_wpart(int maxN, int nbatch)
{
    return (size_t)nbatch * std::max(LZ_SPLITS, (maxN + LZ_VCOLS - 1) / LZ_VCOLS) * maxN;
}

template <typename T>
static cudaError_t lz_step(const T *A, const int64_t *aofs, size_t astride, int ld, const int32_t *blk_ls,
                           const int32_t *batch_blocks, int nbatch, int maxN, size_t vstride, T *V, T *wpart, T *alpha,
                           T *beta, int mmax, int j, const uint8_t *done, cudaStream_t st)
{
    const int nsp = lz_splits<T>(maxN, nbatch);
    cudaError_t e = launch_after(k_lz_matvec<T>, dim3((maxN + LzTile<T>::v - 1) / LzTile<T>::v, nsp, nbatch),
                                 dim3(LZ_THREADS), 0, st, A, aofs, astride, ld, blk_ls, batch_blocks, vstride,
                                 (const T *)V, wpart, maxN, j, done);
    if (e == cudaSuccess)
        e = launch_after(k_lz_orth<T>, dim3(LZ_CTAS * nbatch), dim3(LZ_THREADS), lz_smem<T>(maxN, mmax), st, blk_ls,
                         batch_blocks, vstride, V, (const T *)wpart, nsp, maxN, alpha, beta, mmax, j, done);
    return e;
}

cudaError_t zb_lz_start(const float *W32, int ld32, const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch,
                        int maxN, size_t vstride, double *V, float *V32, float *wpart32, float *ab32, uint64_t seed,
                        cudaStream_t st)
{
    const size_t vstride32 = (size_t)LZ_PRE * maxN;
    float *alpha = ab32, *beta = ab32 + (size_t)nbatch * LZ_PRE;
    // FP32 steps: about as many as take the vector to FP32's 1e-6 (40 at N = 300, over a hundred at N = 2000); too few
    // cost FP64 steps, three times as long
    const int steps = std::min(std::min(LZ_PRE, maxN), 16 + maxN / 12);
    cudaError_t e = cudaMemsetAsync(ab32, 0, sizeof(float) * 2 * nbatch * LZ_PRE, st);
    if (e != cudaSuccess) return e;
    k_lz_init<float><<<nbatch, 1024, 0, st>>>(blk_ls, batch_blocks, vstride32, V32, seed);
    e = cudaGetLastError();
    for (int j = 0; j < steps && e == cudaSuccess; ++j)
        e = lz_step<float>(W32, nullptr, (size_t)ld32 * maxN, ld32, blk_ls, batch_blocks, nbatch, maxN, vstride32, V32,
                           wpart32, alpha, beta, LZ_PRE, j, nullptr, st);
    if (e != cudaSuccess) return e;
    k_lz_ritz<<<nbatch, 1024, 0, st>>>(blk_ls, batch_blocks, vstride32, V32, alpha, beta, steps, vstride, V);
    return cudaGetLastError();
}

cudaError_t zb_lz_step(const double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks,
                       int nbatch, int maxN, size_t vstride, double *V, double *wpart, double *alpha, double *beta,
                       int mmax, int j, const uint8_t *done, cudaStream_t st)
{
    return lz_step<double>(W, wofs, 0, 0, blk_ls, batch_blocks, nbatch, maxN, vstride, V, wpart, alpha, beta, mmax, j,
                           done, st);
}

cudaError_t zb_lz_prepare(int maxN, int mmax)
{
    cudaError_t e = cudaFuncSetAttribute(k_lz_orth<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)lz_smem<double>(maxN, mmax));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_lz_orth<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)lz_smem<float>(maxN, LZ_PRE));
    return e;
}

cudaError_t zb_form_m(double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch,
                      const double *xxd, cudaStream_t st)
{
    k_form_m<<<dim3(256, nbatch), 256, 0, st>>>(W, wofs, blk_ls, batch_blocks, xxd);
    return cudaGetLastError();
}

int zb_chol_np(int maxN) { return (maxN + CH_M - 1) / CH_M * CH_M; }
int zb_chol_ldt(int maxN) { return (maxN + CH_P - 1) / CH_P * CH_P; }
size_t zb_chol_digits(int maxN) { return (size_t)CH_DIG * zb_chol_np(maxN) * zb_chol_ldt(maxN); }
size_t zb_chol_work(int maxN, int nbatch) { return (size_t)nbatch * (2 * zb_chol_np(maxN) + CH_P); }

cudaError_t zb_cholesky(const CUtensorMap *tm_a, const CUtensorMap *tm_b, double *W, const int64_t *wofs,
                        const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch, int maxN, const double *xxd,
                        int32_t *status, uint16_t *dig, double *work, int *err, cudaStream_t st)
{
    const int np = zb_chol_np(maxN), ldt = zb_chol_ldt(maxN);
    double *sc = work, *nrm = sc + (size_t)nbatch * np, *piv = nrm + (size_t)nbatch * np;
    cudaError_t e = cudaFuncSetAttribute(k_ch_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_ch_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CH_TRSM_SMEM);
    if (e != cudaSuccess) return e;
    k_ch_init<<<nbatch, 256, 0, st>>>(W, wofs, blk_ls, batch_blocks, xxd, sc, nrm, np, status);
    e = cudaGetLastError();
    for (int i0 = 0; i0 < maxN && e == cudaSuccess; i0 += CH_P) {
        e = launch_after(k_ch_update, dim3((maxN - i0 + CH_M - 1) / CH_M, nbatch), dim3(CH_THREADS), CH_SMEM, st, *tm_a,
                         *tm_b, W, wofs, blk_ls, batch_blocks, xxd, (const double *)sc, np, status, i0, err);
        if (e == cudaSuccess)
            e = launch_after(k_ch_diag, dim3(nbatch), dim3(256), 0, st, W, wofs, blk_ls, batch_blocks, status, i0, piv);
        if (e == cudaSuccess && maxN - i0 > CH_P)
            e = launch_after(k_ch_trsm, dim3((maxN - i0 - CH_P + 31) / 32, nbatch), dim3(128), CH_TRSM_SMEM, st, W, wofs, blk_ls,
                             batch_blocks, xxd, (const double *)sc, nrm, np, status, i0, (const double *)piv, dig, ldt);
    }
    return e;
}

cudaError_t zb_pd_lengths(const int32_t *blk_ls, const int32_t *batch_blocks, int nbatch, const int32_t *status,
                          int32_t *ulen, uint8_t *skip, cudaStream_t st)
{
    k_pd_lengths<<<dim3(8, nbatch), 256, 0, st>>>(blk_ls, batch_blocks, status, ulen, skip);
    return cudaGetLastError();
}

cudaError_t zb_psd_block(double *Wb, double *M, int N, int ls, int32_t *ulen, uint8_t *skip, int32_t *piv,
                         int32_t *rank, int32_t *status, double *work, cudaStream_t st)
{
    k_psd_block<<<1, 1024, 0, st>>>(Wb, M, N, ls, ulen, skip, piv, rank, status, work);
    return cudaGetLastError();
}

cudaError_t zb_pack(const double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks,
                    int nbatch, const int64_t *uoff, const int32_t *ulen, double *U64, float *U32,
                    __nv_bfloat16 *Uhi, __nv_bfloat16 *Ulo, cudaStream_t st)
{
    k_pack<<<dim3(512, nbatch), 256, 0, st>>>(W, wofs, blk_ls, batch_blocks, uoff, ulen, U64, U32, Uhi, Ulo);
    return cudaGetLastError();
}

cudaError_t zb_unpack_dense(const double *U64, const int64_t *uoff, const int32_t *ulen, int p, int bs, double *xa,
                            cudaStream_t st)
{
    k_unpack_dense<<<2048, 256, 0, st>>>(U64, uoff, ulen, p, bs, xa);
    return cudaGetLastError();
}

int zb_dgv_splits(int n, int p) { return dgv_splits(n, p); }

cudaError_t zb_dgv(const int8_t *G, int ldx, const double *xv, const double *freq, const int32_t *perm,
                   const double *eff, int n, int p, double mu, double *part, double *pred, cudaStream_t st)
{
    return dgv_enqueue<DGV_PADDED>(reinterpret_cast<const uint8_t *>(G), ldx, xv, freq, perm, eff, n, p, mu, part, n,
                                   dgv_splits(n, p), pred, st);
}

int zb_dgv_bed(const uint8_t *bed, const double *freq, const double *eff, int n, int p, double *part, int nsplit,
               cudaStream_t st)
{
    return dgv_enqueue_tab<DGV_BED>(bed, ((size_t)n + 3) / 4, nullptr, freq, nullptr, eff, n, p, part, n, nsplit, st);
}

cudaError_t zb_dgv_sum(const double *part, int n, int nsplit, double mu, double *pred, cudaStream_t st)
{
    return dgv_enqueue_sum(part, n, n, nsplit, mu, pred, st);
}

}  // namespace soda

// gram_tc.cuh — genotype Gram G_b'G_b of a batch of subsets on tcgen05, with the xxproduct scaling
// (soda.f90:520-556), included by zbuild.cu.
//
// The codes 0, 1, 2 of a job are E4M3 numbers as they lie in memory: the bytes 0x00, 0x01, 0x02 are 0 and the
// subnormals 2^-9 and 2^-8.  So the int8 matrix is the operand of a kind::f8f6f4 GEMM without any conversion; its
// products are integers times 2^-18, and their FP32 sums are exact while 4 n <= 2^24.
//
// One CTA per 128 x 128 tile of the upper triangle, two CTAs an SM: the FP64 scaling of a tile (about ten
// instructions an element, 40 us on the SM's narrow FP64 pipe) runs while the other CTA's MMAs do.  It is the larger
// part of the kernel (FP64 pipe 45% active, tensor pipe 26%, by ncu): 10 subsets of 2000 SNPs and 20,000 individuals
// take 0.62 ms, 7.1 ms with dp4a on the integer pipe.
//
// Warps 0-3 scale and store, warp 4 loads 128 SNPs x 128 individuals of both sides by TMA (128-byte swizzle), warp 5
// issues the MMAs.
#pragma once
#include <cuda.h>
#include "tc.cuh"

namespace soda {

constexpr int GR_T = 128;                    // SNPs per tile side
constexpr int GR_K = 128;                    // individuals per stage
constexpr int GR_NS = 3;                     // stages in flight
constexpr int GR_BYTES = GR_T * GR_K;        // one side of a stage
constexpr size_t GR_SMEM = 1024 + (size_t)GR_NS * 2 * GR_BYTES;
constexpr int GR_THREADS = 192;
constexpr int GR_NMAX = 1 << 22;             // individuals: 4 n <= 2^24

// res = (S - n pa pb) / sqrt(pa qa pb qb) for the SNP pair (a, b), a the later position, 0 where one is
// monomorphic; p = 2 f, q = 1 - f.  A division an element would take longer than everything else, so each SNP has
// 1 / sqrt(p q) in twice the working precision (Dekker, "A floating-point technique for extending the available
// precision", Numer. Math. 18, 1971), and a quotient is a product: two roundings, of the numerator and of the result.
// With rounded standard deviations the diagonal was off by their rounding twice, more than the rest of it.
struct GramCol {
    double p, np, inv, lo;
};
__device__ __forceinline__ GramCol gram_col(double f, int n)
{
    const double ep = 2.220446049250313e-16, q = __dsub_rn(1.0, f);
    GramCol c;
    c.p = __dmul_rn(f, 2.0);
    c.np = __dmul_rn((double)n, c.p);
    c.inv = c.lo = 0.0;
    if (f <= ep || q <= ep) return c;
    const double ql = __dsub_rn(__dsub_rn(1.0, q), f);   // 1 - f = q + ql
    const double v = __dmul_rn(c.p, q), vl = fma(c.p, ql, fma(c.p, q, -v));
    c.inv = 1.0 / sqrt(v);
    const double s = __dmul_rn(c.inv, c.inv), sl = fma(c.inv, c.inv, -s);
    c.lo = 0.5 * c.inv * (fma(-v, s, 1.0) - fma(v, sl, vl * s));   // half of 1 - (v + vl) inv^2
    return c;
}
// num (inva + loa) (invb + lob), rounded once.
__device__ __forceinline__ double gram_scale(double num, double inva, double loa, double invb, double lob)
{
    const double r = __dmul_rn(inva, invb);
    return fma(num, r, num * fma(loa, invb, fma(inva, lob, fma(inva, invb, -r))));
}

__global__ void __launch_bounds__(GR_THREADS, 2)
    k_gram_tc(const __grid_constant__ CUtensorMap tm_g, int ldx, const int32_t *blk_ls, const int32_t *batch_blocks,
              const int64_t *wofs, const double *freq, const int32_t *perm, int n, double *W, float *W32, int ld32,
              size_t stride32, int *err)
{
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    __shared__ uint64_t s_full[GR_NS], s_free[GR_NS], s_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    __shared__ double s_np[GR_T], s_inv[GR_T], s_lo[GR_T];
    const int b = batch_blocks[blockIdx.y];
    const int ls = blk_ls[b], N = blk_ls[b + 1] - ls, nt = (N + GR_T - 1) / GR_T;
    // the upper-triangular tile (ti, tj), ti <= tj
    int t = blockIdx.x, ti = 0;
    while (ti < nt && t >= nt - ti) { t -= nt - ti; ++ti; }
    if (ti >= nt) return;
    const int tj = ti + t;
    unsigned char *raw0 = smem_dyn + ((1024u - (tc::smem_u32(smem_dyn) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ns = ldx / GR_K;
    if (tid == 0) {
        for (int i = 0; i < GR_NS; ++i) {
            tc::mbar_init(&s_full[i], 1);
            tc::mbar_init(&s_free[i], 1);
        }
        tc::mbar_init(&s_done, 1);
        tc::mbar_fence_init();
        s_err = 0;
    }
    if (warp == 5) tc::tmem_alloc(&s_tmem, 128);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = s_tmem;
    const bool diag = ti == tj;
    if (warp == 4) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tm_g);
            int issued = 0;
            for (int s = 0; s < ns; ++s) {
                const int sl = s % GR_NS;
                if (s >= GR_NS && !tc::mbar_wait(&s_free[sl], ((s / GR_NS) - 1) & 1, tc::BUILD_WAIT_NS)) {
                    s_err = 1;
                    break;
                }
                unsigned char *dst = raw0 + (size_t)sl * 2 * GR_BYTES;
                tc::mbar_expect_tx(&s_full[sl], diag ? GR_BYTES : 2 * GR_BYTES);
                tc::tma_load_2d(dst, &tm_g, s * GR_K, ls + ti * GR_T, &s_full[sl]);
                if (!diag) tc::tma_load_2d(dst + GR_BYTES, &tm_g, s * GR_K, ls + tj * GR_T, &s_full[sl]);
                issued = s + 1;
            }
            // no copy may still be in flight into this CTA's shared memory when it exits
            for (int s = max(0, issued - GR_NS); s < issued; ++s)
                if (!tc::mbar_wait(&s_full[s % GR_NS], (s / GR_NS) & 1, tc::BUILD_WAIT_NS)) s_err = 1;
        }
    } else if (warp == 5) {
        const bool leader = tc::elect_one();
        const uint32_t idesc = tc::idesc_e4m3(GR_T, GR_T);
        for (int s = 0; s < ns; ++s) {
            const int sl = s % GR_NS;
            if (!__all_sync(0xffffffffu, tc::mbar_wait(&s_full[sl], (s / GR_NS) & 1, tc::BUILD_WAIT_NS))) {
                s_err = 1;
                break;
            }
            tc::fence_after_sync();
            if (leader) {
                const uint32_t a = tc::smem_u32(raw0 + (size_t)sl * 2 * GR_BYTES), bb = diag ? a : a + GR_BYTES;
#pragma unroll
                for (int kk = 0; kk < GR_K / 32; ++kk)
                    tc::mma_e4m3(tm, tc::desc_sw128(a + 32 * kk, 1024), tc::desc_sw128(bb + 32 * kk, 1024), idesc,
                                 (s | kk) != 0 ? 1u : 0u);
                tc::mma_commit(&s_free[sl]);
            }
            __syncwarp();
        }
        if (leader) tc::mma_commit(&s_done);
        __syncwarp();
    } else {
        const int j = ti * GR_T + tid;   // this thread's row; its columns are the tile's tj side
        GramCol row = gram_col(j < N ? freq[perm[ls + j]] : 0.0, n);
        {
            const int k = tj * GR_T + tid;
            const GramCol c = gram_col(k < N ? freq[perm[ls + k]] : 0.0, n);
            s_np[tid] = c.np;
            s_inv[tid] = c.inv;
            s_lo[tid] = c.lo;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (!tc::mbar_wait(&s_done, 0, tc::BUILD_WAIT_NS)) s_err = 1;   // every stage: up to 32,768
        tc::fence_after_sync();
        double *Wb = W + wofs[b];
        float *Fb = W32 ? W32 + blockIdx.y * stride32 : nullptr;
#pragma unroll 1
        for (int g = 0; g < GR_T / 8; ++g) {
            float v[8];
            tc::tmem_ld8(tm + ((uint32_t)(32 * warp) << 16) + 8 * g, v);
            tc::tmem_wait_ld();
            const int k0 = tj * GR_T + 8 * g;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int k = k0 + e;
                if (j >= N || k >= N || k < j) continue;
                const double num = fma(-s_np[8 * g + e], row.p, (double)(v[e] * 262144.0f));
                const double res = gram_scale(num, row.inv, row.lo, s_inv[8 * g + e], s_lo[8 * g + e]);
                Wb[(size_t)j + (size_t)k * N] = res;
                Wb[(size_t)k + (size_t)j * N] = res;
                if (Fb) {
                    Fb[(size_t)j + (size_t)k * ld32] = (float)res;
                    Fb[(size_t)k + (size_t)j * ld32] = (float)res;
                }
            }
        }
        tc::fence_before_sync();
    }
    __syncthreads();
    if (tid == 0 && s_err) atomicExch(err, 1);
    if (warp == 5) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, 128);
    }
}

}  // namespace soda

// lanczos.cuh — largest eigenvalue of every subset's X_b'X_b (power_method, soda.f90:378-401), included by zbuild.cu.
//
// Fully reorthogonalised Lanczos in FP64, started from a vector that LZ_PRE steps of the same recurrence in FP32 have
// already turned towards the top eigenvector: the FP64 steps, whose products with the matrix are bound by the FP64
// pipe (N^2 multiply-adds, 64 us for 10 subsets of 2000) as well as by twice the bytes, only have to take the error
// from FP32's 1e-6 down, and they decide when the eigenvalue has converged, as they did from a random start.
//
// A step is a product with the matrix (k_lz_matvec: tiles of rows x column splits, so that a few subsets fill the
// chip) and the recurrence with its reorthogonalisation (k_lz_orth: a cluster of LZ_CTAS CTAs per subset, which
// exchange their partial dot products through distributed shared memory; on one SM the dot products alone were 110 us
// of its FP64 pipe).  Measured, 10 subsets of 2000 SNPs (n = 20,000, LD blocks): 128 FP32 steps of 32 +
// 21 us and 40 FP64 steps of 84 + 27 us, 11.4 ms, against 46.7 ms for 112 FP64 steps of 279 + 139 us; with other data
// of the same kind 24 FP64 steps did, 9.8 ms.  The eigenvalue is off by 1.25e-16 (relative rms, 44 subsets of 96 to
// 1000 SNPs; 1.33e-16 from a random start).
#pragma once
#include <cooperative_groups.h>
#include "rng.cuh"
#include "tc.cuh"

namespace soda {

constexpr int LZ_PRE = 128;      // FP32 steps at most
constexpr int LZ_CTAS = 8;       // CTAs of a subset's recurrence
constexpr int LZ_THREADS = 256;
constexpr int LZ_SPLITS = 16;    // column splits of a product, more only for their LZ_VCOLS columns
constexpr int LZ_VCOLS = 2048;   // columns of a split at most (its part of the vector is staged in shared memory)

template <typename T>
__device__ __forceinline__ T lz_warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum over the block, the same in every thread
template <typename T>
__device__ __forceinline__ T lz_block_sum(T v, T *sh /* >= 33 */)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = lz_warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        const T t = lz_warp_sum(lane < nw ? sh[lane] : (T)0.0);
        if (lane == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

// Start vector: the i-th uniform of the (seed, subset, P_POWER) stream, like the reference's random start
// (soda.f90:390), normalised.  V: [batch][mmax][N], subsets vstride apart.
template <typename T>
__global__ void __launch_bounds__(1024) k_lz_init(const int32_t *blk_ls, const int32_t *batch_blocks, size_t vstride,
                                                  T *V, uint64_t seed)
{
    __shared__ double sh[33];
    const int b = batch_blocks[blockIdx.x];
    const int N = blk_ls[b + 1] - blk_ls[b];
    T *v = V + vstride * blockIdx.x;
    double ss = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        CRng R;
        crng_init(R, seed, 0, 0, b, P_POWER);
        R.c3 += (uint32_t)(i >> 1);
        double x = crng_unit(R);
        if (i & 1) x = crng_unit(R);
        v[i] = (T)x;
        ss += x * x;
    }
    const double inv = 1.0 / sqrt(lz_block_sum(ss, sh));
    for (int i = threadIdx.x; i < N; i += blockDim.x) v[i] = (T)((double)v[i] * inv);
}

// wpart[(batch * splits + split) * ldw + i] = the split's columns' part of (A v_j)_i.  A is symmetric and its columns
// are contiguous: a warp takes 64 (FP64) or 128 (FP32: 16-byte loads, columns padded to ld) rows and every eighth
// column, and the eight warps' sums are added in order.
template <typename T>
struct LzTile { static constexpr int v = sizeof(T) == 8 ? 64 : 128; };

template <typename T>
__global__ void __launch_bounds__(LZ_THREADS)
    k_lz_matvec(const T *A0, const int64_t *aofs, size_t astride, int ld, const int32_t *blk_ls,
                const int32_t *batch_blocks, size_t vstride, const T *V, T *wpart, int ldw, int j, const uint8_t *done)
{
    constexpr int TILE = LzTile<T>::v, RPT = TILE / 32;
    __shared__ T s_v[LZ_VCOLS];
    __shared__ T s_p[LZ_THREADS / 32][TILE];
    const int bi = blockIdx.z, b = batch_blocks[bi], nsp = gridDim.y;
    const int N = blk_ls[b + 1] - blk_ls[b];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i0 = blockIdx.x * TILE;
    tc::pdl_trigger();
    tc::pdl_wait();
    if (i0 >= N || (done && done[bi])) return;
    const int lda = ld > 0 ? ld : N;
    const T *A = A0 + (aofs ? aofs[b] : (int64_t)(astride * bi));
    const T *v = V + vstride * bi + (size_t)j * N;
    const int k0 = (int)((long long)N * blockIdx.y / nsp), k1 = (int)((long long)N * (blockIdx.y + 1) / nsp);
    for (int k = threadIdx.x; k < k1 - k0; k += LZ_THREADS) s_v[k] = v[k0 + k];
    __syncthreads();
    T acc[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) acc[q] = (T)0.0;
    if constexpr (sizeof(T) == 4) {
        const T *a = A + i0 + 4 * lane;   // rows past N: inside the padded column, not used
        const bool in = i0 + 4 * lane < ld;
        if (in) {
#pragma unroll 8
            for (int k = k0 + warp; k < k1; k += LZ_THREADS / 32) {
                const float4 x = *reinterpret_cast<const float4 *>(a + (size_t)k * lda);
                const T y = s_v[k - k0];
                acc[0] = fmaf(x.x, y, acc[0]);
                acc[1] = fmaf(x.y, y, acc[1]);
                acc[2] = fmaf(x.z, y, acc[2]);
                acc[3] = fmaf(x.w, y, acc[3]);
            }
        }
#pragma unroll
        for (int q = 0; q < RPT; ++q) s_p[warp][4 * lane + q] = acc[q];
    } else {
        const T *a[RPT];   // rows past N repeat the last one and are not used
#pragma unroll
        for (int q = 0; q < RPT; ++q) a[q] = A + min(i0 + 32 * q + lane, N - 1);
#pragma unroll 8
        for (int k = k0 + warp; k < k1; k += LZ_THREADS / 32) {
            const T y = s_v[k - k0];
#pragma unroll
            for (int q = 0; q < RPT; ++q) acc[q] = fma(a[q][(size_t)k * lda], y, acc[q]);
        }
#pragma unroll
        for (int q = 0; q < RPT; ++q) s_p[warp][32 * q + lane] = acc[q];
    }
    __syncthreads();
    if (threadIdx.x < TILE && i0 + (int)threadIdx.x < N) {
        T t = (T)0.0;
#pragma unroll
        for (int w = 0; w < LZ_THREADS / 32; ++w) t += s_p[w][threadIdx.x];
        wpart[((size_t)bi * nsp + blockIdx.y) * ldw + i0 + threadIdx.x] = t;
    }
}

// Sums in twice the working precision (Dekker, "A floating-point technique for extending the available precision",
// Numer. Math. 18, 1971; Ogita, Rump and Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26, 2005).
struct LzSum {
    double hi, lo;
};
__device__ __forceinline__ LzSum lz_plus(LzSum a, double hi, double lo)
{
    const double s = __dadd_rn(a.hi, hi), t = __dsub_rn(s, a.hi);
    const double e = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, t)), __dsub_rn(hi, t));
    return {s, a.lo + lo + e};
}
__device__ __forceinline__ LzSum lz_plus_product(LzSum a, double x, double y)
{
    const double q = __dmul_rn(x, y);
    return lz_plus(a, q, fma(x, y, -q));
}
__device__ __forceinline__ LzSum lz_warp_sum(LzSum a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        a = lz_plus(a, __shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o));
    return a;
}

// Two classical Gram-Schmidt passes of w = A v_j against v_0 .. v_j (the first pass's coefficient of v_j is
// alpha_j; a single pass is not stable: in FP32 the vectors lose their orthogonality within 40 steps), beta_j = |w|
// and v_{j+1} = w / beta_j.  CTA r of the cluster holds elements r * sl .. of the vectors; sums
// over the cluster are added in rank order.  Bound by the exchanges (a cluster barrier and a remote read, about 2 us
// together): one a pass, one for the norm.
//
// v_0 of the FP64 run holds nearly all of the eigenvector, and alpha_0 = v_0'A v_0 nearly all of the eigenvalue: the
// rounding of that one sum, and of |v_0|^2 which is 1 only to rounding, would be the eigenvalue's.  So alpha_0 is the
// quotient of both, summed in twice the precision.
template <typename T>
__global__ void __cluster_dims__(LZ_CTAS, 1, 1) __launch_bounds__(LZ_THREADS)
    k_lz_orth(const int32_t *blk_ls, const int32_t *batch_blocks, size_t vstride, T *V, const T *wpart, int nsp, int ldw,
              T *alpha, T *beta, int mmax, int j, const uint8_t *done)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int NW = LZ_THREADS / 32, PASSES = 2;
    extern __shared__ __align__(16) unsigned char lz_smem[];
    __shared__ T s_nrm[NW];
    __shared__ LzSum s_q[2];                        // this CTA's parts of v_0'w and v_0'v_0
    const bool quotient = sizeof(T) == 8 && j == 0;
    const int bi = blockIdx.x / LZ_CTAS, rank = (int)cl.block_rank();
    const int b = batch_blocks[bi];
    const int N = blk_ls[b + 1] - blk_ls[b], sl = (N + LZ_CTAS - 1) / LZ_CTAS;
    const int lo = min(N, rank * sl), cnt = min(N, lo + sl) - lo;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    T *s_h = reinterpret_cast<T *>(lz_smem);        // [PASSES][mmax] this CTA's partial dot products
    T *s_ht = s_h + 2 * mmax;                       // [mmax] the cluster's
    T *w = s_ht + mmax;                             // [sl]
    tc::pdl_trigger();
    tc::pdl_wait();
    if (done && done[bi]) return;                   // the same for the whole cluster
    T *Vb = V + vstride * bi + lo;                  // v_t's slice at Vb + t * N
    for (int i = tid; i < cnt; i += LZ_THREADS) {
        T x = (T)0.0;
        for (int q = 0; q < nsp; ++q) x += wpart[((size_t)bi * nsp + q) * ldw + lo + i];
        w[i] = x;
    }
    T nrm = (T)0.0, a = (T)0.0;
#pragma unroll
    for (int pass = 0; pass < PASSES; ++pass) {
        __syncthreads();
        T *h = s_h + pass * mmax;
        for (int t = 4 * warp; t <= j; t += 4 * NW) {   // four dot products at a time: their loads overlap
            T s[4] = {(T)0.0, (T)0.0, (T)0.0, (T)0.0};
            const T *vt[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) vt[q] = Vb + (size_t)min(t + q, j) * N;
#pragma unroll 4
            for (int i = lane; i < cnt; i += 32) {
                const T x = w[i];
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] += vt[q][i] * x;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) s[q] = lz_warp_sum(s[q]);
            if (lane < 4 && t + lane <= j) h[t + lane] = lane == 0 ? s[0] : (lane == 1 ? s[1] : (lane == 2 ? s[2] : s[3]));
        }
        if (quotient && pass == 0 && warp < 2) {
            LzSum s = {0.0, 0.0};
            for (int i = lane; i < cnt; i += 32) s = lz_plus_product(s, (double)Vb[i], warp == 0 ? (double)w[i] : (double)Vb[i]);
            s = lz_warp_sum(s);
            if (lane == 0) s_q[warp] = s;
        }
        cl.sync();
        for (int t = tid; t <= j; t += LZ_THREADS) {
            T s = (T)0.0;
#pragma unroll
            for (int q = 0; q < LZ_CTAS; ++q) s += cl.map_shared_rank(h, q)[t];
            if (quotient && pass == 0) {
                LzSum x[2] = {{0.0, 0.0}, {0.0, 0.0}};
                for (int q = 0; q < LZ_CTAS; ++q)
                    for (int k = 0; k < 2; ++k) {
                        const LzSum r = cl.map_shared_rank(s_q, q)[k];
                        x[k] = lz_plus(x[k], r.hi, r.lo);
                    }
                // (hi + lo) / (hi' + lo') with hi' near 1
                const double n = x[1].hi + x[1].lo, a0 = x[0].hi / n;
                s = (T)(a0 + ((fma(-a0, n, x[0].hi) + x[0].lo) - a0 * (x[1].hi - n + x[1].lo)) / n);
            }
            s_ht[t] = s;
        }
        __syncthreads();
        if (pass == 0) a = s_ht[j];
        nrm = (T)0.0;
        for (int i = tid; i < cnt; i += LZ_THREADS) {
            T x = w[i];
#pragma unroll 16
            for (int t = 0; t <= j; ++t) x -= s_ht[t] * Vb[(size_t)t * N + i];
            w[i] = x;
            nrm += x * x;
        }
    }
    nrm = lz_warp_sum(nrm);
    if (lane == 0) s_nrm[warp] = nrm;
    cl.sync();
    // the cluster's NW * LZ_CTAS = 64 partial norms, two a lane
    nrm = cl.map_shared_rank(s_nrm, lane / NW)[lane % NW] + cl.map_shared_rank(s_nrm, lane / NW + LZ_CTAS / 2)[lane % NW];
    static_assert(NW * LZ_CTAS == 64, "two partial norms a lane");
    const T bt = t_sqrt(lz_warp_sum(nrm));
    cl.barrier_arrive();   // this CTA reads no other's shared memory any more
    if (rank == 0 && tid == 0) {
        alpha[(size_t)bi * mmax + j] = a;
        beta[(size_t)bi * mmax + j] = bt;
    }
    if (j + 1 < mmax && j + 1 < N) {
        T *vn = Vb + (size_t)(j + 1) * N;
        const T inv = bt > (T)0.0 ? (T)1.0 / bt : (T)0.0;
        for (int i = tid; i < cnt; i += LZ_THREADS) vn[i] = w[i] * inv;
    }
    cl.barrier_wait();     // no CTA leaves while another still reads its shared memory
}

// The start vector of the FP64 run: the Ritz vector of the FP32 run's m steps.  Its tridiagonal matrix T has the top
// eigenvalue theta (32-way multisection with Sturm counts); (theta + shift) I - T is positive definite, so inverse
// iteration needs no pivoting.  Where that gives no usable vector, the FP32 run's own start is kept.
__global__ void __launch_bounds__(1024)
    k_lz_ritz(const int32_t *blk_ls, const int32_t *batch_blocks, size_t vstride32, const float *V32,
              const float *alpha32, const float *beta32, int steps, size_t vstride, double *V)
{
    __shared__ double sh[33];
    __shared__ float s_a[LZ_PRE], s_b[LZ_PRE], s_s[LZ_PRE], s_l[LZ_PRE], s_d[LZ_PRE];
    const int bi = blockIdx.x, b = batch_blocks[bi];
    const int N = blk_ls[b + 1] - blk_ls[b], m = min(steps, N);
    const int tid = threadIdx.x, lane = tid & 31;
    const float *V0 = V32 + vstride32 * bi;
    if (tid < m) {
        s_a[tid] = alpha32[(size_t)bi * LZ_PRE + tid];
        s_b[tid] = tid + 1 < m ? beta32[(size_t)bi * LZ_PRE + tid] : 0.0f;
        s_s[tid] = 1.0f;
    }
    __syncthreads();
    if (tid < 32) {
        float lo = 3.4e38f, hi = -3.4e38f;
        for (int i = lane; i < m; i += 32) {
            const float r = (i > 0 ? s_b[i - 1] : 0.0f) + s_b[i];
            lo = fminf(lo, s_a[i]);
            hi = fmaxf(hi, s_a[i] + r);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        for (int round = 0; round < 5; ++round) {   // the interval shrinks 33-fold a round
            const float step = (hi - lo) * (1.0f / 33.0f), x = lo + step * (float)(lane + 1);
            bool above = true;                      // x is above every eigenvalue: all pivots of T - x I negative
            float q = s_a[0] - x;
            for (int i = 1; i < m && above; ++i) {
                above = q < 0.0f;
                q = s_a[i] - x - __fdividef(s_b[i - 1] * s_b[i - 1], q);
            }
            above = above && q < 0.0f;
            const unsigned ok = __ballot_sync(0xffffffffu, above);
            const int f = ok ? __ffs(ok) - 1 : 32;
            hi = f < 32 ? lo + step * (float)(f + 1) : hi;
            lo = lo + step * (float)f;
        }
        if (lane == 0) {
            const float theta = hi + 2e-6f * fabsf(hi), tiny = fmaxf(1e-7f * fabsf(hi), 1e-30f);
            for (int i = 0; i < m; ++i) {
                float d = theta - s_a[i];
                if (i > 0) d -= s_b[i - 1] * s_l[i - 1];
                d = fmaxf(d, tiny);
                s_d[i] = 1.0f / d;
                s_l[i] = s_b[i] * s_d[i];
            }
            for (int it = 0; it < 3; ++it) {
                for (int i = 1; i < m; ++i) s_s[i] += s_l[i - 1] * s_s[i - 1];
                float big = 0.0f;
                for (int i = m - 1; i >= 0; --i) {
                    s_s[i] = s_s[i] * s_d[i] + (i + 1 < m ? s_l[i] * s_s[i + 1] : 0.0f);
                    big = fmaxf(big, fabsf(s_s[i]));
                }
                const float inv = 1.0f / big;
                for (int i = 0; i < m; ++i) s_s[i] *= inv;
            }
        }
    }
    __syncthreads();
    double nn = 0.0;
    double *v = V + vstride * bi;
    for (int i = tid; i < N; i += 1024) {
        float x = 0.0f;
#pragma unroll 8
        for (int t = 0; t < m; ++t) x = fmaf(s_s[t], V0[(size_t)t * N + i], x);
        v[i] = (double)x;
        nn += (double)x * (double)x;
    }
    nn = lz_block_sum(nn, sh);
    if (!(nn > 1e-2 && nn < 1e30)) {
        nn = 0.0;
        for (int i = tid; i < N; i += 1024) {
            v[i] = (double)V0[i];
            nn += (double)V0[i] * (double)V0[i];
        }
        nn = lz_block_sum(nn, sh);
    }
    const double inv = 1.0 / sqrt(nn);   // (what rounding leaves of |v_0|^2 - 1 is no matter: alpha_0 is a quotient)
    for (int i = tid; i < N; i += 1024) v[i] *= inv;
}

}  // namespace soda

// chol_tc.cuh — U = chol(d I - A), upper (choleskyPD, soda.f90:8-47), for a batch of subsets, included by zbuild.cu.
//
// N^3 / 3 FP64 operations a subset are bound by GB300's FP64 pipe (10 subsets of 2000 SNPs: 21 ms at its full rate).
// All but the panels' own work is products of rows of U that are already known, so it runs on the tensor cores in
// exact integer arithmetic, by splitting FP64 numbers into 8-bit digits (Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication", Numer. Algorithms 59, 2012):
//
//   * column j of U is bounded by sqrt(M_jj), M = d I - A, because M_jj is the sum of its squares.  With 2^e_j above
//     that bound, U_tj = 2^(e_j + 1) sum_s d_s 256^-s, s = 1 .. 7: seven digits of -128 .. 128, exact in bf16, which
//     hold U to 2^-56 of the bound;
//   * the product of digits s and t belongs to level s + t.  Products are at most 2^14, so the FP32 sums of a level
//     (at most seven pairs) are exact over 128 rows of U.  Levels 2 .. 9 (34 pairs) are kept, in one tensor-memory
//     accumulator each; what levels 10 and up hold is below 2^-61 of the bounds' product a row, of either sign: about
//     sqrt(N) 2^-64 over N rows;
//   * every 128 rows the levels are added into one 64-bit integer per element, in units of 2^-62 of the bounds'
//     product (Cauchy-Schwarz keeps the whole sum within the bounds' product).
// So C = M - sum_t U_ti U_tj is rounded once, where a chain of N FP64 multiply-adds rounds at every term.
//
// Left-looking over panels of CH_P rows: k_ch_update forms the panel's rows of M minus the products of all earlier
// rows; k_ch_diag factors its diagonal block; k_ch_trsm solves for the rest and leaves the digits of the new rows.
// The factorisation fails (status) on a pivot that is not positive, or, the same thing noticed earlier, when a
// column's squares exceed M_jj.
//
// Measured, 10 subsets of 2000 SNPs: updates 3.2 ms, diagonal blocks 2.9, substitution 2.6 (the last two bound by the
// FP64 pipe, which takes any warp's instruction 64 cycles), against 31.9 ms of FP64 kernels (rank-32 updates 25.6,
// panels 6.3).  U'U + A - d I, with A exact, is 1.5e-17 d at N = 300 and n = 700, 1.4e-17 d at 600 and 1,500, 1.3e-17 d
// at 1000 and 2,000 (rms; 1.9e-17, 1.8e-17 and 1.9e-17 with the FP64 kernels and their Gram).
#pragma once
#include <cuda.h>
#include "tc.cuh"

namespace soda {

constexpr int CH_P = 64;                     // rows of a panel (columns of an update tile)
constexpr int CH_M = 128;                    // columns of M an update CTA takes (MMA rows)
constexpr int CH_K = 32;                     // rows of U per stage (64-byte swizzled operands)
constexpr int CH_DIG = 7;                    // digits
constexpr int CH_LEV = 8;                    // levels 2 .. 9
constexpr int CH_GROUP = 4;                  // stages between two drains of the accumulators: 128 rows
constexpr int CH_NS = 2;                     // stages in flight
constexpr int CH_A = CH_M * CH_K * 2, CH_B = CH_P * CH_K * 2;   // bytes of a digit's tiles
constexpr int CH_STAGE = CH_DIG * (CH_A + CH_B);
constexpr size_t CH_SMEM = 1024 + (size_t)CH_NS * CH_STAGE;
constexpr int CH_THREADS = 320;              // 8 epilogue warps, TMA, MMA
static_assert(7 * CH_GROUP * CH_K * (1 << 14) <= (1 << 24), "FP32 sums of a level are exact");
static_assert(CH_LEV * CH_P == 512, "tensor memory");

// Per column: sc = 2^e_j > sqrt(M_jj); M_jj <= 0 fails.  nrm (the squares of the column's rows so far) starts at 0.
__global__ void __launch_bounds__(256) k_ch_init(const double *W, const int64_t *wofs, const int32_t *blk_ls,
                                                 const int32_t *batch_blocks, const double *xxd, double *sc, double *nrm,
                                                 int np, int32_t *status)
{
    const int b = batch_blocks[blockIdx.x];
    const int N = blk_ls[b + 1] - blk_ls[b];
    const double *A = W + wofs[b], d = xxd[b];
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
        double s = 1.0;
        if (j < N) {
            const double m = d - A[(size_t)j + (size_t)j * N];
            if (!(m > 0.0)) status[b] = j + 1;
            else s = __hiloint2double((((__double2hiint(sqrt(m)) >> 20) & 0x7FF) + 1) << 20, 0);
        }
        sc[(size_t)blockIdx.x * np + j] = s;
        nrm[(size_t)blockIdx.x * np + j] = 0.0;
    }
}

// Rows i0 .. i0 + CH_P - 1 of M - U'U (the rows of U above i0), columns j0 = i0 + CH_M blockIdx.x .. of the upper
// triangle, in place of A.  Accumulator rows are the columns j, its columns the panel's rows i.
__global__ void __launch_bounds__(CH_THREADS, 1)
    k_ch_update(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, double *W,
                const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks, const double *xxd,
                const double *sc, int np, int32_t *status, int i0, int *err)
{
    extern __shared__ __align__(1024) unsigned char smem_dyn[];
    __shared__ uint64_t s_full[CH_NS], s_free[CH_NS], s_done, s_read;
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;
    __shared__ double s_sc[CH_P];
    tc::pdl_trigger();
    tc::pdl_wait();
    const int b = batch_blocks[blockIdx.y];
    const int N = blk_ls[b + 1] - blk_ls[b], j0 = i0 + CH_M * blockIdx.x;
    if (__syncthreads_or(j0 >= N || status[b] != 0)) return;   // the same answer in every thread
    unsigned char *raw0 = smem_dyn + ((1024u - (tc::smem_u32(smem_dyn) & 1023u)) & 1023u);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ns = i0 / CH_K, ngr = (ns + CH_GROUP - 1) / CH_GROUP;
    if (tid == 0) {
        for (int i = 0; i < CH_NS; ++i) {
            tc::mbar_init(&s_full[i], 1);
            tc::mbar_init(&s_free[i], 1);
        }
        tc::mbar_init(&s_done, 1);
        tc::mbar_init(&s_read, 8);   // the epilogue warps
        tc::mbar_fence_init();
        s_err = 0;
    }
    if (tid < CH_P) s_sc[tid] = sc[(size_t)blockIdx.y * np + min(i0 + tid, np - 1)];
    if (warp == 9) tc::tmem_alloc(&s_tmem, 512);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = s_tmem;
    if (warp == 8) {
        if (lane == 0) {
            tc::tma_prefetch_desc(&tm_a);
            tc::tma_prefetch_desc(&tm_b);
            const int row0 = (int)blockIdx.y * CH_DIG * np;
            int issued = 0;
            for (int s = 0; s < ns; ++s) {
                const int sl = s % CH_NS;
                if (s >= CH_NS && !tc::mbar_wait(&s_free[sl], ((s / CH_NS) - 1) & 1, tc::BUILD_WAIT_NS)) {
                    s_err = 1;
                    break;
                }
                unsigned char *dst = raw0 + (size_t)sl * CH_STAGE;
                tc::mbar_expect_tx(&s_full[sl], CH_STAGE);
#pragma unroll 1
                for (int q = 0; q < CH_DIG; ++q) {
                    tc::tma_load_2d(dst + q * CH_A, &tm_a, s * CH_K, row0 + q * np + j0, &s_full[sl]);
                    tc::tma_load_2d(dst + CH_DIG * CH_A + q * CH_B, &tm_b, s * CH_K, row0 + q * np + i0, &s_full[sl]);
                }
                issued = s + 1;
            }
            // no copy may still be in flight into this CTA's shared memory when it exits
            for (int s = max(0, issued - CH_NS); s < issued; ++s)
                if (!tc::mbar_wait(&s_full[s % CH_NS], (s / CH_NS) & 1, tc::BUILD_WAIT_NS)) s_err = 1;
        }
    } else if (warp == 9) {
        const bool leader = tc::elect_one();
        const uint32_t idesc = tc::idesc_bf16(CH_M, CH_P);
        bool ok = true;
        for (int s = 0; s < ns && ok; ++s) {
            const int sl = s % CH_NS;
            const bool first = s % CH_GROUP == 0;
            if (first && s > 0) ok = tc::mbar_wait(&s_read, (s / CH_GROUP - 1) & 1, tc::BUILD_WAIT_NS);   // the last group is drained
            ok = ok && tc::mbar_wait(&s_full[sl], (s / CH_NS) & 1, tc::BUILD_WAIT_NS);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                s_err = 1;
                break;
            }
            tc::fence_after_sync();
            if (leader) {
                const uint32_t base = tc::smem_u32(raw0 + (size_t)sl * CH_STAGE);
                const uint64_t a0 = tc::desc_sw64(base), b0 = tc::desc_sw64(base + CH_DIG * CH_A);
#pragma unroll
                for (int kk = 0; kk < CH_K / 16; ++kk)
#pragma unroll
                    for (int lev = 2; lev < 2 + CH_LEV; ++lev)
#pragma unroll
                        for (int p = 1; p <= CH_DIG; ++p) {
                            const int q = lev - p, p0 = lev - CH_DIG > 1 ? lev - CH_DIG : 1;   // p0: the level's first pair
                            if (q < 1 || q > CH_DIG) continue;
                            tc::mma_bf16(tm + (lev - 2) * CH_P, a0 + (((p - 1) * CH_A + kk * 32) >> 4),
                                         b0 + (((q - 1) * CH_B + kk * 32) >> 4), idesc,
                                         first && kk == 0 && p == p0 ? 0u : 1u);
                        }
                tc::mma_commit(&s_free[sl]);
                if (s % CH_GROUP == CH_GROUP - 1 || s == ns - 1) tc::mma_commit(&s_done);
            }
            __syncwarp();
        }
    } else {
        // lane quadrant of the warp, and its half of the panel's rows
        const int qd = warp & 3, h = warp >> 2;
        long long acc[CH_P / 2];
#pragma unroll
        for (int c = 0; c < CH_P / 2; ++c) acc[c] = 0;
        const uint32_t ta = tm + ((uint32_t)(32 * qd) << 16) + h * (CH_P / 2);
        for (int g = 0; g < ngr; ++g) {
            bool ok = tc::mbar_wait(&s_done, g & 1, tc::BUILD_WAIT_NS);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                s_err = 1;
                break;
            }
            tc::fence_after_sync();
#pragma unroll
            for (int c0 = 0; c0 < CH_P / 2; c0 += 8) {
                float v[CH_LEV][8];
#pragma unroll
                for (int l = 0; l < CH_LEV; ++l) tc::tmem_ld8(ta + l * CH_P + c0, v[l]);
                tc::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    long long t = 0;
#pragma unroll
                    for (int l = 0; l < CH_LEV - 1; ++l) t += (long long)__float2int_rn(v[l][e]) << (8 * (CH_LEV - 2 - l));
                    t += (__float2int_rn(v[CH_LEV - 1][e]) + 128) >> 8;
                    acc[c0 + e] += t;
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&s_read);
        }
        const int j = j0 + 32 * qd + lane;
        if (j < N) {
            double *col = W + wofs[b] + (size_t)j * N + i0 + h * (CH_P / 2);
            // M in the sum's units, an exact scaling by a power of two; the difference is an integer, rounded once
            const int ej = __double2hiint(sc[(size_t)blockIdx.y * np + j]) >> 20;
            const double d = xxd[b];
#pragma unroll
            for (int c = 0; c < CH_P / 2; ++c) {
                const int i = i0 + h * (CH_P / 2) + c;
                if (i > j) continue;
                const double m = i == j ? d - col[c] : -col[c];
                const int e = (__double2hiint(s_sc[h * (CH_P / 2) + c]) >> 20) + ej - 1023 - 62;   // of the unit
                const double up = __hiloint2double((2046 - e) << 20, 0), unit = __hiloint2double(e << 20, 0);
                col[c] = (double)(__double2ll_rn(m * up) - acc[c]) * unit;
            }
        }
    }
    __syncthreads();
    if (tid == 0 && s_err) {
        status[b] = -1;
        atomicExch(err, 1);
    }
    if (warp == 9) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tm, 512);
    }
}

// 1 / sqrt(p) and sqrt(p) from an FP32 seed, one third-order step of Householder's method (The Numerical Treatment of a
// Single Nonlinear Equation, 1970: the binomial series of (1 - e)^-1/2 to e^2) and, for the root, a correction by its
// exact remainder (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990).  FP64's own square root and division lie on the critical path of every pivot, where a dependent
// instruction takes 64 cycles.  The root is off by at most a unit in the last place, 1 / sqrt(p) by at most two.
__device__ __forceinline__ void ch_rsqrt(double p, double &inv, double &root)
{
    if (!(p > 1e-30 && p < 1e30)) {
        root = sqrt(p);
        inv = 1.0 / root;
        return;
    }
    const double y = (double)rsqrtf((float)p);
    const double e = fma(-(p * y), y, 1.0);                   // |e| < 2^-21
    inv = fma(y * e, fma(e, 0.375, 0.5), y);                  // y (1 + e/2 + 3 e^2 / 8), error e^3
    const double r = p * inv;
    root = fma(0.5 * inv, fma(-r, r, p), r);
}
// c / root with inv = 1 / root, corrected by its exact remainder (Markstein): at most a unit in the last place off.
__device__ __forceinline__ double ch_div(double c, double root, double inv)
{
    const double x = c * inv;
    return fma(fma(-x, root, c), inv, x);
}

// The panel's diagonal block, in steps of 8: a warp factors 8 x 8 with a column a lane, a thread a column solves the
// rest of its rows, and the warps take the rank-8 update's rows.  Bound by the chain of FP64 instructions: about 17 a
// pivot in the factoring warp, 52 a step in the solving ones; 92 us a panel (121 us in steps of 16).  A step's eight
// products are summed by themselves: taken out of the block's entries one at a time, each would be rounded at the size
// of M, and the pivots were off by as much as 64 such roundings.  inv: the pivots'
// reciprocals, for k_ch_trsm.
constexpr int CH_D = 8;

__global__ void __launch_bounds__(256) k_ch_diag(double *W, const int64_t *wofs, const int32_t *blk_ls,
                                                 const int32_t *batch_blocks, int32_t *status, int i0, double *piv)
{
    __shared__ double T[CH_P][CH_P + 1];
    __shared__ double s_inv[CH_P];
    __shared__ int s_fail;
    tc::pdl_trigger();
    tc::pdl_wait();
    const int b = batch_blocks[blockIdx.x];
    const int N = blk_ls[b + 1] - blk_ls[b];
    if (i0 >= N || status[b] != 0) return;
    const int nb = min(CH_P, N - i0);
    double *A = W + wofs[b] + (size_t)i0 * N + i0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int t = tid; t < CH_P * CH_P; t += 256) {
        const int r = t % CH_P, c = t / CH_P;
        // rows and columns past the subset: the identity, which changes nothing
        T[r][c] = r < nb && c < nb ? (r <= c ? A[(size_t)r + (size_t)c * N] : 0.0) : (r == c ? 1.0 : 0.0);
    }
    if (tid == 0) s_fail = 0;
    __syncthreads();
    for (int kb = 0; kb < CH_P; kb += CH_D) {
        if (warp == 0) {
            const int l = lane & (CH_D - 1), c = kb + l;
            double x[CH_D];
#pragma unroll
            for (int r = 0; r < CH_D; ++r) x[r] = T[kb + r][c];
#pragma unroll
            for (int r = 0; r < CH_D; ++r) {
                const double p = __shfl_sync(0xffffffffu, x[r], r);
                if (!(p > 0.0) && lane == 0 && !s_fail) s_fail = i0 + kb + r + 1;
                double inv, root;
                ch_rsqrt(p, inv, root);
                if (lane == r) s_inv[kb + r] = inv;
                x[r] = l == r ? root : ch_div(x[r], root, inv);
#pragma unroll
                for (int q = r + 1; q < CH_D; ++q) x[q] = fma(-__shfl_sync(0xffffffffu, x[r], q), x[r], x[q]);
            }
            if (lane < CH_D)
#pragma unroll
                for (int r = 0; r < CH_D; ++r)
                    if (r <= lane) T[kb + r][c] = x[r];
        }
        __syncthreads();
        if (s_fail) break;
        const int c = kb + CH_D + tid;
        if (c < CH_P) {
            double x[CH_D];
#pragma unroll
            for (int r = 0; r < CH_D; ++r) x[r] = T[kb + r][c];
#pragma unroll
            for (int r = 0; r < CH_D; ++r) {
                x[r] = ch_div(x[r], T[kb + r][kb + r], s_inv[kb + r]);
#pragma unroll
                for (int q = r + 1; q < CH_D; ++q) x[q] = fma(-T[kb + r][kb + q], x[r], x[q]);
            }
#pragma unroll
            for (int r = 0; r < CH_D; ++r) T[kb + r][c] = x[r];
        }
        __syncthreads();
        for (int r = kb + CH_D + warp; r < CH_P; r += 8) {
            double m[CH_D];
#pragma unroll
            for (int q = 0; q < CH_D; ++q) m[q] = -T[kb + q][r];
            for (int cc = (r & ~31) + lane; cc < CH_P; cc += 32) {
                double s = m[0] * T[kb][cc];
#pragma unroll
                for (int q = 1; q < CH_D; ++q) s = fma(m[q], T[kb + q][cc], s);
                if (cc >= r) T[r][cc] += s;
            }
        }
        __syncthreads();
    }
    if (s_fail) {
        if (tid == 0) status[b] = s_fail;
        return;
    }
    for (int t = tid; t < CH_P * CH_P; t += 256) {
        const int r = t % CH_P, c = t / CH_P;
        if (r <= c && c < nb) A[(size_t)r + (size_t)c * N] = T[r][c];
    }
    if (tid < CH_P) piv[(size_t)blockIdx.x * CH_P + tid] = s_inv[tid];
}

// The panel's rows for 32 columns right of it: substitution in blocks of 16 rows, the columns' squares, and the digits
// of the new rows, [digit][column][row], eight rows a 16-byte store.  A block is solved by one warp, a column a lane
// (the warp changes with the block and the CTA, so that all of an SM's FP64 pipes are used), and four warps take its
// products out of the rows below: 1120 instructions in a chain, 64 cycles each, in place of 2400 for a column a thread: 85 us a
// panel of 10 subsets of 2000 SNPs, 161 us before.
constexpr int CH_S = 16;
constexpr size_t CH_TRSM_SMEM = sizeof(double) * (CH_P * CH_P + CH_P * 32 + CH_P);

__global__ void __launch_bounds__(128)
    k_ch_trsm(double *W, const int64_t *wofs, const int32_t *blk_ls, const int32_t *batch_blocks, const double *xxd,
              const double *sc, double *nrm, int np, int32_t *status, int i0, const double *piv, uint16_t *dig, int ldt)
{
    extern __shared__ __align__(16) double ch_smem[];
    __shared__ double s_ss[CH_P / CH_S][32];
    double (*T)[CH_P] = reinterpret_cast<double (*)[CH_P]>(ch_smem);                   // row r of the block's factor
    double (*C)[32] = reinterpret_cast<double (*)[32]>(ch_smem + CH_P * CH_P);         // the columns
    double *s_inv = ch_smem + CH_P * CH_P + CH_P * 32;
    tc::pdl_trigger();
    tc::pdl_wait();
    const int b = batch_blocks[blockIdx.y];
    const int N = blk_ls[b + 1] - blk_ls[b], c0 = i0 + CH_P + 32 * blockIdx.x;
    if (__syncthreads_or(c0 >= N || status[b] != 0)) return;   // (columns of other CTAs may fail meanwhile)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, j = c0 + lane;
    double *A = W + wofs[b];
    for (int t = tid; t < CH_P * CH_P; t += 128) {
        const int r = t % CH_P, c = t / CH_P;
        if (r <= c) T[r][c] = A[(size_t)(i0 + r) + (size_t)(i0 + c) * N];
    }
    for (int t = tid; t < CH_P * 32; t += 128) {
        const int r = t % CH_P, c = t / CH_P;
        C[r][c] = c0 + c < N ? A[(size_t)(i0 + r) + (size_t)(c0 + c) * N] : 0.0;
    }
    if (tid < CH_P) s_inv[tid] = piv[(size_t)blockIdx.y * CH_P + tid];
    __syncthreads();
    for (int kb = 0; kb < CH_P; kb += CH_S) {
        if (warp == ((kb / CH_S + blockIdx.x) & 3)) {
            double x[CH_S], ss = 0.0;
#pragma unroll
            for (int r = 0; r < CH_S; ++r) x[r] = C[kb + r][lane];
#pragma unroll
            for (int r = 0; r < CH_S; ++r) {
                x[r] = ch_div(x[r], T[kb + r][kb + r], s_inv[kb + r]);
                ss = fma(x[r], x[r], ss);
#pragma unroll
                for (int q = r + 1; q < CH_S; ++q) x[q] = fma(-T[kb + r][kb + q], x[r], x[q]);
            }
#pragma unroll
            for (int r = 0; r < CH_S; ++r) C[kb + r][lane] = x[r];
            s_ss[kb / CH_S][lane] = ss;
        }
        __syncthreads();
        if (kb + CH_S < CH_P) {
            double x[CH_S];
#pragma unroll
            for (int q = 0; q < CH_S; ++q) x[q] = -C[kb + q][lane];
            for (int r = kb + CH_S + warp; r < CH_P; r += 4) {
                double s = C[r][lane];
#pragma unroll
                for (int q = 0; q < CH_S; ++q) s = fma(T[kb + q][r], x[q], s);
                C[r][lane] = s;
            }
            __syncthreads();
        }
    }
    for (int t = tid; t < CH_P * 32; t += 128) {
        const int r = t % CH_P, c = t / CH_P;
        if (c0 + c < N) A[(size_t)(i0 + r) + (size_t)(c0 + c) * N] = C[r][c];
    }
    if (j >= N) return;
    const size_t o = (size_t)blockIdx.y * np + j;
    if (warp == 0) {
        // the squares of a column never exceed M_jj (its diagonal entry is still A's) when M is positive definite
        const double ss = nrm[o] + ((s_ss[0][lane] + s_ss[1][lane]) + (s_ss[2][lane] + s_ss[3][lane]));
        nrm[o] = ss;
        if (!(ss <= (xxd[b] - A[(size_t)j + (size_t)j * N]) * (1.0 + 1e-9))) status[b] = i0 + CH_P + 1;
    }
    const double q55 = 36028797018963968.0 / sc[o];   // 2^55 / 2^e_j: one unit is 2^-55 of the bound
    uint16_t *dst = dig + ((size_t)blockIdx.y * CH_DIG * np + j) * ldt + i0;
    for (int r0 = CH_S * warp; r0 < CH_S * (warp + 1); r0 += 8) {
        uint32_t w[CH_DIG][4];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            long long v = __double2ll_rn(C[r0 + e][lane] * q55);
#pragma unroll
            for (int s = CH_DIG - 1; s >= 0; --s) {
                const int dgt = s > 0 ? (int)(signed char)(v & 0xFF) : (int)v;
                v = (v - dgt) >> 8;
                // an integer of at most 256 in magnitude is exact in bf16: the top half of its FP32 bits
                const uint32_t bits = __float_as_uint((float)dgt) >> 16;
                if (e & 1) w[s][e >> 1] |= bits << 16;
                else w[s][e >> 1] = bits;
            }
        }
#pragma unroll
        for (int s = 0; s < CH_DIG; ++s)
            *reinterpret_cast<uint4 *>(dst + (size_t)s * np * ldt + r0) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
}

}  // namespace soda

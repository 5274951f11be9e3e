// sweep.cu — per-iteration kernels of the SODA Gibbs sampler.
//
// One iteration (models.f90:129-574) is, per chain:
//   mu draw                              k_mu_partial + k_mu_apply   (models.f90:130-132)
//   for each subset b (sequential):
//     rhs_j = x_j'r + u_j'ra (+d g_j) and the per-SNP draw
//                                        k_rhs (rhs_kernel.cuh)      (models.f90:146-162, 211-256, 350-413)
//     r += X_b delta, ra += U_b delta    k_update                    (models.f90:164-174, 258-272, 415-430)
//   single-site updates of skipped SNPs  k_skipped                   (models.f90:178-193, 276-320, 433-495)
//   class counts, sum g^2, sum r^2       k_stats
//   sigma2_g, sigma2_e, pi draws, trace  k_hyper                     (models.f90:194, 321-325, 496-522, 549-569)
//   ra redraw, posterior accumulators    k_post                      (models.f90:523-548)
//   residual recalibration               k_recal_partial/_apply      (models.f90:571-573)
// All chains of the context advance together inside each launch.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "rng.cuh"
#include "state.cuh"
#include "sweep.cuh"
#include "tc.cuh"
#include <algorithm>
#include <vector>

namespace soda {

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_sumf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block sum; every thread gets the total.  blockDim.x % 32 == 0.
__device__ double block_sum(double v, double *sh /* >= 33 doubles */)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        double t = lane < nw ? sh[lane] : 0.0;
        t = warp_sum(t);
        if (lane == 0) sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

__device__ __forceinline__ int cur_rep(const Dev &D) { return *((volatile int32_t *)&D.ctl->rep); }

// Residual stores: the FP64 master and, for the FP32-core rhs, its FP32 copy,
// or, when the tensor-core rhs runs, the bf16 hi/mid/lo split of the FP32
// value that it loads by TMA.
__device__ __forceinline__ void split_store(uint16_t *sp, size_t o, size_t part, float f)
{
    uint32_t h, m, l;
    tc::split3(f, h, m, l);
    sp[o] = (uint16_t)h;
    sp[o + part] = (uint16_t)m;
    sp[o + 2 * part] = (uint16_t)l;
}
__device__ __forceinline__ void store_r(const Dev &D, int c, int i, double v)
{
    const size_t o = (size_t)c * D.ldr + i;
    D.r[o] = v;
    if (!D.tc) D.r32[o] = (float)v;   // read only by the FP32-core dot products
    if (D.rsp) split_store(D.rsp, o, (size_t)D.chains * D.ldr, (float)v);
}
__device__ __forceinline__ void store_ra(const Dev &D, int c, int i, double v)
{
    const size_t o = (size_t)c * D.ldra + i;
    D.ra[o] = v;
    D.ra32[o] = (float)v;
    if (D.rasp) split_store(D.rasp, o, (size_t)D.chains * D.ldra, (float)v);
}

__device__ __forceinline__ void flag_err(const Dev &D, int code)
{
    atomicExch(&D.ctl->err, code);
}

// A draw past the end of an injected-draw tape sets the same error code as a
// site needing more uniforms than its record holds.
constexpr int ERR_TAPE = CRNG_TAPE_OVERRUN;

// The draw stream of one site: Philox keyed by (seed, chain, rep, slot,
// purpose), or, with an injected-draw tape, the site's record (chain 0; site
// numbering of sodagpu_set_tape).
__device__ __forceinline__ void crng_site(CRng &R, const Dev &D, int c, int rep, int slot, int purpose)
{
    crng_init(R, D.seed, c, rep, slot, purpose);
    if (!D.tape) return;
    int site;
    switch (purpose) {
    case P_MU: site = 0; break;
    case P_VARA: site = 1; break;
    case P_VARE: site = 2; break;
    case P_PI: site = 3 + slot; break;
    case P_RA: site = 3 + D.ngroup + slot; break;
    default: site = D.tape_snp0 + slot; break;   // P_SNP, P_SKIP: by SNP id
    }
    R.tover = &D.ctl->err;
    if (rep >= 0 && rep < D.tape_reps && site < D.tape_sites) {
        R.tape = D.tape + ((size_t)rep * D.tape_sites + site) * SODAGPU_TAPE_W;
    } else {
        flag_err(D, ERR_TAPE);
    }
}

// ---------------------------------------------------------------------------
// Per-SNP conditional draw inside a subset (models.f90:146-161 BayesA, 211-255
// BayesB, 350-412 C/Cpi/R/Rc), in FP64, or in FP32 arithmetic for the FP32/FP8
// sweeps (GB300 executes FP64 at a small fraction of its FP32 rate); the state
// stays FP64.
//
// A draw is a chain of dependent transcendental operations on the critical path
// of every subset, and most of it does not depend on the right-hand side: what
// a subset's draws share (DrawSub, one per chain) and what is the SNP's own
// (DrawSnp: its uniforms, the normal and gamma variates, the locus variance's
// terms) is computed before the rhs kernel has finished.
// ---------------------------------------------------------------------------
constexpr int DRAW_PRE = 4;   // mixture classes with prefetched constants

template <typename T>
struct DrawSub {
    T vare, scale_va, zz_vare;
    // class k: log pi of group 1, log(gamma_k sigma2_g zz / sigma2_e + 1), the denominators of the score and
    // of the conditional mean, the conditional standard deviation
    T logp[DRAW_PRE], ld[DRAW_PRE], den[DRAW_PRE], v1[DRAW_PRE], sd[DRAW_PRE];
    // FP64: class k's score is b_k + c_k rhs^2 (b_k: DrawSnp), the quotient rhs^2 / (den sigma2_e) / 2 as one factor
    T c[DRAW_PRE];
};

// Class k of chain S in a subset with d = zz (k = 0 also fills what all classes share).
template <typename T>
__device__ __forceinline__ void draw_sub(const Dev &D, const ChainScal *S, int k, double zz, DrawSub<T> &q)
{
    const T vare = (T)S->vare, zt = (T)zz;
    const T zz_vare = (T)(zz / S->vare);
    if (k == 0) {
        q.vare = vare;
        q.scale_va = (T)S->scale_va;
        q.zz_vare = zz_vare;
    }
    const bool in = k < D.nmix;
    q.logp[k] = in ? (T)S->log_p[k * D.ngroup] : (T)0.0;
    const T gp = in ? (T)S->gp[k] : (T)0.0;
    q.ld[k] = t_log(gp * zz_vare + (T)1.0);
    q.den[k] = zt + (in ? (T)S->vare_gp[k] : (T)0.0);
    q.v1[k] = zt + vare / gp;
    q.sd[k] = t_sqrt(vare / q.v1[k]);
    if constexpr (sizeof(T) == 8) q.c[k] = k > 0 ? 0.5 / (q.den[k] * vare) : 0.0;
}

template <typename T>
struct DrawSnp {
    T u;                   // class uniform (BayesB and the mixtures)
    NormalPre<T> z;
    GammaPre<T> gam;       // BayesA/B
    T ld, den, sd, sdv;    // BayesA/B: from the locus variance
    T b[DRAW_PRE], c;      // FP64 scores: what does not depend on the right-hand side (c: BayesB's factor)
    bool plain;            // a standard deviation is 0: the draws follow the plain order at their use
    int err;
};

// Advances R past the uniforms that the SNP's draw takes (up to the class uniform when `plain`).
template <typename T>
__device__ __forceinline__ void draw_ahead(const Dev &D, const ChainScal *S, const DrawSub<T> &q, T zz, T vs, int sg,
                                           CRng &R, DrawSnp<T> &a)
{
    const int m = D.method;
    a.plain = false;
    a.err = 0;
    if (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) {
        a.den = zz + q.vare / vs;
        a.sd = t_sqrt(q.vare / a.den);
        a.plain = a.sd <= (T)0.0;
        if (m == SODAGPU_BAYES_B) {
            a.ld = t_log(vs * q.zz_vare + (T)1.0);
            a.sdv = t_sqrt(vs);
            a.plain = a.plain || a.sdv <= (T)0.0;
            a.u = crng_unit_t<T>(R);
            if constexpr (sizeof(T) == 8) {
                a.c = 0.5 / (a.den * q.vare);
                a.b[0] = S->log_p[0];
                a.b[1] = S->log_p[D.ngroup] - 0.5 * a.ld;
            }
        }
        if (a.plain) return;
        a.z = normal_pre<T>(R);
        a.gam = gamma_pre<T>((T)0.5 * ((T)D.df_va + (T)1.0), R, &a.err);
        return;
    }
    a.u = crng_unit_t<T>(R);
    a.z = normal_pre<T>(R);
    if constexpr (sizeof(T) == 8) {
#pragma unroll
        for (int k = 0; k < DRAW_PRE; ++k)
            if (k < D.nmix) a.b[k] = S->log_p[sg + k * D.ngroup] - (k > 0 ? 0.5 * q.ld[k] : 0.0);
    }
}

// x <= 700, false for a NaN: by the words, an FP64 comparison takes the narrow pipe 64 cycles a warp.
__device__ __forceinline__ bool at_most_700(double x)
{
    const int hi = __double2hiint(x), c = 0x4085E000;   // the upper word of 700
    return hi < c || (hi == c && __double2loint(x) == 0);
}

// The class (1-based) for the FP64 scores b_k + c_k r2 of up to DRAW_PRE classes: the first whose cumulative weight
// exceeds u times their sum, weights exp(s_k - s_0), or relative to the largest score where that could overflow; there a
// class more than 700 below the largest has none, as in the reference, which matters for u = 0.  (The
// probabilities of models.f90:366-379 one by one take up to twelve exponentials and four divisions, 16 and 10 FP64
// instructions of 64 cycles each, in every warp with a SNP outside the first class.)
__device__ __forceinline__ int draw_class64(double r2, const double (&b)[DRAW_PRE], const double (&c)[DRAW_PRE],
                                            int nm, double u)
{
    double w[DRAW_PRE], ref = b[0];
    bool big = false;
#pragma unroll
    for (int k = 0; k < DRAW_PRE; ++k) {
        w[k] = k == 0 ? b[0] : (k < nm ? fma(r2, c[k], b[k]) : -1e308);
        big = big || w[k] - b[0] > 700.0;
    }
    if (big) {
#pragma unroll
        for (int k = 1; k < DRAW_PRE; ++k) ref = fmax(ref, w[k]);
#pragma unroll
        for (int k = 0; k < DRAW_PRE; ++k)
            if (ref - w[k] > 700.0) w[k] = -1e308;
    }
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < DRAW_PRE; ++k)
        if (k < nm) {
            w[k] = k == 0 && !big ? 1.0 : exp(w[k] - ref);
            sum = sum + w[k];
        }
    const double us = u * sum;
    double cum = 0.0;
    int flag = 1;
    bool done = false;
#pragma unroll
    for (int k = 0; k < DRAW_PRE; ++k)
        if (k < nm && !done) {
            cum = cum + w[k];
            if (us < cum) {
                flag = k + 1;
                done = true;
            }
        }
    return flag;
}

// Returns delta = g_old - g_new; gold = g and cl = class of the SNP in this chain, sg = its group - 1.
template <typename T>
__device__ __forceinline__ double draw_snp(const Dev &D, const ChainScal *S, int c, int snploc, T rhs, T zz,
                                           const DrawSub<T> &q, DrawSnp<T> &a, CRng &R, double gold, int cl, int sg)
{
    const size_t o = (size_t)c * D.p + snploc;
    const T vare = q.vare;
    T gk = (T)gold;
    const int m = D.method, ng = D.ngroup;
    if (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) {
        const T df_va = (T)D.df_va;
        int flag = 2;
        if (m == SODAGPU_BAYES_A || cl > 1) rhs = rhs + zz * gk;
        if (m == SODAGPU_BAYES_B && sizeof(T) == 8) {
            // the inclusion comes first: u < 1 / (1 + exp(s_1 - s_2)), which is 0 above 700 as in the reference
            const T d = a.b[0] - (a.b[1] + a.c * (rhs * rhs));
            flag = at_most_700(d) && a.u * ((T)1.0 + t_exp(d)) < (T)1.0 ? 2 : 1;
        } else if (m == SODAGPU_BAYES_B) {
            const T s1 = q.logp[0];
            const T uhat = rhs / a.den;
            const T s2 = (T)-0.5 * (a.ld - (rhs * uhat / vare)) + q.logp[1];
            const T clike = s1 - s2;
            T sk;
            if (clike > (T)700.0) sk = (T)0.0;
            else if (clike < (T)-700.0) sk = (T)1.0;
            else sk = (T)1.0 / ((T)1.0 + t_exp(clike));
            flag = a.u < sk ? 2 : 1;
        }
        const T mean = flag == 1 ? (T)0.0 : rhs / a.den, sd = flag == 1 ? a.sdv : a.sd;
        if (a.plain) {
            gk = t_rnorm<T>(mean, sd, R);
            a.gam = gamma_pre<T>((T)0.5 * (df_va + (T)1.0), R, &a.err);
        } else {
            gk = normal_from(mean, sd, a.z);
        }
        const double gnew = flag == 1 ? 0.0 : (double)gk;
        D.g[o] = gnew;
        if (m == SODAGPU_BAYES_B) D.cls[o] = flag;
        const T scale = (gk * gk + q.scale_va * df_va) / (df_va + (T)1.0);
        D.vara_s[o] = (double)scinvchi2_from(df_va + (T)1.0, scale, a.gam);
        return gold - gnew;
    }
    // BayesC / Cpi / R / Rc
    if (cl > 1) rhs = rhs + zz * gk;
    const int nm = D.nmix;
    int flag = 1;
    T v1, sd;
    if (nm <= DRAW_PRE) {
        if constexpr (sizeof(T) == 8) {
            flag = draw_class64(rhs * rhs, a.b, q.c, nm, a.u);
        } else {
            // every loop unrolled: the scores stay in registers
            T sv[DRAW_PRE];
#pragma unroll
            for (int kk = 0; kk < DRAW_PRE; ++kk) {
                const T lp = ng > 1 && kk < nm ? (T)S->log_p[sg + kk * ng] : q.logp[kk];
                sv[kk] = lp;
                if (kk > 0 && kk < nm) {
                    const T uhat = rhs / q.den[kk];
                    sv[kk] = (T)-0.5 * (q.ld[kk] - (rhs * uhat / vare)) + lp;
                }
            }
            T ssculm = (T)0.0;
            bool done = false;
#pragma unroll
            for (int kk = 0; kk < DRAW_PRE; ++kk) {
                if (kk < nm && !done) {
                    T sk = (T)0.0;
                    bool overflow = false;
#pragma unroll
                    for (int j = 0; j < DRAW_PRE; ++j) {
                        if (j < nm && j != kk && !overflow) {
                            const T clike = sv[j] - sv[kk];
                            if (clike > (T)700.0) overflow = true;
                            else if (clike >= (T)-700.0) sk = sk + t_exp(clike);
                        }
                    }
                    ssculm = ssculm + (overflow ? (T)0.0 : (T)1.0 / ((T)1.0 + sk));
                    if (a.u < ssculm) {
                        flag = kk + 1;
                        done = true;
                    }
                }
            }
        }
        v1 = q.v1[1];
        sd = q.sd[1];
#pragma unroll
        for (int k = 2; k < DRAW_PRE; ++k)
            if (k == flag - 1) {
                v1 = q.v1[k];
                sd = q.sd[k];
            }
        if (flag == 1) v1 = (T)1.0;
    } else {
        T sv[MAXDIST];
        sv[0] = (T)S->log_p[sg];
        for (int kk = 1; kk < nm; ++kk) {
            const T logdetV = t_log((T)S->gp[kk] * q.zz_vare + (T)1.0);
            const T uhat = rhs / (zz + (T)S->vare_gp[kk]);
            sv[kk] = (T)-0.5 * (logdetV - (rhs * uhat / vare)) + (T)S->log_p[sg + kk * ng];
        }
        T ssculm = (T)0.0;
        for (int kk = 0; kk < nm; ++kk) {
            const T skk = sv[kk];
            T sk = (T)0.0;
            bool overflow = false;
            for (int j = 0; j < nm; ++j) {
                if (j == kk) continue;
                const T clike = sv[j] - skk;
                if (clike < (T)-700.0) continue;
                if (clike > (T)700.0) { overflow = true; break; }
                sk = sk + t_exp(clike);
            }
            ssculm = ssculm + (overflow ? (T)0.0 : (T)1.0 / ((T)1.0 + sk));
            if (a.u < ssculm) { flag = kk + 1; break; }
        }
        v1 = zz + vare / (flag == 1 ? (T)1.0 : (T)S->gp[flag - 1]);
        sd = t_sqrt(vare / v1);
    }
    double gnew = 0.0;
    if (flag != 1) {
        const T mean = rhs / v1;
        gnew = (double)(sd <= (T)0.0 ? mean : normal_from(mean, sd, a.z));
    }
    D.cls[o] = flag;
    D.g[o] = gnew;
    return gold - gnew;
}

}  // namespace soda

#include "rhs_kernel.cuh"

namespace soda {

// ---------------------------------------------------------------------------
// iteration start and the mu draw
// ---------------------------------------------------------------------------
constexpr int MU_THREADS = 256;
constexpr int MU_ROWS = 4 * MU_THREADS;   // rows per CTA of the mu kernels and of the sum of r^2
static_assert(MU_ROWS == (MU_THREADS / 32) * ROW_TILE, "k_mu_apply gives a row tile to each warp");

__host__ __device__ inline int mu_grid(int n) { return (n + MU_ROWS - 1) / MU_ROWS; }

__device__ __forceinline__ void iter_begin_body(const Dev &D, const VB &vb)
{
    tc::pdl_trigger();
    tc::pdl_wait();
    RunCtl *ctl = D.ctl;
    const int rep = ctl->rep + 1;
    ctl->rep = rep;
    if (rep % D.thin == 0) ctl->trace_iter += 1;
}

__global__ void  k_iter_begin(Dev D)
{
    iter_begin_body(D, vb_native());
}


// The mu draw (models.f90:130-132) in two passes over r.  The first sums MU_ROWS rows per CTA, and the last
// CTA of a chain to finish (a ticket that wraps to zero) adds the chain's partial sums and draws; the second
// applies the draw.  Both are bound by their launch and one pass over r (16 bytes a row and chain): at n =
// 50,000 and 16 chains they take 29 us, against 244 us when every CTA of the second pass added all partial
// sums by itself, one after another.
__device__ __forceinline__ void mu_partial_body(const Dev &D, const VB &vb)
{
    __shared__ double sh[33];
    __shared__ int s_last;
    tc::pdl_trigger();
    tc::pdl_wait();
    const int c = vb.y, rep = cur_rep(D);
    ChainScal *S = &D.scal[c];
    const double mu_old = S->mu[(rep - 1) & 1];
    const double *r = D.r + (size_t)c * D.ldr;
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < MU_ROWS / MU_THREADS; ++q) {
        const int i = vb.x * MU_ROWS + q * MU_THREADS + threadIdx.x;
        if (i < D.n) v += r[i] + mu_old;
    }
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) {
        D.rpart[(size_t)c * D.nr_ctas + vb.x] = t;
        __threadfence();
        s_last = atomicInc(&S->mu_ticket, (unsigned)(vb.nx - 1)) == (unsigned)(vb.nx - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double w = 0.0;
    for (int q = threadIdx.x; q < vb.nx; q += MU_THREADS) w += __ldcg(D.rpart + (size_t)c * D.nr_ctas + q);
    const double tot = block_sum(w, sh);
    if (threadIdx.x == 0) {
        CRng R;
        crng_site(R, D, c, rep, 0, P_MU);
        const double nn = (double)D.n;
        S->mu[rep & 1] = d_rnorm(tot / nn, sqrt(S->vare / nn), R);
    }
}

__global__ void __launch_bounds__(MU_THREADS) k_mu_partial(Dev D)
{
    mu_partial_body(D, vb_native());
}


// A warp takes a tile of ROW_TILE rows, four consecutive ones a lane (16-byte loads and stores of r, 8-byte
// ones of its bf16 split), and leaves the tile's sum for the FP8 centring.  Rows n .. ldr-1 stay zero.
__device__ __forceinline__ void mu_apply_body(const Dev &D, const VB &vb)
{
    tc::pdl_trigger();
    tc::pdl_wait();
    const int c = vb.y, rep = cur_rep(D), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = vb.x * (MU_THREADS / 32) + warp;
    if (tile >= D.nr_ctas) return;
    const ChainScal *S = &D.scal[c];
    const double mu_old = S->mu[(rep - 1) & 1], mu = S->mu[rep & 1];
    const int i0 = tile * ROW_TILE + 4 * lane;
    const size_t o = (size_t)c * D.ldr + i0;
    double2 *r2 = reinterpret_cast<double2 *>(D.r + o);
    const double2 ra = r2[0], rb = r2[1];
    double v[4] = {ra.x, ra.y, rb.x, rb.y};
    float f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = i0 + k < D.n ? (v[k] + mu_old) - mu : 0.0;
        f[k] = (float)v[k];
    }
    r2[0] = make_double2(v[0], v[1]);
    r2[1] = make_double2(v[2], v[3]);
    if (!D.tc) *reinterpret_cast<float4 *>(D.r32 + o) = make_float4(f[0], f[1], f[2], f[3]);
    if (D.rsp) {
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) tc::split3(f[k], h[k], m[k], l[k]);
        const size_t part = (size_t)D.chains * D.ldr;
        *reinterpret_cast<uint2 *>(D.rsp + o) = make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
        *reinterpret_cast<uint2 *>(D.rsp + o + part) = make_uint2(m[0] | m[1] << 16, m[2] | m[3] << 16);
        *reinterpret_cast<uint2 *>(D.rsp + o + 2 * part) = make_uint2(l[0] | l[1] << 16, l[2] | l[3] << 16);
    }
    if (D.precision == SODAGPU_FP8) {
        const double t = warp_sum((v[0] + v[1]) + (v[2] + v[3]));
        if (lane == 0) D.rsum[(size_t)c * D.nr_ctas + tile] = t;
    }
}

__global__ void __launch_bounds__(MU_THREADS) k_mu_apply(Dev D)
{
    mu_apply_body(D, vb_native());
}


}  // namespace soda

#include "update_kernel.cuh"
#include "rhs_tc.cuh"
#include "update_tc.cuh"

namespace soda {

// ---------------------------------------------------------------------------
// Single-site updates, one CTA per chain, SNPs in order: the SNPs the pivoted
// fallback skips (models.f90:178-193, 276-320, 433-495) and, for the regular
// sampler, every SNP (regular_bayes, models.f90:717-859).  The reference reads
// module copies of log_p / vare_gp for skipped SNPs that its parallel regions
// never assign; the current values are used.
//
// The SNPs are a serial chain, so what counts is the latency of one: GB300's FP64
// pipe takes 64 cycles for a warp's instruction (a quarter of the SM each), and a
// logarithm is thirty of them.  All that does not depend on the residual - the
// uniforms, the normal and gamma variates, the class scores' constants - is
// computed beforehand by k_skipped_pre, in parallel over the SNPs; k_skipped is
// left with the dot product (four warps, one on each quarter; the residual in
// shared memory, the next SNP's codes and constants loaded ahead), one
// multiply-add and one exponential per class, in parallel lanes, and a comparison.
// n = 2,326, BayesR: 3.4 us a SNP, against 7.1 us when the draw did it all.
//
// The chain is serial only where a SNP changes the residual.  A SNP outside the
// model that stays outside leaves it as it is, and after burn-in that is nearly all
// of them; so k_skipped_spec draws SS_SPEC consecutive SNPs at once against the same
// residual, keeps the draws up to and including the first that changes it, applies
// that change and goes on behind it: the draws of the serial chain exactly, 24 SNPs
// a round at 2% in the model.  The same data: 0.54 us a SNP.  Chains with more than a
// quarter of the SNPs in the model (and BayesA's, with all of them) go one by one.
// ---------------------------------------------------------------------------
constexpr int SS_SMEM_MAX = 200 * 1024;   // residual in shared memory up to 25,600 individuals
constexpr int SS_CHUNK = 16384;           // SNPs per pair of launches: bounds the records
constexpr int SS_HEAD = 12;               // a record's doubles before the (c_k, b_k) pairs of the classes
enum { SS_U = 0, SS_POS, SS_SNP, SS_RR, SS_SN, SS_DEN, SS_SD, SS_SDV, SS_GD, SS_GV, SS_GW, SS_FLAGS };
constexpr int SS_CTAS = 8;                // CTAs of a chain's cluster in k_skipped_spec, four warps each
constexpr int SS_SPEC = 4 * SS_CTAS;      // SNPs a round
constexpr double SS_SMALL = 1.0, SS_PLAIN = 2.0;   // SS_FLAGS: gamma shape below 1; a standard deviation is 0

int sweep_skip_stride(int nmix) { return SS_HEAD + 2 * nmix; }
size_t sweep_skip_records(int nskipped, int chains, int nmix)
{
    return (size_t)std::min(nskipped, SS_CHUNK) * chains * sweep_skip_stride(nmix);
}

// Record of skipped SNP t0 + t (of cnt) of chain c.  Class k's score, for right-hand side rhs, is b_k + c_k rhs^2
// (models.f90:362-366 with the quotient rhs^2 / ((zz + sigma2_e / gamma) sigma2_e) as one factor).
__device__ __forceinline__ void skipped_pre_body(const Dev &D, const VB &vb, int t0, int cnt)
{
    const int t = vb.x * 64 + threadIdx.x, c = vb.y;
    if (t >= cnt) return;
    const int rep = cur_rep(D), snp = D.iskipped[t0 + t], m = D.method, nm = D.nmix, ng = D.ngroup;
    const ChainScal *S = &D.scal[c];
    const double vare = S->vare, zz = D.xpx[snp], zz_vare = zz / vare;
    const int stride = SS_HEAD + 2 * nm;
    double *q = D.ssrec + ((size_t)c * min(D.nskipped, SS_CHUNK) + t) * stride;
    CRng R;
    crng_site(R, D, c, rep, snp, P_SKIP);
    q[SS_POS] = (double)D.pos_of[snp];
    q[SS_SNP] = (double)snp;
    // how many of the chunk's SNPs are in the model (cleared before the launch)
    if (m != SODAGPU_BAYES_A && D.cls[(size_t)c * D.p + snp] > 1) atomicAdd(&D.ssdense[c], 1);
    if (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) {
        const double vs = D.vara_s[(size_t)c * D.p + snp];
        DrawSub<double> sub;
        sub.vare = vare;
        sub.zz_vare = zz_vare;
        DrawSnp<double> a;
        a.u = a.ld = a.sdv = 0.0;
        draw_ahead(D, S, sub, zz, vs, 0, R, a);
        q[SS_U] = a.u;
        q[SS_DEN] = a.den;
        q[SS_SD] = a.sd;
        q[SS_SDV] = a.sdv;
        q[SS_FLAGS] = a.plain ? SS_PLAIN : (a.gam.small ? SS_SMALL : 0.0);
        if (!a.plain) {
            q[SS_RR] = a.z.rr;
            q[SS_SN] = a.z.sn;
            q[SS_GD] = a.gam.d;
            q[SS_GV] = a.gam.v;
            q[SS_GW] = a.gam.wp;
        }
        if (m == SODAGPU_BAYES_B) {
            q[SS_HEAD] = 0.0;
            q[SS_HEAD + 1] = S->log_p[0];
            q[SS_HEAD + 2] = 0.5 / (a.den * vare);
            q[SS_HEAD + 3] = S->log_p[ng] - 0.5 * a.ld;
        }
        if (a.err) flag_err(D, 1);
        return;
    }
    const int sg = D.grp[snp] - 1;
    q[SS_U] = crng_unit(R);
    const NormalPre<double> z = normal_pre<double>(R);
    q[SS_RR] = z.rr;
    q[SS_SN] = z.sn;
    q[SS_HEAD] = 0.0;
    q[SS_HEAD + 1] = S->log_p[sg];
    for (int k = 1; k < nm; ++k) {
        q[SS_HEAD + 2 * k] = 0.5 / ((zz + S->vare_gp[k]) * vare);
        q[SS_HEAD + 2 * k + 1] = S->log_p[sg + k * ng] - 0.5 * log(S->gp[k] * zz_vare + 1.0);
    }
}

__global__ void __launch_bounds__(64) k_skipped_pre(Dev D, int t0, int cnt)
{
    skipped_pre_body(D, vb_native(), t0, cnt);
}

// The class of a SNP (1-based) from its uniform u and this lane's class score s (lanes 0 .. nm-1; all 32 enter): the
// first class whose cumulative weight exceeds u times their sum, weights exp(s_k - s_0), or relative to the largest
// score where that could overflow (draw_class64).
__device__ __forceinline__ int skipped_class(double s, double u, int nm)
{
    const int lane = threadIdx.x & 31;
    const double d = s - __shfl_sync(0xffffffffu, s, 0);
    double w = d;
    if (__ballot_sync(0xffffffffu, lane < nm && d > 700.0)) {
        double top = lane < nm ? s : -1e308;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
        w = top - s > 700.0 ? -1e308 : s - top;
    }
    w = lane < nm ? exp(w) : 0.0;
    for (int o = 1; o < nm; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += v;
    }
    const double sum = __shfl_sync(0xffffffffu, w, nm - 1);
    const unsigned hit = __ballot_sync(0xffffffffu, lane < nm && u * sum < w);
    return hit ? __ffs(hit) : 1;
}

// The draws of a record whose standard deviation is 0, in the plain order (A/B; practically never).
static __device__ __noinline__ void skipped_plain(const Dev &D, int c, int rep, int snp, double mean, double sd,
                                                  double &gt, GammaPre<double> &gam)
{
    CRng R;
    int err = 0;
    crng_site(R, D, c, rep, snp, P_SKIP);
    if (D.method == SODAGPU_BAYES_B) crng_unit(R);
    gt = t_rnorm<double>(mean, sd, R);
    gam = gamma_pre<double>(0.5 * (D.df_va + 1.0), R, &err);
    if (err) flag_err(D, 1);
}

// The draw of SNP snp of chain c from its dot product, by a warp (the same in every lane): its new effect and class and
// upd = g_old - g_new.  gk, cl: the SNP's effect and class; cb: this lane's class constants; q: its record, u its
// uniform.
struct SkippedDraw {
    double upd, gt;
    int flag;
    GammaPre<double> gam;
};
__device__ __forceinline__ SkippedDraw skipped_draw(const Dev &D, const ChainScal *S, int c, int rep, int snp,
                                                    double dot, double gk, int cl, double zz, double2 cb,
                                                    const double *q, double u)
{
    const int lane = threadIdx.x & 31, m = D.method, nm = D.nmix;
    SkippedDraw x;
    double rhs = dot;
    if (m == SODAGPU_BAYES_A || cl > 1) rhs = rhs + zz * gk;
    x.flag = 2;
    if (m != SODAGPU_BAYES_A) {
        const double s = lane == 0 ? cb.y : fma(rhs * rhs, cb.x, cb.y);
        if (m == SODAGPU_BAYES_B) {   // the inclusion comes first: u < 1 / (1 + exp(s_1 - s_2)), 0 above 700
            const double d = __shfl_sync(0xffffffffu, s, 0) - __shfl_sync(0xffffffffu, s, 1);
            x.flag = at_most_700(d) && u * (1.0 + exp(d)) < 1.0 ? 2 : 1;
        } else {
            x.flag = skipped_class(s, u, nm);
        }
    }
    x.upd = x.gt = 0.0;
    if (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) {
        const double mean = x.flag == 1 ? 0.0 : rhs / q[SS_DEN], sd = x.flag == 1 ? q[SS_SDV] : q[SS_SD];
        x.gam = {q[SS_GD], q[SS_GV], q[SS_GW], q[SS_FLAGS] == SS_SMALL};
        if (q[SS_FLAGS] == SS_PLAIN) {
            skipped_plain(D, c, rep, snp, mean, sd, x.gt, x.gam);
        } else {
            const NormalPre<double> z = {q[SS_RR], q[SS_SN]};
            x.gt = normal_from(mean, sd, z);
        }
        x.upd = x.flag == 1 ? (cl > 1 ? gk : 0.0) : gk - x.gt;
    } else if (x.flag != 1) {
        const double vare = S->vare, v1 = zz + vare / S->gp[x.flag - 1], sd = sqrt(vare / v1), mean = rhs / v1;
        const NormalPre<double> z = {q[SS_RR], q[SS_SN]};
        x.gt = sd <= 0.0 ? mean : normal_from(mean, sd, z);
        x.upd = gk - x.gt;
    } else if (cl > 1) {
        x.upd = gk;
    }
    return x;
}

// Writes the draw (one thread).
__device__ __forceinline__ void skipped_commit(const Dev &D, const ChainScal *S, int c, int snp, const SkippedDraw &x)
{
    const int m = D.method;
    const size_t o = (size_t)c * D.p + snp;
    if (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) {
        D.g[o] = x.flag == 1 ? 0.0 : x.gt;
        if (m == SODAGPU_BAYES_B) D.cls[o] = x.flag;
        const double scale = (x.gt * x.gt + S->scale_va * D.df_va) / (D.df_va + 1.0);
        D.vara_s[o] = scinvchi2_from(D.df_va + 1.0, scale, x.gam);
        return;
    }
    D.g[o] = x.gt;
    D.cls[o] = x.flag;
}

// Whether chain c's chunk of cnt SNPs goes through k_skipped_spec (residual in shared memory, few SNPs in the model).
__device__ __forceinline__ bool skipped_speculates(const Dev &D, int c, int cnt)
{
    return D.method != SODAGPU_BAYES_A && 4 * D.ssdense[c] <= cnt;
}

// NT threads: 128 with the residual in shared memory, 512 (for the loads in flight) with it in global memory.
template <int NT>
__device__ __forceinline__ void skipped_body(const Dev &D, const VB &vb, int t0, int cnt)
{
    constexpr bool SMEM = NT == 128;
    constexpr int NW = NT / 32, AHEAD = 8;   // words of codes a thread loads ahead (four individuals each)
    extern __shared__ __align__(16) double s_r[];
    __shared__ double s_part[NW];
    __shared__ double s_upd;
    const int c = vb.x, rep = cur_rep(D);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nm = D.nmix;
    if (SMEM && skipped_speculates(D, c, cnt)) return;
    const ChainScal *S = &D.scal[c];
    double *rg = D.r + (size_t)c * D.ldr, *r = SMEM ? s_r : rg;
    // four consecutive individuals a word; rows n .. ldr-1 of the residual are zero, and stay so
    const int words = (D.n + 3) / 4;
    if (SMEM) {
        for (int i = tid; i < 4 * words; i += NT) s_r[i] = rg[i];
    }
    const int stride = SS_HEAD + 2 * nm;
    const double *rec = D.ssrec + (size_t)c * min(D.nskipped, SS_CHUNK) * stride;
    // what a SNP needs besides the residual, loaded while the SNP before it is drawn
    struct Next {
        uint32_t code[AHEAD];
        const uint32_t *col;
        double x0, x1, x2, gk, zz, u;
        double2 cb;
        int snp, cl;
    };
    // (the SNP's id and position come in one and two turns before that: no load waits for another's address)
    auto fetch = [&](int t, int snp, int k, Next &x) {
        if (t >= cnt) return;
        x.snp = snp;
        x.col = reinterpret_cast<const uint32_t *>(D.G + (size_t)k * D.ldx);
#pragma unroll
        for (int w = 0; w < AHEAD; ++w) x.code[w] = tid + w * NT < words ? __ldg(x.col + tid + w * NT) : 0u;
        const double2 xa = *reinterpret_cast<const double2 *>(D.xv + (size_t)k * 4);
        x.x0 = xa.x;
        x.x1 = xa.y;
        x.x2 = D.xv[(size_t)k * 4 + 2];
        if (warp == 0) {
            const size_t o = (size_t)c * D.p + x.snp;
            x.gk = D.g[o];
            x.cl = D.cls[o];
            x.zz = D.xpx[x.snp];
            x.u = rec[(size_t)t * stride + SS_U];
            x.cb = lane < nm ? make_double2(rec[(size_t)t * stride + SS_HEAD + 2 * lane],
                                            rec[(size_t)t * stride + SS_HEAD + 2 * lane + 1])
                             : make_double2(0.0, 0.0);
        }
    };
    Next cur, nxt;
    auto snp_at = [&](int t) { return D.iskipped[t0 + min(t, cnt - 1)]; };
    int snp1 = snp_at(1), pos1 = D.pos_of[snp1], snp2 = snp_at(2);
    fetch(0, snp_at(0), D.pos_of[snp_at(0)], cur);
    if (SMEM) __syncthreads();
    for (int t = 0; t < cnt; ++t) {
        fetch(t + 1, snp1, pos1, nxt);
        const int pos2 = D.pos_of[snp2], snp3 = snp_at(t + 3);
        auto pick = [&](uint32_t g) { return g == 0u ? cur.x0 : (g == 1u ? cur.x1 : cur.x2); };
        double p0 = 0.0;
        auto dot4 = [&](int i, uint32_t cw) {
            const double2 a = *reinterpret_cast<const double2 *>(r + i), b = *reinterpret_cast<const double2 *>(r + i + 2);
            p0 = fma(a.x, pick(cw & 3u), p0);
            p0 = fma(a.y, pick(cw >> 8 & 3u), p0);
            p0 = fma(b.x, pick(cw >> 16 & 3u), p0);
            p0 = fma(b.y, pick(cw >> 24 & 3u), p0);
        };
#pragma unroll
        for (int w = 0; w < AHEAD; ++w)
            if (tid + w * NT < words) dot4(4 * (tid + w * NT), cur.code[w]);
#pragma unroll 4
        for (int w = AHEAD; tid + w * NT < words; ++w) dot4(4 * (tid + w * NT), __ldg(cur.col + tid + w * NT));
        p0 = warp_sum(p0);
        if (lane == 0) s_part[warp] = p0;
        __syncthreads();
        if (warp == 0) {
            double d;
            if (NW == 4) {
                d = (s_part[0] + s_part[1]) + (s_part[2] + s_part[3]);
            } else {
                d = warp_sum(lane < NW ? s_part[lane] : 0.0);
            }
            const SkippedDraw x = skipped_draw(D, S, c, rep, cur.snp, d, cur.gk, cur.cl, cur.zz, cur.cb,
                                               rec + (size_t)t * stride, cur.u);
            if (lane == 0) {
                s_upd = x.upd;
                skipped_commit(D, S, c, cur.snp, x);
            }
        }
        __syncthreads();
        const double upd = s_upd;
        if (upd != 0.0) {
            auto add4 = [&](int i, uint32_t cw) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (i + e < D.n) r[i + e] = fma(pick(cw >> (8 * e) & 3u), upd, r[i + e]);
            };
#pragma unroll
            for (int w = 0; w < AHEAD; ++w)
                if (tid + w * NT < words) add4(4 * (tid + w * NT), cur.code[w]);
            for (int w = AHEAD; tid + w * NT < words; ++w) add4(4 * (tid + w * NT), __ldg(cur.col + tid + w * NT));
        }
        cur = nxt;
        snp1 = snp2;
        pos1 = pos2;
        snp2 = snp3;
    }
    if (SMEM) {
        __syncthreads();
        for (int i = tid; i < D.n; i += NT) rg[i] = s_r[i];
    }
}

// Rounds of SS_SPEC SNPs, a warp each, over a cluster of SS_CTAS CTAs that all hold the residual; the warps exchange
// their updates through distributed shared memory.  Bound by a warp's FP64 pipe: n / 32 multiply-adds of 64 cycles a
// round, and the draw's exponential.
__device__ __forceinline__ void skipped_spec_body(const Dev &D, int c, int t0, int cnt)
{
    namespace cg = cooperative_groups;
    constexpr int NT = 128, AHEAD = 8;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double s_r[];
    __shared__ double s_upd[2][4];            // this CTA's warps' updates, by the round's parity
    if (!skipped_speculates(D, c, cnt)) return;   // the same for the whole cluster
    const int rep = cur_rep(D), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nm = D.nmix, mine = 4 * rank + warp;
    const ChainScal *S = &D.scal[c];
    double *rg = D.r + (size_t)c * D.ldr;
    const int words = (D.n + 3) / 4, stride = SS_HEAD + 2 * nm;
    for (int i = tid; i < 4 * words; i += NT) s_r[i] = rg[i];
    const double *rec = D.ssrec + (size_t)c * min(D.nskipped, SS_CHUNK) * stride;
    __syncthreads();
    int par = 0;
    for (int t = 0; t < cnt; par ^= 1) {
        const bool in = t + mine < cnt;
        SkippedDraw x;
        x.upd = 0.0;
        int snp = 0;
        if (in) {
            const double *q = rec + (size_t)(t + mine) * stride;
            snp = (int)q[SS_SNP];
            const int k = (int)q[SS_POS];
            const double u = q[SS_U];
            const double2 cb = lane < nm ? make_double2(q[SS_HEAD + 2 * lane], q[SS_HEAD + 2 * lane + 1])
                                         : make_double2(0.0, 0.0);
            const uint32_t *col = reinterpret_cast<const uint32_t *>(D.G + (size_t)k * D.ldx);
            const double x0 = D.xv[(size_t)k * 4], x1 = D.xv[(size_t)k * 4 + 1], x2 = D.xv[(size_t)k * 4 + 2];
            const size_t o = (size_t)c * D.p + snp;
            const double gk = D.g[o], zz = D.xpx[snp];
            const int cls = D.cls[o];
            double p0 = 0.0;
            for (int w0 = lane; w0 < words; w0 += 32 * AHEAD) {
                uint32_t cw[AHEAD];
#pragma unroll
                for (int v = 0; v < AHEAD; ++v) cw[v] = w0 + 32 * v < words ? __ldg(col + w0 + 32 * v) : 0u;
#pragma unroll
                for (int v = 0; v < AHEAD; ++v) {
                    const int i = 4 * (w0 + 32 * v);
                    if (w0 + 32 * v >= words) break;
                    const double2 a = *reinterpret_cast<const double2 *>(s_r + i);
                    const double2 b = *reinterpret_cast<const double2 *>(s_r + i + 2);
                    auto pick = [&](uint32_t g) { return g == 0u ? x0 : (g == 1u ? x1 : x2); };
                    p0 = fma(a.x, pick(cw[v] & 3u), p0);
                    p0 = fma(a.y, pick(cw[v] >> 8 & 3u), p0);
                    p0 = fma(b.x, pick(cw[v] >> 16 & 3u), p0);
                    p0 = fma(b.y, pick(cw[v] >> 24 & 3u), p0);
                }
            }
            x = skipped_draw(D, S, c, rep, snp, warp_sum(p0), gk, cls, zz, cb, q, u);
        }
        if (lane == 0) s_upd[par][warp] = in ? x.upd : 0.0;
        cl.sync();
        // every warp looks at all updates: SNP t + l's lies in CTA l / 4.  (The other parity's slots are written only
        // after the next barrier.)
        const double ul = cl.map_shared_rank(&s_upd[par][0], lane >> 2)[lane & 3];
        const unsigned hit = __ballot_sync(0xffffffffu, ul != 0.0);
        const int f = hit ? __ffs(hit) - 1 : SS_SPEC - 1;   // the last SNP of the round whose draw stands
        if (in && mine <= f && lane == 0) skipped_commit(D, S, c, snp, x);
        if (hit) {
            const double upd = __shfl_sync(0xffffffffu, ul, f);
            const int k = (int)rec[(size_t)(t + f) * stride + SS_POS];
            const uint32_t *col = reinterpret_cast<const uint32_t *>(D.G + (size_t)k * D.ldx);
            const double x0 = D.xv[(size_t)k * 4], x1 = D.xv[(size_t)k * 4 + 1], x2 = D.xv[(size_t)k * 4 + 2];
            __syncthreads();   // every warp has read the residual of this round
            for (int w = tid; w < words; w += NT) {
                const uint32_t cw = __ldg(col + w);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t g = cw >> (8 * e) & 3u;
                    if (4 * w + e < D.n) s_r[4 * w + e] = fma(g == 0u ? x0 : (g == 1u ? x1 : x2), upd, s_r[4 * w + e]);
                }
            }
            __syncthreads();
        }
        t += f + 1;
    }
    if (rank == 0)
        for (int i = tid; i < D.n; i += NT) rg[i] = s_r[i];
    cl.sync();   // no CTA leaves while another still reads its shared memory
}

__global__ void __cluster_dims__(SS_CTAS, 1, 1) __launch_bounds__(128) k_skipped_spec(Dev D, int t0, int cnt)
{
    skipped_spec_body(D, blockIdx.x / SS_CTAS, t0, cnt);
}

template <int NT>
__global__ void __launch_bounds__(NT) k_skipped(Dev D, int t0, int cnt)
{
    skipped_body<NT>(D, vb_native(), t0, cnt);
}

// Shared memory of k_skipped<128>, 0 when the residual does not fit (then k_skipped<512> runs).
static size_t skipped_smem(int n)
{
    const size_t b = sizeof(double) * 4 * (size_t)((n + 3) / 4);
    return b <= (size_t)SS_SMEM_MAX ? b : 0;
}


// ---------------------------------------------------------------------------
// per-iteration statistics: class counts and sum g^2 per (group, class),
// sum r^2 (models.f90:194, 321-325, 496-503, 515)
// ---------------------------------------------------------------------------
// CTAs 0..NSTAT-1 of a chain take the SNPs, the others MU_ROWS rows of r each.  One pass serves all (group, class)
// cells; the counts go through integer atomics.  With up to STAT_FAST cells a warp adds the squares of its 32 SNPs cell
// by cell (sparse chains have a few non-zero effects per warp) into its own row of shared sums, in a fixed order: seven
// FP64 instructions, of 64 cycles each, for a cell with several.  From STAT_LARGE SNPs and up to STAT_OWN cells a
// thread has sums of its own in shared memory, one FP64 instruction for a warp's 32 SNPs, and STAT_AHEAD loads in
// flight.  The iteration's kernels beside the subsets', p = 500,000, 16 chains, a quarter of the effects not zero: 235 us
// by warps, 105 us by threads; p = 200,000, one chain of BayesA: 44 and 34 us; p = 12,000, 12 cells, 16 chains: 48 and
// 51 us, for the sums' clearing and reduction, so smaller jobs stay with the warps.  More than STAT_FAST cells take one
// pass over the SNPs each (p = 12,000, 12 cells, 16 chains: 13 us in one pass, 122 us in twelve).
constexpr int STAT_OWN = 16, STAT_FAST = 64, STAT_AHEAD = 4;
constexpr int STAT_LARGE = STAT_AHEAD * NSTAT * 256;   // a full turn of every thread

__device__ __forceinline__ void stats_body(const Dev &D, const VB &vb)
{
    __shared__ double sh[33];
    __shared__ double s_sum[STAT_OWN * 256];
    __shared__ int s_cnt[STAT_FAST];
    static_assert(8 * STAT_FAST <= STAT_OWN * 256, "the warps' rows of sums fit");
    tc::pdl_trigger();
    tc::pdl_wait();
    const int c = vb.y;
    if (vb.x >= NSTAT) {
        const int rb = vb.x - NSTAT;
        const double *r = D.r + (size_t)c * D.ldr;
        double v2 = 0.0;
#pragma unroll
        for (int q = 0; q < MU_ROWS / 256; ++q) {
            const int i = rb * MU_ROWS + q * 256 + threadIdx.x;
            if (i < D.n) v2 += r[i] * r[i];
        }
        const double t = block_sum(v2, sh);
        if (threadIdx.x == 0) D.rpart[(size_t)c * D.nr_ctas + rb] = t;
        return;
    }
    const int ngm = D.ngroup * D.nmix;
    const size_t base = (size_t)c * D.p;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ngm <= STAT_OWN && D.p >= STAT_LARGE) {
        constexpr int STEP = NSTAT * 256;
        double *own = s_sum + threadIdx.x;
        for (int e = 0; e < ngm; ++e) own[256 * e] = 0.0;
        if (threadIdx.x < ngm) s_cnt[threadIdx.x] = 0;
        __syncthreads();
        for (int j0 = vb.x * 256 + 32 * warp; j0 < D.p; j0 += STAT_AHEAD * STEP) {
            int e[STAT_AHEAD];
            double gj[STAT_AHEAD];
#pragma unroll
            for (int q = 0; q < STAT_AHEAD; ++q) {
                const int64_t j = (int64_t)j0 + q * STEP + lane;
                e[q] = j < D.p ? (D.grp[j] - 1) + (D.cls[base + j] - 1) * D.ngroup : -1;
                gj[q] = j < D.p ? D.g[base + j] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < STAT_AHEAD; ++q) {
                const unsigned same = __match_any_sync(0xffffffffu, e[q]);
                if (e[q] >= 0 && lane == __ffs(same) - 1) atomicAdd(&s_cnt[e[q]], __popc(same));
                // not zero, by its bits: an FP64 comparison would take the pipe as long as the addition
                if (__double_as_longlong(gj[q]) << 1) own[256 * e[q]] = fma(gj[q], gj[q], own[256 * e[q]]);
            }
        }
        __syncthreads();
        for (int e = warp; e < ngm; e += 8) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) t += s_sum[256 * e + 32 * w + lane];
            t = warp_sum(t);
            if (lane == 0) {
                const size_t o = ((size_t)c * NSTAT + vb.x) * ngm + e;
                D.statpart[o] = t;
                D.cntpart[o] = s_cnt[e];
            }
        }
        return;
    }
    if (ngm <= STAT_FAST) {
        double (*s_acc)[STAT_FAST] = reinterpret_cast<double (*)[STAT_FAST]>(s_sum);
        for (int e = threadIdx.x; e < 8 * ngm; e += 256) s_acc[e / ngm][e % ngm] = 0.0;
        if (threadIdx.x < ngm) s_cnt[threadIdx.x] = 0;
        __syncthreads();
        for (int j0 = vb.x * 256 + 32 * warp; j0 < D.p; j0 += NSTAT * 256) {
            const int j = j0 + lane;
            int e = -1;
            double v = 0.0;
            if (j < D.p) {
                e = (D.grp[j] - 1) + (D.cls[base + j] - 1) * D.ngroup;
                const double gj = D.g[base + j];
                v = gj * gj;
            }
            const unsigned same = __match_any_sync(0xffffffffu, e);
            if (e >= 0 && lane == __ffs(same) - 1) atomicAdd(&s_cnt[e], __popc(same));
            unsigned todo = __ballot_sync(0xffffffffu, v != 0.0);
            while (todo) {   // one cell at a time, in the order of its first lane
                const int src = __ffs(todo) - 1, e0 = __shfl_sync(0xffffffffu, e, src);
                const unsigned in = __ballot_sync(0xffffffffu, v != 0.0 && e == e0);
                if (__popc(in) == 1) {
                    if (lane == src) s_acc[warp][e0] += v;
                } else {
                    const double t = warp_sum(v != 0.0 && e == e0 ? v : 0.0);
                    if (lane == 0) s_acc[warp][e0] += t;
                }
                __syncwarp();
                todo &= ~in;
            }
        }
        __syncthreads();
        for (int e = threadIdx.x; e < ngm; e += 256) {
            double t = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) t += s_acc[w][e];
            const size_t o = ((size_t)c * NSTAT + vb.x) * ngm + e;
            D.statpart[o] = t;
            D.cntpart[o] = s_cnt[e];
        }
        return;
    }
    for (int e = 0; e < ngm; ++e) {
        const int eg = e % D.ngroup, em = e / D.ngroup;
        double v = 0.0;
        int cnt = 0;
        for (int j = vb.x * 256 + threadIdx.x; j < D.p; j += NSTAT * 256) {
            const int cl = D.cls[base + j];
            if (D.grp[j] - 1 == eg && cl - 1 == em) {
                const double gj = D.g[base + j];
                v += gj * gj;
                ++cnt;
            }
        }
        const double tv = block_sum(v, sh);
        const double tc = block_sum((double)cnt, sh);
        if (threadIdx.x == 0) {
            const size_t o = ((size_t)c * NSTAT + vb.x) * ngm + e;
            D.statpart[o] = tv;
            D.cntpart[o] = (int32_t)tc;
        }
    }
}

__global__ void __launch_bounds__(256) k_stats(Dev D)
{
    stats_body(D, vb_native());
}


// The hyper-parameter draws of a chain, one CTA.  They are bound by the latency of a few FP64 draws, so the
// three that do not depend on one another run at once: sigma2_g in warp 0, sigma2_e in warp 1, and pi in the
// others, a lane for each of its gamma variates.  With the sums before them and the tables after them spread over
// the CTA's threads, a chain of BayesR takes 18 us (62 us when one thread did it all, 28 us with one thread a group).
constexpr int HYPER_THREADS = 256;

__device__ __forceinline__ void hyper_body(const Dev &D, const VB &vb)
{
    __shared__ double s_rr;
    tc::pdl_trigger();
    tc::pdl_wait();
    const int c = vb.x, rep = cur_rep(D), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int NW = HYPER_THREADS / 32;
    ChainScal *S = &D.scal[c];
    const int ng = D.ngroup, nm = D.nmix, ngm = ng * nm, m = D.method;
    // sums over the CTAs of k_stats: cell e by warp e % NW, sum r^2 by the last warp
    for (int e = warp; e < ngm; e += NW) {
        double v = 0.0;
        int cnt = 0;
        for (int t = lane; t < NSTAT; t += 32) {
            const size_t o = ((size_t)c * NSTAT + t) * ngm + e;
            v += D.statpart[o];
            cnt += D.cntpart[o];
        }
        v = warp_sum(v);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0) {
            S->varindist[e] = v;
            // BayesA tracks no class counts (models.f90:194): its trace shows none
            S->snpindist[e] = m == SODAGPU_BAYES_A ? 0 : cnt;
        }
    }
    if (warp == NW - 1) {
        double rr = 0.0;
        for (int t = lane; t < mu_grid(D.n); t += 32) rr += D.rpart[(size_t)c * D.nr_ctas + t];
        rr = warp_sum(rr);
        if (lane == 0) s_rr = rr;
    }
    __syncthreads();
    int err = 0;
    if (tid == 0) {
        if (m == SODAGPU_BAYES_B) {
            S->included = S->snpindist[ng];
            S->varindist[0] = 0.0;
        } else if (m != SODAGPU_BAYES_A) {
            int excl = 0;
            for (int i = 0; i < ng; ++i) excl += S->snpindist[i];
            S->included = D.p - excl;
            double scale = 0.0;
            for (int i = 0; i < ng; ++i)
                for (int j = 1; j < nm; ++j) scale = scale + S->varindist[i + j * ng] / D.mix[j];
            scale = (scale + S->scale_va * D.df_va) / (D.df_va + (double)S->included);
            CRng R;
            crng_site(R, D, c, rep, 0, P_VARA);
            S->vara = d_rscinvchi2((double)S->included + D.df_va, scale, R, &err);
            for (int j = 0; j < nm; ++j) S->gp[j] = D.mix[j] * S->vara;
        }
    } else if (tid == 32) {
        const double nn = (double)D.n;
        const double scale = (s_rr + D.scale_ve * D.df_ve) / (nn + D.df_ve);
        CRng R;
        crng_site(R, D, c, rep, 0, P_VARE);
        S->vare = d_rscinvchi2(nn + D.df_ve, scale, R, &err);
    } else if (warp >= 2 && (m == SODAGPU_BAYES_CPI || m == SODAGPU_BAYES_R || m == SODAGPU_BAYES_RC)) {
        // pi ~ Dirichlet(counts + alpha) of each group (models.f90:517-522).  The nm gamma variates of a group come from
        // one stream, one after another, 5 us each; nearly always each takes exactly three uniforms, so nm lanes draw
        // them at once from those places, and where one but the last took more, its group's first lane draws them in
        // turn.  From an injected-draw tape always in turn: a guessed place could run past a record that is long enough
        const int per = 32 / nm, sub = lane / nm, j = lane - sub * nm, first = sub * nm;
        const bool guess = D.tape == nullptr;
        for (int i0 = (warp - 2) * per; i0 < ng; i0 += (NW - 2) * per) {
            const int i = i0 + sub;
            const bool in = sub < per && i < ng;
            CRng R;
            GammaPre<double> gam;
            gam.taken = 3;
            double x = 0.0;
            int gerr = 0;
            if (in && guess) {
                crng_site(R, D, c, rep, i, P_PI);
                crng_skip(R, 3 * j);
                gam = gamma_pre<double>((double)S->snpindist[i + j * ng] + D.alpha[j], R, &gerr);
                x = gamma_from(1.0, gam);
            }
            const unsigned odd = __ballot_sync(0xffffffffu, in && (!guess || (j < nm - 1 && gam.taken != 3)));
            const bool redo = in && (odd >> first & ((1u << nm) - 1u)) != 0;
            double y[MAXDIST];
            if (redo) {
                gerr = 0;
                if (j == 0) {
                    crng_site(R, D, c, rep, i, P_PI);
                    for (int q = 0; q < nm; ++q)
                        y[q] = d_rgamma((double)S->snpindist[i + q * ng] + D.alpha[q], 1.0, R, &gerr);
                }
            }
            double sx = 0.0;
            for (int q = 0; q < nm; ++q) {
                double v = __shfl_sync(0xffffffffu, x, min(first + q, 31));
                const double w = __shfl_sync(0xffffffffu, redo && j == 0 ? y[q] : 0.0, min(first, 31));
                if (redo) v = w;
                if (j == q) x = v;
                sx = sx + v;
            }
            if (in) S->p[i + j * ng] = x / sx;
            err |= gerr;
        }
    }
    if (err) flag_err(D, 1);
    __syncthreads();
    const bool keep = rep > D.burnin && rep % D.thin == 0;
    const double mu = S->mu[rep & 1];
    for (int e = tid; e < ngm; e += HYPER_THREADS) {
        if (keep) {
            // soda_bayes keeps varstore for every method (models.f90:530), regular_bayes
            // not for BayesA (models.f90:893-896)
            if (!(D.regular && m == SODAGPU_BAYES_A)) S->varstore[e] = S->varstore[e] + S->varindist[e];
            if (m != SODAGPU_BAYES_A) {
                S->snpstore[e] = S->snpstore[e] + S->snpindist[e];
                if (m != SODAGPU_BAYES_B && m != SODAGPU_BAYES_C) S->pstore[e] = S->pstore[e] + S->p[e];
            }
        }
        // log_p for the next iteration (models.f90:198-199, 330-338)
        if (m != SODAGPU_BAYES_A) S->log_p[e] = log(S->p[e]);
    }
    if (m != SODAGPU_BAYES_A)
        for (int j = 1 + tid; j < nm; j += HYPER_THREADS) S->vare_gp[j] = S->vare / S->gp[j];
    if (tid == 0) {
        S->keep = keep;
        if (keep) {
            S->counter += 1;
            S->mu_store = S->mu_store + mu;
            S->vare_store = S->vare_store + S->vare;
            if (m != SODAGPU_BAYES_A) S->included_store = S->included_store + S->included;
            if (m != SODAGPU_BAYES_A && m != SODAGPU_BAYES_B) S->vara_store = S->vara_store + S->vara;
        }
    }
    if (rep % D.thin == 0) {
        RunCtl *ctl = D.ctl;
        const int row = (ctl->trace_iter - 1) * D.chains + c;
        if (ctl->trace && row >= 0 && row < ctl->trace_cap) {
            sodagpu_trace_row *tr = ctl->trace + row;
            if (tid == 0) {
                tr->chain = c;
                tr->rep = rep;
                tr->included = S->included;
                tr->pad = 0;
                tr->mu = mu;
                tr->vare = S->vare;
                tr->vara = S->vara;
            }
            for (int j = tid; j < MAXDIST; j += HYPER_THREADS) {
                tr->snpindist[j] = j < nm ? S->snpindist[j * ng] : 0;
                tr->varindist[j] = j < nm ? S->varindist[j * ng] : 0.0;
            }
        }
    }
}

__global__ void __launch_bounds__(HYPER_THREADS) k_hyper(Dev D)
{
    hyper_body(D, vb_native());
}


// ra redraw (models.f90:523-525) and the per-SNP accumulators (528, 535-538, 544): the loads of POST_AHEAD SNPs are in
// flight before the first store.  p = 500,000, 16 chains, means kept: the kernels beside the subsets' take 145 us an
// iteration, 189 us with one SNP at a time.
constexpr int POST_AHEAD = 4;

__device__ __forceinline__ void post_body(const Dev &D, const VB &vb)
{
    tc::pdl_trigger();
    tc::pdl_wait();
    const int c = vb.y, rep = cur_rep(D);
    const ChainScal *S = &D.scal[c];
    const int t0 = vb.x * blockDim.x + threadIdx.x, stride = vb.nx * blockDim.x;
    // FP64 draws, spread over the FP64 pipes, of which each SM has one per four warps: every CTA takes an equal share of
    // the rows, and CTAs that follow one another on an SM take theirs in different warps.  16 x 2000 rows: 18.6 us (26 us
    // when the first CTAs of a chain did all of them, 23 us when the first warp of every CTA did)
    const int turn = vb.x + vb.y * vb.nx, lin = (threadIdx.x + 32 * (turn + turn / 152)) & 255;
    double sd = 0.0;
    for (int i = lin * vb.nx + vb.x; i < D.naind; i += stride) {
        if (sd == 0.0) sd = sqrt(S->vare);
        CRng R;
        crng_site(R, D, c, rep, i, P_RA);
        store_ra(D, c, i, d_rnorm(0.0, sd, R));
    }
    if (!S->keep) return;
    const int m = D.method;
    const bool locus = m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B;
    for (int64_t j = t0; j < D.p; j += (int64_t)POST_AHEAD * stride) {
        double g[POST_AHEAD], gs[POST_AHEAD], v[POST_AHEAD], vs[POST_AHEAD];
        size_t at[POST_AHEAD];
        uint32_t cnt[POST_AHEAD];
#pragma unroll
        for (int q = 0; q < POST_AHEAD; ++q) {
            const int64_t jq = j + (int64_t)q * stride;
            const bool in = jq < D.p;
            const size_t o = (size_t)c * D.p + (in ? jq : j);
            g[q] = D.g[o];
            gs[q] = D.gstore[o];
            v[q] = locus ? D.vara_s[o] : 0.0;
            vs[q] = locus ? D.vara_sstore[o] : 0.0;
            at[q] = m != SODAGPU_BAYES_A ? o * D.nmix + (D.cls[o] - 1) : 0;
        }
#pragma unroll
        for (int q = 0; q < POST_AHEAD; ++q) cnt[q] = m != SODAGPU_BAYES_A ? D.indist[at[q]] : 0u;
#pragma unroll
        for (int q = 0; q < POST_AHEAD; ++q) {
            const int64_t jq = j + (int64_t)q * stride;
            if (jq >= D.p) break;
            const size_t o = (size_t)c * D.p + jq;
            D.gstore[o] = gs[q] + g[q];
            if (m != SODAGPU_BAYES_A) D.indist[at[q]] = cnt[q] + 1u;
            if (locus) D.vara_sstore[o] = vs[q] + v[q];
        }
    }
}

__global__ void __launch_bounds__(256) k_post(Dev D)
{
    post_body(D, vb_native());
}


// compute_residuals (utilities.f90:609-614), every `recal` iterations.  The two kernels are launched every
// iteration (the iteration is a captured graph) and return at once on the others, so their grids hold
// RECAL_CTAS CTAs that walk the (rows, column split, chain) tiles: one CTA a tile cost 302 us an iteration in
// CTA launches alone at n = 50,000 and 16 chains.
//
// A tile's SNPs with an effect are gathered in shared memory, 256 at a time and in order, so that the loads of their
// codes do not wait for one another: with the effect and the centring table looked up for each SNP by each thread, the
// loop was a chain of three loads, whose rate was the number of resident CTAs (and these are half of what
// an SM holds).  An iteration that recalibrates takes longer by, p = 20,000: n = 50,000, one chain of BayesA: 3.7 ms;
// n = 50,000, 4 chains, half of the effects zero: 7.1 ms; n = 20,000, 16 chains: 8.9 ms (9.7, 32.2 and 41.0 ms; 3.9, 14.9
// and 24.0 ms with one CTA a tile).
constexpr int RECAL_CHUNK = 256;

__device__ __forceinline__ void recal_partial_body(const Dev &D, const VB &vb, int force)
{
    __shared__ double s_x[RECAL_CHUNK][4];   // the values of codes 0, 1, 2 and the effect
    __shared__ int s_k[RECAL_CHUNK], s_cnt[RECAL_CHUNK / 32];
    tc::pdl_trigger();
    tc::pdl_wait();
    const int rep = cur_rep(D);
    if (!force && (D.recal <= 0 || rep % D.recal != 0)) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles = (D.n + 255) / 256, total = tiles * RECAL_SPLIT * D.chains;
    const int per = (D.p + RECAL_SPLIT - 1) / RECAL_SPLIT;
    for (int t = vb.x; t < total; t += vb.nx) {
        const int c = t / (tiles * RECAL_SPLIT), split = (t / tiles) % RECAL_SPLIT;
        const int i = (t % tiles) * 256 + tid;
        const int k0 = split * per, k1 = min(D.p, k0 + per);
        double acc = 0.0;
        const double *g = D.g + (size_t)c * D.p;
        const int8_t *col = D.G + min(i, D.n - 1);
        for (int c0 = k0; c0 < k1; c0 += RECAL_CHUNK) {
            const int k = c0 + tid;
            const double gj = k < k1 ? g[D.perm[k]] : 0.0;
            const unsigned in = __ballot_sync(0xffffffffu, gj != 0.0);
            if (lane == 0) s_cnt[warp] = __popc(in);
            __syncthreads();   // also: every use of the previous chunk is done
            int at = 0, m = 0;
#pragma unroll
            for (int w = 0; w < RECAL_CHUNK / 32; ++w) {
                at += w < warp ? s_cnt[w] : 0;
                m += s_cnt[w];
            }
            if (gj != 0.0) {
                at += __popc(in & ((1u << lane) - 1u));
                s_k[at] = k;
#pragma unroll
                for (int q = 0; q < 3; ++q) s_x[at][q] = D.xv[(size_t)k * 4 + q];
                s_x[at][3] = gj;
            }
            __syncthreads();
#pragma unroll 8
            for (int q = 0; q < m; ++q) acc = acc + s_x[q][col[(size_t)s_k[q] * D.ldx]] * s_x[q][3];
        }
        if (i < D.n) D.recal_part[((size_t)c * RECAL_SPLIT + split) * D.ldr + i] = acc;
    }
}

__global__ void __launch_bounds__(256) k_recal_partial(Dev D, int force)
{
    recal_partial_body(D, vb_native(), force);
}


__device__ __forceinline__ void recal_apply_body(const Dev &D, const VB &vb, int force, int mu_slot)
{
    tc::pdl_trigger();
    tc::pdl_wait();
    const int rep = cur_rep(D);
    if (!force && (D.recal <= 0 || rep % D.recal != 0)) return;
    const int tiles = (D.n + 255) / 256, total = tiles * D.chains;
    const int slot = mu_slot >= 0 ? mu_slot : (rep & 1);
    for (int t = vb.x; t < total; t += vb.nx) {
        const int c = t / tiles, i = (t % tiles) * 256 + threadIdx.x;
        if (i >= D.n) continue;
        double d = 0.0;
        for (int s = 0; s < RECAL_SPLIT; ++s) d = d + D.recal_part[((size_t)c * RECAL_SPLIT + s) * D.ldr + i];
        store_r(D, c, i, D.y[i] - d - D.scal[c].mu[slot]);
    }
}

__global__ void __launch_bounds__(256) k_recal_apply(Dev D, int force, int mu_slot)
{
    recal_apply_body(D, vb_native(), force, mu_slot);
}


// ---------------------------------------------------------------------------
// chain initialisation (models.f90:56-128)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_init_chain(Dev D, double vara0, double scale_va0)
{
    __shared__ double sh[33];
    const int c = blockIdx.x, m = D.method, ng = D.ngroup, nm = D.nmix;
    ChainScal *S = &D.scal[c];
    const double nn = (double)D.n;
    double sy = 0.0;
    for (int i = threadIdx.x; i < D.n; i += blockDim.x) sy += D.y[i];
    sy = block_sum(sy, sh);
    const double mu = sy / nn;
    double rr = 0.0, vy = 0.0;
    for (int i = threadIdx.x; i < D.n; i += blockDim.x) {
        const double v = (D.y[i] - 0.0) - mu;
        store_r(D, c, i, v);
        rr += v * v;
        vy += (D.y[i] - mu) * (D.y[i] - mu);
    }
    rr = block_sum(rr, sh);
    vy = block_sum(vy, sh);
    if (threadIdx.x == 0) {
        S->mu[0] = mu;
        S->mu[1] = mu;
        S->scale_va = scale_va0;
        S->vara = vara0;
        S->counter = 0;
        S->mu_ticket = 0;
        S->keep = 0;
        S->err = 0;
        S->included = 0;
        S->mu_store = S->vare_store = S->vara_store = S->included_store = 0.0;
        for (int e = 0; e < MAXGM; ++e) {
            S->snpstore[e] = S->pstore[e] = S->varstore[e] = 0.0;
            S->varindist[e] = 0.0;
            S->snpindist[e] = 0;
            S->p[e] = 0.0;
            S->log_p[e] = 0.0;
        }
        if (m != SODAGPU_BAYES_A) {
            if (m == SODAGPU_BAYES_B || m == SODAGPU_BAYES_C) {
                for (int i = 0; i < ng; ++i) {
                    S->p[i] = D.pizero;
                    S->p[i + ng] = 1.0 - D.pizero;
                }
            } else {
                for (int i = 0; i < ng; ++i) {
                    S->p[i] = 0.5;
                    double s = 0.0;
                    for (int j = 1; j < nm; ++j) S->p[i + j * ng] = 1.0 / D.mix[j];
                    for (int j = 1; j < nm; ++j) s = s + S->p[i + j * ng];
                    for (int j = 1; j < nm; ++j) S->p[i + j * ng] = 0.5 * S->p[i + j * ng] / s;
                }
            }
        }
        if (D.df_va <= 0.0) {
            const double vary = vy / (nn - 1.0);
            if (m == SODAGPU_BAYES_A) {
                S->vara = S->scale_va * vary / D.p;
            } else if (m == SODAGPU_BAYES_B) {
                S->vara = S->scale_va * vary / D.p / S->p[ng];
            } else {
                for (int i = 0; i < ng; ++i) {
                    double dp = 0.0;
                    for (int j = 0; j < nm; ++j) dp = dp + S->p[i + j * ng] * D.mix[j];
                    S->vara = S->vara + dp;
                }
                S->vara = S->scale_va * vary / D.p / S->vara;
            }
            S->scale_va = 0.0;
        } else {
            S->vara = S->scale_va * D.df_va / (D.df_va + 2.0);
        }
        for (int j = 0; j < nm; ++j) S->gp[j] = D.mix[j] * S->vara;
        const double scale = (rr + D.scale_ve * D.df_ve) / (nn + D.df_ve);
        CRng R;
        crng_site(R, D, c, 0, 0, P_VARE);
        int err = 0;
        S->vare = d_rscinvchi2(nn + D.df_ve, scale, R, &err);
        if (err) flag_err(D, 1);
        if (m != SODAGPU_BAYES_A) {
            for (int e = 0; e < ng * nm; ++e) S->log_p[e] = log(S->p[e]);
            for (int j = 1; j < nm; ++j) S->vare_gp[j] = S->vare / S->gp[j];
        }
    }
    __syncthreads();
    const double sd = sqrt(S->vare);
    for (int i = threadIdx.x; i < D.bs; i += blockDim.x) {
        double v = 0.0;
        if (i < D.naind) {
            CRng R;
            crng_site(R, D, c, 0, i, P_RA);
            v = d_rnorm(0.0, sd, R);
        }
        store_ra(D, c, i, v);
    }
}

__global__ void __launch_bounds__(256) k_init_snp(Dev D)
{
    const int c = blockIdx.y;
    const double vara = D.scal[c].vara;
    const int m = D.method;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < D.p; j += gridDim.x * blockDim.x) {
        const size_t o = (size_t)c * D.p + j;
        D.g[o] = 0.0;
        D.cls[o] = m == SODAGPU_BAYES_A ? 1 : 2;
        D.vara_s[o] = (m == SODAGPU_BAYES_A || m == SODAGPU_BAYES_B) ? vara : 0.0;
        D.gstore[o] = 0.0;
        D.vara_sstore[o] = 0.0;
        for (int q = 0; q < D.nmix; ++q) D.indist[o * D.nmix + q] = 0u;
    }
}

// ---------------------------------------------------------------------------
// host-side launch helpers
// ---------------------------------------------------------------------------
struct ProfScope {
    ProfHook *h;
    cudaStream_t st;
    int slot;
    ProfScope(ProfHook *h_, cudaStream_t st_, int cls) : h(h_), st(st_), slot(-1)
    {
        if (h && h->n < h->cap) {
            slot = h->n++;
            h->cls[slot] = cls;
            cudaEventRecord(h->ev[2 * slot], st);
        }
    }
    ~ProfScope()
    {
        if (slot >= 0) cudaEventRecord(h->ev[2 * slot + 1], st);
    }
};

// Launch with programmatic stream serialization: the kernel may start while
// the previous one in the stream finishes; it calls griddepcontrol.wait before
// reading that kernel's results.
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
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

// Tensor-core subset: rhs tiles of 128 SNPs x K splits (one wave of one CTA
// per SM), then the update (row tiles of r on the tensor cores, ra tiles on
// the FP32 cores; two CTAs per SM).
template <int CT>
static cudaError_t launch_block_tc(const Dev &D, int b, int nblk_snps, int sm_count, const TcMaps *maps,
                                   cudaStream_t st, ProfHook *prof, bool rhs_only)
{
    const int mtiles = (nblk_snps + TC_TM - 1) / TC_TM;
    const int nrhs = maps->h_rtab[(size_t)b * D.tstride + mtiles];
    cudaError_t e;
    {
        ProfScope ps(prof, st, PROF_RHS);
        e = launch_pdl(k_rhs_tc<CT>, dim3(nrhs), dim3(TC_THREADS), RhsTc<CT>::SMEM, st, maps->rsp, maps->usp,
                       maps->rasp, D, b);
    }
    if (e != cudaSuccess) return e;
    {
        const int span = mtiles * TC_TM;
        ProfScope ps(prof, st, PROF_DRAW);
        e = launch_pdl(k_draw<SODAGPU_FP8, CT, true>, dim3((span * CT + 255) / 256), dim3(256), 0, st, D, b, 0, span);
    }
    if (e != cudaSuccess || rhs_only) return e != cudaSuccess ? e : cudaGetLastError();
    {
        ProfScope ps(prof, st, PROF_UPDATE);
        e = launch_pdl(k_update_tc<CT>, dim3(std::min(sm_count, TV_MAXG)), dim3(TV_THREADS), UpdTc<CT>::SMEM, st,
                       maps->d, maps->usp64, D, b);

    }
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

// K splits of a subset's rhs tiles: `ctas` CTAs in all, but no more than give every split the same number of
// genotype stages (a split with one stage fewer only waits for the others).
static int rhs_splits(int ctas, int mtiles, int nst)
{
    int ks = std::max(1, std::min({ctas / std::max(1, mtiles), RHS_KSPLIT_MAX_CC, nst}));
    const int per = (nst + ks - 1) / ks;
    return (nst + per - 1) / per;
}

template <int MODE, int CT>
static cudaError_t launch_block(const Dev &D, int b, int nblk_snps, int sm_count, const TcMaps *maps, cudaStream_t st,
                               ProfHook *prof, bool rhs_only)
{
    if constexpr (MODE == SODAGPU_FP8 && CT >= 4) {
        if (D.tc) return launch_block_tc<CT>(D, b, nblk_snps, sm_count, maps, st, prof, rhs_only);
    }
    constexpr int MTS = 8 * SptOf<CT>::v;
    const int mtiles = (nblk_snps + MTS - 1) / MTS;
    const int nst = (D.ldx + RhsCfg<MODE>::KST - 1) / RhsCfg<MODE>::KST;
    const int ks = rhs_splits(sm_count * rhs_per_sm<MODE, CT>(), mtiles, nst);
    cudaError_t e;
    {
        ProfScope ps(prof, st, PROF_RHS);
        e = launch_pdl(k_rhs<MODE, CT>, dim3(mtiles * ks), dim3(256), rhs_smem_bytes<MODE, CT>(), st, D, b, ks);
    }
    if (e != cudaSuccess) return e;
    {
        ProfScope ps(prof, st, PROF_DRAW);
        constexpr int NT = DrawThreads<CT, false>::v;
        e = launch_pdl(k_draw<MODE, CT, false>, dim3((nblk_snps * CT + NT - 1) / NT), dim3(NT), 0, st, D, b, ks,
                       nblk_snps);
    }
    if (e != cudaSuccess || rhs_only) return e != cudaSuccess ? e : cudaGetLastError();
    const int ntile = D.nr_ctas + (D.bs + UT - 1) / UT;
    {
        ProfScope ps(prof, st, PROF_UPDATE);
        e = launch_pdl(k_update<MODE, CT>, dim3(ntile), dim3(32 * UpdWarps<MODE, CT>::v),
                       update_smem_bytes_ct<MODE, CT>(D.bs), st, D, b);
    }
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_block_mode(const Dev &D, int b, int nsnp, int sm_count, const TcMaps *maps, cudaStream_t st,
                                    ProfHook *prof, bool rhs_only = false)
{
    switch (D.chains) {
    case 1: return launch_block<MODE, 1>(D, b, nsnp, sm_count, maps, st, prof, rhs_only);
    case 2: return launch_block<MODE, 2>(D, b, nsnp, sm_count, maps, st, prof, rhs_only);
    case 4: return launch_block<MODE, 4>(D, b, nsnp, sm_count, maps, st, prof, rhs_only);
    case 8: return launch_block<MODE, 8>(D, b, nsnp, sm_count, maps, st, prof, rhs_only);
    case 16: return launch_block<MODE, 16>(D, b, nsnp, sm_count, maps, st, prof, rhs_only);
    default: return cudaErrorInvalidValue;
    }
}

int sweep_chain_count_supported(int c) { return c == 1 || c == 2 || c == 4 || c == 8 || c == 16; }

// Every kernel of an iteration asks for the largest shared-memory carveout,
// so that consecutive kernels never wait for the SMs to repartition L1 and
// shared memory (microseconds per kernel boundary otherwise).
template <typename K>
static cudaError_t max_carveout(K *kern)
{
    return cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
}

template <int MODE, bool TC>
static cudaError_t carve_draw()
{
    cudaError_t e = cudaSuccess;
    if constexpr (!TC) {
        e = max_carveout(k_draw<MODE, 1, false>);
        if (e == cudaSuccess) e = max_carveout(k_draw<MODE, 2, false>);
    }
    if (e == cudaSuccess) e = max_carveout(k_draw<MODE, 4, TC>);
    if (e == cudaSuccess) e = max_carveout(k_draw<MODE, 8, TC>);
    if (e == cudaSuccess) e = max_carveout(k_draw<MODE, 16, TC>);
    return e;
}

static cudaError_t carve_all()
{
    cudaError_t e = carve_draw<SODAGPU_FP64, false>();
    if (e == cudaSuccess) e = carve_draw<SODAGPU_FP32, false>();
    if (e == cudaSuccess) e = carve_draw<SODAGPU_FP8, false>();
    if (e == cudaSuccess) e = carve_draw<SODAGPU_FP8, true>();
    if (e == cudaSuccess) e = max_carveout(k_iter_begin);
    if (e == cudaSuccess) e = max_carveout(k_mu_partial);
    if (e == cudaSuccess) e = max_carveout(k_mu_apply);
    if (e == cudaSuccess) e = max_carveout(k_skipped_pre);
    if (e == cudaSuccess) e = max_carveout(k_skipped_spec);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_skipped_spec, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM_MAX);
    if (e == cudaSuccess) e = max_carveout(k_skipped<128>);
    if (e == cudaSuccess) e = max_carveout(k_skipped<512>);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_skipped<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM_MAX);
    if (e == cudaSuccess) e = max_carveout(k_stats);
    if (e == cudaSuccess) e = max_carveout(k_hyper);
    if (e == cudaSuccess) e = max_carveout(k_post);
    if (e == cudaSuccess) e = max_carveout(k_recal_partial);
    if (e == cudaSuccess) e = max_carveout(k_recal_apply);
    return e;
}

template <int MODE, int CT>
static cudaError_t set_update_smem(int bs)
{
    cudaError_t e = cudaFuncSetAttribute(k_update<MODE, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)update_smem_bytes_ct<MODE, CT>(bs));
    return e == cudaSuccess ? max_carveout(k_update<MODE, CT>) : e;
}

template <int MODE>
static cudaError_t set_update_smem_mode(int bs)
{
    cudaError_t e = set_update_smem<MODE, 1>(bs);
    if (e == cudaSuccess) e = set_update_smem<MODE, 2>(bs);
    if (e == cudaSuccess) e = set_update_smem<MODE, 4>(bs);
    if (e == cudaSuccess) e = set_update_smem<MODE, 8>(bs);
    if (e == cudaSuccess) e = set_update_smem<MODE, 16>(bs);
    return e;
}

template <int MODE, int CT>
static cudaError_t set_rhs_smem()
{
    cudaError_t e = cudaFuncSetAttribute(k_rhs<MODE, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)rhs_smem_bytes<MODE, CT>());
    return e == cudaSuccess ? max_carveout(k_rhs<MODE, CT>) : e;
}

template <int MODE>
static cudaError_t set_rhs_smem_mode()
{
    cudaError_t e = set_rhs_smem<MODE, 1>();
    if (e == cudaSuccess) e = set_rhs_smem<MODE, 2>();
    if (e == cudaSuccess) e = set_rhs_smem<MODE, 4>();
    if (e == cudaSuccess) e = set_rhs_smem<MODE, 8>();
    if (e == cudaSuccess) e = set_rhs_smem<MODE, 16>();
    return e;
}

template <int CT>
static cudaError_t set_tc_smem()
{
    cudaError_t e = cudaFuncSetAttribute(k_rhs_tc<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)RhsTc<CT>::SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_update_tc<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)UpdTc<CT>::SMEM);
    if (e == cudaSuccess) e = max_carveout(k_rhs_tc<CT>);
    if (e == cudaSuccess) e = max_carveout(k_update_tc<CT>);

    return e;
}

int sweep_tc_supported(int precision, int chains, int bs)
{
    return precision == SODAGPU_FP8 && (chains == 4 || chains == 8 || chains == 16) && bs <= TV_MAXQ * TV_K;
}

int sweep_tc_update_tiles(int n) { return (n + TV_N - 1) / TV_N; }

size_t sweep_tc_vpart_floats(int n, int bs, int chains, int sm_count)
{
    const size_t slots = (size_t)sweep_tc_update_tiles(n) + (size_t)((bs + TV_N - 1) / TV_N) + (size_t)sm_count;
    return slots * (size_t)chains * TV_N;
}

int sweep_tc_rows(int chains) { return ((3 * chains + 15) / 16) * 16; }

__global__ void __launch_bounds__(256) k_tc_prepare(int8_t *G, Dev D, uint16_t *usp)
{
    for (int k = blockIdx.x; k < D.p; k += gridDim.x) {
        const double inv = D.xv[(size_t)k * 4 + 3];
        const double sc = inv != 0.0 ? 1.0 / inv : 1.0;
        const int len = D.ulen[k];
        const int64_t off = D.uoff[k];
        for (int i = threadIdx.x; i < D.ldu; i += blockDim.x) {
            const double v = i < len ? D.U64[off + i] * sc : 0.0;
            const __nv_bfloat16 h = __double2bfloat16(v);
            const double r1 = v - (double)__bfloat162float(h);
            const __nv_bfloat16 m = __double2bfloat16(r1);
            const __nv_bfloat16 l = __double2bfloat16(r1 - (double)__bfloat162float(m));
            usp[(size_t)k * D.ldu + i] = __bfloat16_as_ushort(h);
            usp[((size_t)D.p + k) * D.ldu + i] = __bfloat16_as_ushort(m);
            usp[((size_t)2 * D.p + k) * D.ldu + i] = __bfloat16_as_ushort(l);
        }
        if (inv == 0.0)
            for (int i = threadIdx.x; i < D.ldx; i += blockDim.x) G[(size_t)k * D.ldx + i] = 0;
    }
}

cudaError_t sweep_tc_prepare(int8_t *G, const Dev &D, cudaStream_t st)
{
    if (!D.usp || D.ldu <= 0) return cudaErrorInvalidValue;
    k_tc_prepare<<<std::min(D.p, 4096), 256, 0, st>>>(G, D, const_cast<uint16_t *>(D.usp));
    return cudaGetLastError();
}

int sweep_tc_code_blocks(const int *blk_sizes, int nb, int32_t *qoff)
{
    int tot = 0;
    for (int b = 0; b < nb; ++b) {
        qoff[b] = tot;
        tot += (blk_sizes[b] + TC_TM - 1) / TC_TM;
    }
    qoff[nb] = tot;
    return tot;
}

// Packed code block (q2, t): positions 128 (q2 - qoff[b]) .. of subset b x individuals 256 t .. (see
// TC_PACKED_BLOCK); positions past the subset and individuals past n hold 0.  One thread per 16-byte word
// (group g of 64 individuals, position k): four 16-byte loads of the position's column of G (64 bytes never
// straddle ldx, a multiple of 128), each folded into one 32-bit word.
__global__ void __launch_bounds__(256) k_tile_codes(const int8_t *G, Dev D, uint8_t *Gt, long long nblocks)
{
    constexpr int WORDS = TC_PACKED_BLOCK / 16;
    const long long total = nblocks * WORDS;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long blk = idx / WORDS;
        const int wi = (int)(idx - blk * WORDS), g = wi / TC_TM, k = wi - g * TC_TM;
        const int q2 = (int)(blk / D.nvt), t = (int)(blk - (long long)q2 * D.nvt);
        int lo = 0, hi = D.nb - 1;   // the subset: last b with qoff[b] <= q2
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (D.qoff[mid] <= q2) lo = mid;
            else hi = mid - 1;
        }
        const int ls = D.blk_ls[lo], N = D.blk_ls[lo + 1] - ls, r = (q2 - D.qoff[lo]) * TC_TM + k;
        const int i0 = t * TV_N + 64 * g;
        uint32_t out[4] = {0u, 0u, 0u, 0u};
        if (r < N && i0 + 64 <= D.ldx) {
            const uint4 *src = reinterpret_cast<const uint4 *>(G + (size_t)(ls + r) * D.ldx + i0);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const uint4 v = src[w];   // individuals 16 w + 4 b + j: byte j of word b
                out[w] = (v.x & 0x03030303u) | ((v.y & 0x03030303u) << 2) | ((v.z & 0x03030303u) << 4) |
                         ((v.w & 0x03030303u) << 6);
            }
        }
        *reinterpret_cast<uint4 *>(Gt + blk * TC_PACKED_BLOCK + (size_t)wi * 16) =
            make_uint4(out[0], out[1], out[2], out[3]);
    }
}

// The individual-major copy: one thread per (block, stage, individual) writes
// that individual's 16 bytes, reading its 64 codes of the stage one position
// (column of G) at a time; a warp's 32 individuals read 32 consecutive bytes
// of each column.
__global__ void __launch_bounds__(256) k_tile_codes_ind(const int8_t *G, Dev D, uint8_t *Gu, long long nblocks)
{
    constexpr int WORDS = TC_PACKED_BLOCK / 16;   // 2 stages x 256 individuals
    const long long total = nblocks * WORDS;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long blk = idx / WORDS;
        const int wi = (int)(idx - blk * WORDS), st = wi / TV_N, il = wi - st * TV_N;
        const int q2 = (int)(blk / D.nvt), t = (int)(blk - (long long)q2 * D.nvt);
        int lo = 0, hi = D.nb - 1;   // the subset: last b with qoff[b] <= q2
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (D.qoff[mid] <= q2) lo = mid;
            else hi = mid - 1;
        }
        const int ls = D.blk_ls[lo], N = D.blk_ls[lo + 1] - ls, r0 = (q2 - D.qoff[lo]) * TC_TM + st * TV_K;
        const int i = t * TV_N + il;
        uint32_t out[4] = {0u, 0u, 0u, 0u};
        if (i < D.n) {
            for (int k = 0; k < TV_K && r0 + k < N; ++k) {
                const uint32_t c = (uint32_t)G[(size_t)(ls + r0 + k) * D.ldx + i] & 3u;
                out[k >> 4] |= c << (8 * (k & 3) + 2 * ((k >> 2) & 3));
            }
        }
        *reinterpret_cast<uint4 *>(Gu + blk * TC_PACKED_BLOCK + (size_t)wi * 16) =
            make_uint4(out[0], out[1], out[2], out[3]);
    }
}

cudaError_t sweep_tc_tile_codes(const int8_t *G, const Dev &D, uint8_t *Gt, uint8_t *Gu, long long nblocks,
                                int sm_count, cudaStream_t st)
{
    if (!Gt || !D.qoff || nblocks <= 0) return cudaErrorInvalidValue;
    const long long words = nblocks * (TC_PACKED_BLOCK / 16);
    const long long grid = std::min<long long>((words + 255) / 256, 16LL * sm_count);
    k_tile_codes<<<(unsigned)grid, 256, 0, st>>>(G, D, Gt, nblocks);
    if (Gu) k_tile_codes_ind<<<(unsigned)grid, 256, 0, st>>>(G, D, Gu, nblocks);
    return cudaGetLastError();
}

int sweep_tc_table_stride(int bs) { return (bs + TC_TM - 1) / TC_TM + 1; }

void sweep_tc_tables(const int *blk_sizes, int nb, int bs, int ldx, int sm_count, int32_t *rtab)
{
    const int stride = sweep_tc_table_stride(bs);
    const int nst = ldx / TC_KC;
    for (int b = 0; b < nb; ++b) {
        const int N = blk_sizes[b], tiles = (N + TC_TM - 1) / TC_TM;
        int32_t *rt = rtab + (size_t)b * stride;
        // K splits in proportion to each tile's MMAs (8 per genotype stage, 4 per U stage), largest
        // remainders first, so that the CTAs (one per SM, all of them) get equal MMA work
        std::vector<long long> w(tiles);
        std::vector<int> ks(tiles), cap(tiles);
        long long W = 0;
        for (int m = 0; m < tiles; ++m) {
            const int T = rhs_tc_stages(nst, N, m, true, nullptr);
            w[m] = 8LL * nst + 4LL * (T - nst);
            cap[m] = std::min(RHS_KSPLIT_MAX, T);
            W += w[m];
        }
        int total = 0;
        for (int m = 0; m < tiles; ++m) {
            ks[m] = std::max(1, std::min(cap[m], (int)(((long long)sm_count * w[m]) / W)));
            total += ks[m];
        }
        while (total < sm_count) {
            int best = -1;
            double bf = -1.0;
            for (int m = 0; m < tiles; ++m) {
                if (ks[m] >= cap[m]) continue;
                const double f = (double)sm_count * (double)w[m] / (double)W - ks[m];
                if (f > bf) {
                    bf = f;
                    best = m;
                }
            }
            if (best < 0) break;
            ++ks[best];
            ++total;
        }
        int acc = 0;
        for (int m = 0; m < tiles; ++m) {
            rt[m] = acc;
            acc += ks[m];
        }
        rt[tiles] = acc;
    }
}

// Raises the dynamic shared-memory limits of the rhs and update kernels (the
// update's for the largest subset size asked for so far in this process:
// the limit is per kernel, and every job's launches must stay within it).
cudaError_t sweep_prepare(int bs)
{
    static int s_max_bs = 0;
    if (bs < s_max_bs) bs = s_max_bs;
    s_max_bs = bs;
    {
        cudaError_t e = carve_all();
        if (e == cudaSuccess) e = set_tc_smem<4>();
        if (e == cudaSuccess) e = set_tc_smem<8>();
        if (e == cudaSuccess) e = set_tc_smem<16>();
        if (e != cudaSuccess) return e;
    }
    cudaError_t e = set_rhs_smem_mode<SODAGPU_FP64>();
    if (e == cudaSuccess) e = set_rhs_smem_mode<SODAGPU_FP32>();
    if (e == cudaSuccess) e = set_rhs_smem_mode<SODAGPU_FP8>();
    if (e != cudaSuccess) return e;
    if (update_smem_bytes_ct<SODAGPU_FP64, 16>(bs) > 220 * 1024) return cudaErrorInvalidValue;
    e = set_update_smem_mode<SODAGPU_FP64>(bs);
    if (e == cudaSuccess) e = set_update_smem_mode<SODAGPU_FP32>(bs);
    if (e == cudaSuccess) e = set_update_smem_mode<SODAGPU_FP8>(bs);
    return e;
}

// CTAs of k_post per chain, and of the recalibration kernels over all of their tiles.
static int post_grid(const Dev &D, int sm_count)
{
    return std::max(1, std::min((D.p + 255) / 256, 4 * sm_count));
}
static int recal_grid(const Dev &D, int splits)
{
    return (int)std::min<long long>((long long)((D.n + 255) / 256) * splits * D.chains, RECAL_CTAS);
}

cudaError_t sweep_enqueue_iteration(const Dev &D, const int *blk_sizes, int sm_count, const TcMaps *maps,
                                    cudaStream_t st, ProfHook *prof)
{
    if (D.tc && !maps) return cudaErrorInvalidValue;
    const int C = D.chains;
    cudaError_t e = cudaSuccess;
    {
        ProfScope ps(prof, st, PROF_MU);
        k_iter_begin<<<1, 1, 0, st>>>(D);
        e = launch_pdl(k_mu_partial, dim3(mu_grid(D.n), C), dim3(MU_THREADS), 0, st, D);
        if (e == cudaSuccess) e = launch_pdl(k_mu_apply, dim3(mu_grid(D.n), C), dim3(MU_THREADS), 0, st, D);
        if (e != cudaSuccess) return e;
    }
    for (int b = 0; b < D.nb; ++b) {
        const int nsnp = blk_sizes[b];
        if (D.precision == SODAGPU_FP64) e = launch_block_mode<SODAGPU_FP64>(D, b, nsnp, sm_count, maps, st, prof);
        else if (D.precision == SODAGPU_FP32)
            e = launch_block_mode<SODAGPU_FP32>(D, b, nsnp, sm_count, maps, st, prof);
        else e = launch_block_mode<SODAGPU_FP8>(D, b, nsnp, sm_count, maps, st, prof);
        if (e != cudaSuccess) return e;
    }
    {
        ProfScope ps(prof, st, PROF_OTHER);
        for (int t0 = 0; t0 < D.nskipped; t0 += SS_CHUNK) {
            const int cnt = std::min(SS_CHUNK, D.nskipped - t0);
            const size_t sm = skipped_smem(D.n);
            e = cudaMemsetAsync(D.ssdense, 0, sizeof(int32_t) * C, st);
            if (e != cudaSuccess) return e;
            k_skipped_pre<<<dim3((cnt + 63) / 64, C), 64, 0, st>>>(D, t0, cnt);
            if (sm) {   // each chain goes through one of the two
                k_skipped_spec<<<SS_CTAS * C, 128, sm, st>>>(D, t0, cnt);
                k_skipped<128><<<C, 128, sm, st>>>(D, t0, cnt);
            } else {
                k_skipped<512><<<C, 512, 0, st>>>(D, t0, cnt);
            }
        }
        e = launch_pdl(k_stats, dim3(NSTAT + mu_grid(D.n), C), dim3(256), 0, st, D);
        if (e == cudaSuccess) e = launch_pdl(k_hyper, dim3(C), dim3(HYPER_THREADS), 0, st, D);
        if (e == cudaSuccess) e = launch_pdl(k_post, dim3(post_grid(D, sm_count), C), dim3(256), 0, st, D);
        if (e == cudaSuccess) e = launch_pdl(k_recal_partial, dim3(recal_grid(D, RECAL_SPLIT)), dim3(256), 0, st, D, 0);
        if (e == cudaSuccess) e = launch_pdl(k_recal_apply, dim3(recal_grid(D, 1)), dim3(256), 0, st, D, 0, -1);
    }
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t sweep_enqueue_init(const Dev &D, double vara0, double scale_va0, int sm_count, cudaStream_t st)
{
    k_init_chain<<<D.chains, 256, 0, st>>>(D, vara0, scale_va0);
    const int pgrid = (D.p + 255) / 256 < 4 * sm_count ? (D.p + 255) / 256 : 4 * sm_count;
    k_init_snp<<<dim3(pgrid > 0 ? pgrid : 1, D.chains), 256, 0, st>>>(D);
    return cudaGetLastError();
}

cudaError_t sweep_enqueue_subset(const Dev &D, int b, int nsnp, int sm_count, const TcMaps *maps, cudaStream_t st,
                                 bool rhs_only)
{
    if (D.tc && !maps) return cudaErrorInvalidValue;
    if (D.precision == SODAGPU_FP64) return launch_block_mode<SODAGPU_FP64>(D, b, nsnp, sm_count, maps, st, nullptr, rhs_only);
    if (D.precision == SODAGPU_FP32) return launch_block_mode<SODAGPU_FP32>(D, b, nsnp, sm_count, maps, st, nullptr, rhs_only);
    return launch_block_mode<SODAGPU_FP8>(D, b, nsnp, sm_count, maps, st, nullptr, rhs_only);
}

// ---------------------------------------------------------------------------
// Loading one chain's state (the inverse of sodagpu_get_state): the residuals
// with every copy derived from them (FP32 copy or bf16 split, and the 128-row
// partial sums of r that the FP8 centring reads), the per-SNP state, and the
// chain scalars with the tables the draws read (models.f90:198-199, 330-338).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(ROW_THREADS) k_set_rows(Dev D, int c, const double *r)
{
    __shared__ double sh[33];
    const int i = blockIdx.x * ROW_TILE + threadIdx.x;
    double v = 0.0;
    if (i < D.n) {
        v = r[i];
        store_r(D, c, i, v);
    }
    const double t = block_sum(v, sh);
    if (threadIdx.x == 0) D.rsum[(size_t)c * D.nr_ctas + blockIdx.x] = t;
}

__global__ void __launch_bounds__(256) k_set_snps(Dev D, int c, const double *g, const int32_t *cls, const double *vs,
                                                  const double *ra, const double *pi, double mu, double vare,
                                                  double vara, int included)
{
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (int j = t0; j < D.p; j += stride) {
        const size_t o = (size_t)c * D.p + j;
        D.g[o] = g[j];
        D.cls[o] = cls[j];
        D.vara_s[o] = vs[j];
    }
    for (int i = t0; i < D.bs; i += stride) store_ra(D, c, i, i < D.naind ? ra[i] : 0.0);
    if (t0 == 0) {
        ChainScal *S = &D.scal[c];
        S->mu[0] = S->mu[1] = mu;
        S->vare = vare;
        S->vara = vara;
        S->included = included;
        const int ngm = D.ngroup * D.nmix;
        if (pi)
            for (int e = 0; e < ngm; ++e) S->p[e] = pi[e];
        for (int j = 0; j < D.nmix; ++j) S->gp[j] = D.mix[j] * vara;
        if (D.method != SODAGPU_BAYES_A) {
            for (int e = 0; e < ngm; ++e) S->log_p[e] = log(S->p[e]);
            for (int j = 1; j < D.nmix; ++j) S->vare_gp[j] = vare / S->gp[j];
        }
    }
}

cudaError_t sweep_set_state(const Dev &D, int c, const double *g, const int32_t *cls, const double *vs,
                            const double *r, const double *ra, const double *pi, double mu, double vare, double vara,
                            int included, cudaStream_t st)
{
    k_set_rows<<<D.nr_ctas, ROW_THREADS, 0, st>>>(D, c, r);
    const int grid = std::max(1, std::min((D.p + 255) / 256, 1024));
    k_set_snps<<<grid, 256, 0, st>>>(D, c, g, cls, vs, ra, pi, mu, vare, vara, included);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Reading one chain's state and starting a run: one launch in place of a copy per array.  A copy of a few hundred
// bytes to the host takes 11 us, and one chain's state was seven of them (one of 100 KB for four scalars): 87 us at
// p = 20,000, 48 us through one kernel that writes to page-locked host memory, which the GPU reaches coherently.
// ---------------------------------------------------------------------------
// out: g, vara_s (nloci each), yadj (nind), yaadj (bs), {mu, vare, vara, included}, then cls (int32); an array whose
// bit of `want` is 0 is left out (sweep_state_layout gives the places).
__global__ void __launch_bounds__(256) k_get_state(Dev D, int c, StateLayout L, unsigned char *out)
{
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    auto put = [&](size_t at, const double *src, int n) {
        double *dst = reinterpret_cast<double *>(out + at);
        for (int i = t0; i < n; i += stride) dst[i] = src[i];
    };
    if (L.want & STATE_G) put(L.g, D.g + (size_t)c * D.p, D.p);
    if (L.want & STATE_VARA_S) put(L.vara_s, D.vara_s + (size_t)c * D.p, D.p);
    if (L.want & STATE_R) put(L.r, D.r + (size_t)c * D.ldr, D.n);
    if (L.want & STATE_RA) put(L.ra, D.ra + (size_t)c * D.ldra, D.bs);
    if (L.want & STATE_CLS) {
        int32_t *dst = reinterpret_cast<int32_t *>(out + L.cls);
        for (int i = t0; i < D.p; i += stride) dst[i] = D.cls[(size_t)c * D.p + i];
    }
    if (t0 == 0) {
        const ChainScal *S = &D.scal[c];
        double *dst = reinterpret_cast<double *>(out + L.scalars);
        dst[0] = S->mu[D.ctl->rep & 1];
        dst[1] = S->vare;
        dst[2] = S->vara;
        dst[3] = (double)S->included;
    }
}

StateLayout sweep_state_layout(const Dev &D, unsigned want)
{
    StateLayout L{};
    L.want = want;
    auto take = [&](unsigned bit, size_t bytes) {
        const size_t at = L.bytes;
        if (want & bit) L.bytes += (bytes + 15) & ~(size_t)15;
        return at;
    };
    L.g = take(STATE_G, sizeof(double) * (size_t)D.p);
    L.vara_s = take(STATE_VARA_S, sizeof(double) * (size_t)D.p);
    L.r = take(STATE_R, sizeof(double) * (size_t)D.n);
    L.ra = take(STATE_RA, sizeof(double) * (size_t)D.bs);
    L.scalars = L.bytes;
    L.bytes += 4 * sizeof(double);
    L.cls = take(STATE_CLS, sizeof(int32_t) * (size_t)D.p);
    return L;
}

cudaError_t sweep_get_state(const Dev &D, int c, const StateLayout &L, unsigned char *out, cudaStream_t st)
{
    const int grid = std::max(1, std::min((std::max(D.p, D.n) + 255) / 256, 152));
    k_get_state<<<grid, 256, 0, st>>>(D, c, L, out);
    return cudaGetLastError();
}

// No trace rows for the next iterations of a job (or of every job of a batch).
__global__ void k_run_begin(Dev D)
{
    D.ctl->trace_iter = 0;
    D.ctl->trace_cap = 0;
    D.ctl->trace_count = 0;
    D.ctl->trace = nullptr;
}
__global__ void k_run_begin_m(const Dev *dev, int njobs)
{
    const int j = threadIdx.x;
    if (j >= njobs) return;
    RunCtl *ctl = dev[j].ctl;
    ctl->trace_iter = 0;
    ctl->trace_cap = 0;
    ctl->trace_count = 0;
    ctl->trace = nullptr;
}
__global__ void k_batch_errors(const Dev *dev, int njobs, int32_t *out)
{
    const int j = threadIdx.x;
    if (j < njobs) out[j] = dev[j].ctl->err;
}

cudaError_t sweep_run_begin(const Dev &D, cudaStream_t st)
{
    k_run_begin<<<1, 1, 0, st>>>(D);
    return cudaGetLastError();
}
cudaError_t sweep_batch_begin(const Dev *ddev, int njobs, cudaStream_t st)
{
    k_run_begin_m<<<1, MAXJOBS, 0, st>>>(ddev, njobs);
    return cudaGetLastError();
}
cudaError_t sweep_batch_errors(const Dev *ddev, int njobs, int32_t *out, cudaStream_t st)
{
    k_batch_errors<<<1, MAXJOBS, 0, st>>>(ddev, njobs, out);
    return cudaGetLastError();
}

cudaError_t sweep_enqueue_recal(const Dev &D, double mu_slot_unused, cudaStream_t st)
{
    (void)mu_slot_unused;
    k_recal_partial<<<recal_grid(D, RECAL_SPLIT), 256, 0, st>>>(D, 1);
    k_recal_apply<<<recal_grid(D, 1), 256, 0, st>>>(D, 1, -1);
    return cudaGetLastError();
}

}  // namespace soda

// ---------------------------------------------------------------------------
// Several jobs in one launch per kernel (the CUDA-core kernels; every job of a
// batch has the same precision and chain count).  Each wrapper finds its job
// and block coordinates (jg_locate) and runs the same body as the plain
// kernel, so a job's results do not depend on the batch it runs in.
// ---------------------------------------------------------------------------
namespace soda {

__global__ void k_iter_begin_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    iter_begin_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(MU_THREADS) k_mu_partial_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    mu_partial_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(MU_THREADS) k_mu_apply_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    mu_apply_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(64) k_skipped_pre_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    skipped_pre_body(G.dev[j], vb, G.arg[j][0], G.arg[j][1]);
}

// One dense-count entry per chain; every job's before k_skipped_pre_m.
__global__ void k_skipped_clear_m(const Dev *dev, int njobs)
{
    const int j = blockIdx.x;
    if (j < njobs && dev[j].ssdense && (int)threadIdx.x < dev[j].chains) dev[j].ssdense[threadIdx.x] = 0;
}

// (the jobs' grids are multiples of a cluster)
__global__ void __cluster_dims__(SS_CTAS, 1, 1) __launch_bounds__(128) k_skipped_spec_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    skipped_spec_body(G.dev[j], vb.x / SS_CTAS, G.arg[j][0], G.arg[j][1]);
}

template <int NT>
__global__ void __launch_bounds__(NT) k_skipped_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    skipped_body<NT>(G.dev[j], vb, G.arg[j][0], G.arg[j][1]);
}

__global__ void __launch_bounds__(256) k_stats_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    stats_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(HYPER_THREADS) k_hyper_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    hyper_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(256) k_post_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    post_body(G.dev[j], vb);
}

__global__ void __launch_bounds__(256) k_recal_partial_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    recal_partial_body(G.dev[j], vb, 0);
}

__global__ void __launch_bounds__(256) k_recal_apply_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    recal_apply_body(G.dev[j], vb, 0, -1);
}

template <int MODE, int CT>
__global__ void __launch_bounds__(256, rhs_per_sm<MODE, CT>()) k_rhs_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    rhs_body<MODE, CT>(G.dev[j], vb, G.arg[j][0], G.arg[j][1]);
}

template <int MODE, int CT>
__global__ void __launch_bounds__(DrawThreads<CT, false>::v, 1) k_draw_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    draw_body<MODE, CT, false>(G.dev[j], vb, G.arg[j][0], G.arg[j][1], G.arg[j][2]);
}

template <int MODE, int CT>
__global__ void __launch_bounds__(32 * UpdWarps<MODE, CT>::v) k_update_m(const __grid_constant__ JobGrid G)
{
    VB vb;
    const int j = jg_locate(G, vb);
    update_body<MODE, CT>(G.dev[j], vb, G.arg[j][0]);
}

namespace {

// Builds the JobGrid of one launch from each job's grid (x, y, z; all zero
// for a job that sits the launch out) and arguments.
struct GridBuilder {
    JobGrid g;
    explicit GridBuilder(const Dev *ddev, int njobs)
    {
        memset(&g, 0, sizeof g);
        g.dev = ddev;
        g.njobs = njobs;
    }
    void set(int j, int gx, int gy, int gz, int a0 = 0, int a1 = 0, int a2 = 0)
    {
        const int n = gx > 0 && gy > 0 && gz > 0 ? gx * gy * gz : 0;
        g.gx[j] = gx > 0 ? gx : 1;
        g.gy[j] = gy > 0 ? gy : 1;
        g.off[j + 1] = g.off[j] + n;
        g.arg[j][0] = a0;
        g.arg[j][1] = a1;
        g.arg[j][2] = a2;
    }
    int total() const { return g.off[g.njobs]; }
};

template <int MODE, int CT>
static cudaError_t multi_step(const BatchPlan &P, int t, cudaStream_t st)
{
    const int nj = P.njobs;
    constexpr int MTS = 8 * SptOf<CT>::v, NT = DrawThreads<CT, false>::v;
    GridBuilder rhs(P.ddev, nj), draw(P.ddev, nj), upd(P.ddev, nj);
    size_t usmem = 0;
    for (int j = 0; j < nj; ++j) {
        const Dev &D = P.hdev[j];
        if (t >= D.nb) {
            rhs.set(j, 0, 0, 0);
            draw.set(j, 0, 0, 0);
            upd.set(j, 0, 0, 0);
            continue;
        }
        const int N = P.blk_sizes[j][t];
        const int mtiles = (N + MTS - 1) / MTS;
        const int ks = P.ksplit[j];
        rhs.set(j, mtiles * ks, 1, 1, t, ks);
        draw.set(j, (N * CT + NT - 1) / NT, 1, 1, t, ks, N);
        upd.set(j, D.nr_ctas + (D.bs + UT - 1) / UT, 1, 1, t);
        usmem = std::max(usmem, update_smem_bytes_ct<MODE, CT>(D.bs));
    }
    if (rhs.total() == 0) return cudaSuccess;
    cudaError_t e = launch_pdl(k_rhs_m<MODE, CT>, dim3(rhs.total()), dim3(256), rhs_smem_bytes<MODE, CT>(), st, rhs.g);
    if (e == cudaSuccess) e = launch_pdl(k_draw_m<MODE, CT>, dim3(draw.total()), dim3(NT), 0, st, draw.g);
    if (e == cudaSuccess)
        e = launch_pdl(k_update_m<MODE, CT>, dim3(upd.total()), dim3(32 * UpdWarps<MODE, CT>::v), usmem, st, upd.g);
    return e;
}

template <int MODE>
static cudaError_t multi_step_mode(const BatchPlan &P, int t, cudaStream_t st)
{
    switch (P.hdev[0].chains) {
    case 1: return multi_step<MODE, 1>(P, t, st);
    case 2: return multi_step<MODE, 2>(P, t, st);
    case 4: return multi_step<MODE, 4>(P, t, st);
    case 8: return multi_step<MODE, 8>(P, t, st);
    case 16: return multi_step<MODE, 16>(P, t, st);
    default: return cudaErrorInvalidValue;
    }
}

template <int MODE, int CT>
static cudaError_t multi_attrs(size_t usmem)
{
    cudaError_t e = cudaFuncSetAttribute(k_rhs_m<MODE, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)rhs_smem_bytes<MODE, CT>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_update_m<MODE, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)usmem);
    if (e == cudaSuccess) e = max_carveout(k_rhs_m<MODE, CT>);
    if (e == cudaSuccess) e = max_carveout(k_draw_m<MODE, CT>);
    if (e == cudaSuccess) e = max_carveout(k_update_m<MODE, CT>);
    return e;
}

template <int MODE>
static cudaError_t multi_attrs_mode(int chains, int max_bs)
{
    switch (chains) {
    case 1: return multi_attrs<MODE, 1>(update_smem_bytes_ct<MODE, 1>(max_bs));
    case 2: return multi_attrs<MODE, 2>(update_smem_bytes_ct<MODE, 2>(max_bs));
    case 4: return multi_attrs<MODE, 4>(update_smem_bytes_ct<MODE, 4>(max_bs));
    case 8: return multi_attrs<MODE, 8>(update_smem_bytes_ct<MODE, 8>(max_bs));
    case 16: return multi_attrs<MODE, 16>(update_smem_bytes_ct<MODE, 16>(max_bs));
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t sweep_multi_prepare(int precision, int chains, int max_bs)
{
    cudaError_t e = sweep_prepare(max_bs);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_skipped_m<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM_MAX);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_skipped_spec_m, cudaFuncAttributeMaxDynamicSharedMemorySize, SS_SMEM_MAX);
    if (e != cudaSuccess) return e;
    if (precision == SODAGPU_FP64) return multi_attrs_mode<SODAGPU_FP64>(chains, max_bs);
    if (precision == SODAGPU_FP32) return multi_attrs_mode<SODAGPU_FP32>(chains, max_bs);
    return multi_attrs_mode<SODAGPU_FP8>(chains, max_bs);
}

template <int MODE, int CT>
static int multi_split(int N, int ldx, int cta_share)
{
    constexpr int MTS = 8 * SptOf<CT>::v;
    const int mtiles = (N + MTS - 1) / MTS;
    const int nst = (ldx + RhsCfg<MODE>::KST - 1) / RhsCfg<MODE>::KST;
    return rhs_splits(cta_share * rhs_per_sm<MODE, CT>(), mtiles, std::max(1, nst));
}

template <int MODE>
static int multi_split_mode(int N, int chains, int ldx, int cta_share)
{
    switch (chains) {
    case 1: return multi_split<MODE, 1>(N, ldx, cta_share);
    case 2: return multi_split<MODE, 2>(N, ldx, cta_share);
    case 4: return multi_split<MODE, 4>(N, ldx, cta_share);
    case 8: return multi_split<MODE, 8>(N, ldx, cta_share);
    default: return multi_split<MODE, 16>(N, ldx, cta_share);
    }
}

int sweep_multi_rhs_split(int precision, int N, int chains, int ldx, int cta_share)
{
    if (precision == SODAGPU_FP64) return multi_split_mode<SODAGPU_FP64>(N, chains, ldx, cta_share);
    if (precision == SODAGPU_FP32) return multi_split_mode<SODAGPU_FP32>(N, chains, ldx, cta_share);
    return multi_split_mode<SODAGPU_FP8>(N, chains, ldx, cta_share);
}

cudaError_t sweep_enqueue_iteration_multi(const BatchPlan &P, int sm_count, cudaStream_t st)
{
    const int nj = P.njobs;
    if (nj < 1 || nj > MAXJOBS) return cudaErrorInvalidValue;
    const int prec = P.hdev[0].precision;
    GridBuilder one(P.ddev, nj), rows(P.ddev, nj);
    int maxnb = 0;
    for (int j = 0; j < nj; ++j) {
        const Dev &D = P.hdev[j];
        one.set(j, 1, 1, 1);
        rows.set(j, mu_grid(D.n), D.chains, 1);
        maxnb = std::max(maxnb, D.nb);
    }
    k_iter_begin_m<<<one.total(), 1, 0, st>>>(one.g);
    cudaError_t e = launch_pdl(k_mu_partial_m, dim3(rows.total()), dim3(MU_THREADS), 0, st, rows.g);
    if (e == cudaSuccess) e = launch_pdl(k_mu_apply_m, dim3(rows.total()), dim3(MU_THREADS), 0, st, rows.g);
    if (e != cudaSuccess) return e;
    for (int t = 0; t < maxnb; ++t) {
        e = prec == SODAGPU_FP64   ? multi_step_mode<SODAGPU_FP64>(P, t, st)
            : prec == SODAGPU_FP32 ? multi_step_mode<SODAGPU_FP32>(P, t, st)
                                   : multi_step_mode<SODAGPU_FP8>(P, t, st);
        if (e != cudaSuccess) return e;
    }
    GridBuilder stats(P.ddev, nj), hyp(P.ddev, nj), post(P.ddev, nj), rp(P.ddev, nj),
        ra(P.ddev, nj);
    int nskip = 0;
    for (int j = 0; j < nj; ++j) {
        const Dev &D = P.hdev[j];
        const int C = D.chains;
        nskip = std::max(nskip, D.nskipped);
        stats.set(j, NSTAT + mu_grid(D.n), C, 1);
        hyp.set(j, C, 1, 1);
        post.set(j, post_grid(D, sm_count), C, 1);
        rp.set(j, recal_grid(D, RECAL_SPLIT), 1, 1);
        ra.set(j, recal_grid(D, 1), 1, 1);
    }
    for (int t0 = 0; t0 < nskip; t0 += SS_CHUNK) {
        // by where the residual is held; a small one's chains each go through one of two kernels
        GridBuilder pre(P.ddev, nj), spec(P.ddev, nj), small(P.ddev, nj), large(P.ddev, nj);
        size_t ssm = 0;
        for (int j = 0; j < nj; ++j) {
            const Dev &D = P.hdev[j];
            const int cnt = std::max(0, std::min(SS_CHUNK, D.nskipped - t0));
            const size_t sm = skipped_smem(D.n);
            pre.set(j, (cnt + 63) / 64, D.chains, 1, t0, cnt);
            spec.set(j, cnt > 0 && sm ? SS_CTAS * D.chains : 0, 1, 1, t0, cnt);
            small.set(j, cnt > 0 && sm ? D.chains : 0, 1, 1, t0, cnt);
            large.set(j, cnt > 0 && !sm ? D.chains : 0, 1, 1, t0, cnt);
            if (cnt > 0) ssm = std::max(ssm, sm);
        }
        k_skipped_clear_m<<<nj, 32, 0, st>>>(P.ddev, nj);
        k_skipped_pre_m<<<pre.total(), 64, 0, st>>>(pre.g);
        if (spec.total() > 0) k_skipped_spec_m<<<spec.total(), 128, ssm, st>>>(spec.g);
        if (small.total() > 0) k_skipped_m<128><<<small.total(), 128, ssm, st>>>(small.g);
        if (large.total() > 0) k_skipped_m<512><<<large.total(), 512, 0, st>>>(large.g);
    }
    e = launch_pdl(k_stats_m, dim3(stats.total()), dim3(256), 0, st, stats.g);
    if (e == cudaSuccess) e = launch_pdl(k_hyper_m, dim3(hyp.total()), dim3(HYPER_THREADS), 0, st, hyp.g);
    if (e == cudaSuccess) e = launch_pdl(k_post_m, dim3(post.total()), dim3(256), 0, st, post.g);
    if (e == cudaSuccess) e = launch_pdl(k_recal_partial_m, dim3(rp.total()), dim3(256), 0, st, rp.g);
    if (e == cudaSuccess) e = launch_pdl(k_recal_apply_m, dim3(ra.total()), dim3(256), 0, st, ra.g);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace soda

// dgv.cuh — genomic values pred = mu + X * effects (compute_dgv, utilities.f90:616-622) for the three callers of
// the library: a job's own codes, a PLINK .bed payload, and the caller's device codes (noalloc.cu).
//
// One genotype per FP64 addition is bound by GB300's FP64 pipe (two lanes a clock and SM: n * p = 1e9 genotypes
// are 1.6 ms of additions alone, and byte-wide loads with a dependent table lookup each took 4.1 ms).  So the
// additions are integer, and there is one for every five SNPs:
//   * w_k = effect_k / sd_k becomes a 64-bit fixed-point number.  The unit of a sub-range of at most DGV_SUB SNPs
//     is 2^(E-62) with 4 * sum |w| < 2^E <= 8 * sum |w|, so no sum overflows and all of them are exact; the rounding
//     of each w is at most 2^-60 of that sum, below the 2^-53 of the running FP64 sum that a chain of additions makes
//     at every term.
//   * the value of a code is (code - 2 f) / sd.  With m the code nearest to 2 f it is split into (code - m) w, summed in
//     integers (they start at the constant -sum m_k w_k), and (m - 2 f) w, which is the
//     same for everyone: their sum over a sub-range is added in FP64 by a tree.  Where one allele is common, code - 2 f
//     is near 0 for nearly everyone, and with 2 f w in place of (m - 2 f) w the two sums would cancel (n = 20,000,
//     f = 1 - 1 / (2 n): 1e-12 of the value).
//   * five SNPs' codes (0..2) make a base-3 index below 243, computed for four individuals at once in the bytes of
//     a word (w0 + 3 w1 + 9 w2 + 27 w3 + 81 w4, no carries), into a table of the group's 243 sums in shared
//     memory.  Per five SNPs and individual: one 8-byte shared load and one 64-bit integer addition.
// The kernel is then bound by the codes' bandwidth and the shared-memory lookups (4.6 wavefronts a warp, bank
// conflicts included) together.  Measured: n = 20,000, p = 50,000, a job's int8 codes 189 us, 5.3 TB/s (4055 us
// before); a .bed payload, n = 4,999, p = 50,000, 143 us (1216 us after its expansion to bytes); the caller's codes
// at n = 1,001, p = 5,003 in 14 us (36 us).  Against 113-bit arithmetic (n = 300 to 1,001, p = 4,000 to 20,000) the
// relative error is 2.5e-16 (rms; 3.2e-16 by frequencies and 4.3e-16 by the table with 2 f w, 6.2e-16 as a chain of
// FP64 additions).
//
// Sub-ranges whose effects are not finite, or whose sum of |w| lies outside 1e-280..1e280, take one FP64 addition
// a genotype, as every sub-range did: an infinite or NaN effect gives what the plain sum gives.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "tc.cuh"

namespace soda {
namespace {   // each translation unit that includes this has kernels of its own

enum { DGV_PADDED = 0, DGV_RAW = 1, DGV_BED = 2 };

constexpr int DGV_GROUP = 5;                    // SNPs per table of 3^5 = 243 sums
constexpr int DGV_TAB = 256;                    // its entries: codes that the caller is about to refuse index up to 255
constexpr int DGV_CHUNK = 8;                    // tables built at a time
constexpr int DGV_SUB = 24 * DGV_CHUNK * DGV_GROUP;   // SNPs that share a fixed-point unit

// Layout of a thread's individuals: byte b of word j is individual dgv_at(j, b) of the tile's 4 * W * NT.
//   DGV_PADDED  int8 codes 0..2, column stride ld a multiple of 128 and columns readable up to it; one 16-byte load
//   DGV_RAW     int8 codes with any column stride and alignment, codes outside 0..2 count as 1; the words of a
//               warp are consecutive
//   DGV_BED     PLINK records of ld bytes; the four 2-bit fields of the bytes of one word
template <int SRC, int NT, int W>
__device__ __forceinline__ int dgv_at(int j, int b)
{
    if (SRC == DGV_PADDED) return 4 * W * (int)threadIdx.x + 4 * j + b;
    if (SRC == DGV_BED) return 4 * W * (int)threadIdx.x + 4 * b + j;
    return 4 * (j * NT + (int)threadIdx.x) + b;
}

// Up to four bytes from a, one load each: the two ends of the buffer.  (Not inlined: the short kernels are bound by
// fetching their own instructions.)
static __device__ __noinline__ uint32_t dgv_bytes(const uint8_t *a, int left)
{
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = j < left ? __ldg(a + j) : 0u;   // all in flight at once
    return v[0] | v[1] << 8 | v[2] << 16 | v[3] << 24;
}

// What a load leaves in registers until its group is looked up: the words, or for sources of any alignment the two
// aligned words around each (nothing may use a loaded value before, or the loads would wait for one another).
template <int SRC, int W>
struct DgvLoad {
    static constexpr int N = SRC == DGV_PADDED ? W : (SRC == DGV_BED ? 2 : 2 * W);
    uint32_t w[N];
};

// Misalignment of SNP k's column, the same for every thread (their offsets are multiples of four bytes).
__device__ __forceinline__ unsigned dgv_mis(const uint8_t *src, size_t ld, int k)
{
    return (unsigned)((uintptr_t)(src + (size_t)k * ld) & 3u);
}

// The words of SNP k of p.  A word may hold codes past the last individual (those of the next SNP): they are valid
// codes of values that nothing reads.  Every byte read lies inside the buffer, src .. end - 1.
template <int SRC, int NT, int W>
__device__ __forceinline__ DgvLoad<SRC, W> dgv_load(const uint8_t *src, const uint8_t *end, size_t ld, int k, int p,
                                                    int t0, int n)
{
    static_assert(SRC == DGV_RAW || W == 4, "one 16-byte load, or 16 fields of a word");
    DgvLoad<SRC, W> r;
    if constexpr (SRC == DGV_PADDED) {
        const int i0 = t0 + dgv_at<SRC, NT, W>(0, 0);
        const uint4 v = i0 < n ? __ldg(reinterpret_cast<const uint4 *>(src + (size_t)k * ld + i0))
                               : make_uint4(0, 0, 0, 0);
        r.w[0] = v.x;
        r.w[1] = v.y;
        r.w[2] = v.z;
        r.w[3] = v.w;
    } else {
        // the aligned words around a cover a - 3 .. a + 7: inside the buffer unless k is one of its first or last SNPs
        const bool near = (size_t)k * ld < 4 || (size_t)(p - 1 - k) * ld < 8;
        const unsigned m = dgv_mis(src, ld, k);
#pragma unroll
        for (int j = 0; j < DgvLoad<SRC, W>::N / 2; ++j) {
            const int i0 = t0 + dgv_at<SRC, NT, W>(j, 0);
            const uint8_t *a = src + (size_t)k * ld + (SRC == DGV_BED ? i0 >> 2 : i0);
            const bool edge = near && (a < src + 3 || a + 8 > end), ok = i0 < n && !edge;
            const uint32_t *w = reinterpret_cast<const uint32_t *>(a - m);
            r.w[2 * j] = ok ? __ldg(w) : 0u;
            r.w[2 * j + 1] = ok ? __ldg(w + 1) : 0u;
            if (edge && i0 < n) {   // the word's bytes, placed where the funnel shift by m will find them
                const uint32_t v = dgv_bytes(a, (int)min((ptrdiff_t)4, end - a));
                r.w[2 * j] = v << (8 * m);
                r.w[2 * j + 1] = m ? v >> (32 - 8 * m) : 0u;
            }
        }
    }
    return r;
}

template <int SRC, int W>
__device__ __forceinline__ uint32_t dgv_codes(const DgvLoad<SRC, W> &r, int j, unsigned mis)
{
    if constexpr (SRC == DGV_PADDED) {
        return r.w[j];
    } else if constexpr (SRC == DGV_BED) {
        uint32_t x = __funnelshift_r(r.w[0], r.w[1], 8 * mis);
        x -= (x >> 1) & 0x55555555u;   // 00,01,10,11 -> 0,1,1,2 (utilities.f90:438-454)
        return (x >> (2 * j)) & 0x03030303u;
    } else {
        // bytes above 2 (any of bits 2-7, or both of bits 0 and 1) become 1
        const uint32_t w = __funnelshift_r(r.w[2 * j], r.w[2 * j + 1], 8 * mis);
        uint32_t bad = (w & 0xFCFCFCFCu) | ((w & (w >> 1) & 0x01010101u) << 2);
        if (bad) {
            bad |= bad >> 4 & 0x0F0F0F0Fu;
            bad |= bad >> 2 & 0x3F3F3F3Fu;
            bad |= bad >> 1;
            bad &= 0x01010101u;
            return (w & ~(bad * 0xFFu)) | bad;
        }
        return w;
    }
}

// SNP k: w = effect / sd (0 for monomorphic SNPs), the code m nearest to 2 f, and xme, the value of that code times the
// effect: the value of a code is (code - 2 f) / sd (xscale, utilities.f90:525-534, 545-552).  From a centring table, or
// from the allele frequency.
__device__ __forceinline__ void dgv_coef(const double *xv, const double *freq, const int32_t *perm,
                                         const double *eff, int k, double &w, double &xme, unsigned &m)
{
    const double e = eff[perm ? perm[k] : k];
    w = xme = 0.0;
    m = 0;
    if (e == 0.0) return;
    if (xv) {
        const double2 lo = *reinterpret_cast<const double2 *>(xv + (size_t)k * 4);
        const double2 hi = *reinterpret_cast<const double2 *>(xv + (size_t)k * 4 + 2);
        w = hi.y * e;
        // the value of least magnitude, by the upper words: an FP64 comparison takes the narrow pipe 64 cycles a warp
        const int h0 = __double2hiint(lo.x) & 0x7FFFFFFF, h1 = __double2hiint(lo.y) & 0x7FFFFFFF;
        const int h2 = __double2hiint(hi.x) & 0x7FFFFFFF;
        m = h0 < h1 ? 0 : (h2 < h1 ? 2 : 1);
        xme = (m == 0 ? lo.x : (m == 1 ? lo.y : hi.x)) * e;
        return;
    }
    const double f = freq[k], eps = 2.220446049250313e-16;
    if (f < eps || (1.0 - f) < eps) {
        w = xme = 0.0 * e;   // NaN for an effect that is not finite, which takes the sub-range to the plain sum
        return;
    }
    const double twop = __dmul_rn(2.0, f);
    w = e / sqrt(__dmul_rn(twop, __dsub_rn(1.0, f)));
    const int h = __double2hiint(twop);   // 1/2 and 3/2: the upper words 0x3FE00000 and 0x3FF80000
    m = h < 0x3FE00000 ? 0 : (h < 0x3FF80000 ? 1 : 2);
    xme = __dsub_rn(m == 0 ? 0.0 : (m == 1 ? 1.0 : 2.0), twop) * w;
}

// A sub-range outside the fixed-point range: the three values of SNP k times its effect, and the plain sums of
// individuals i0 .. i1 - 1 over values of `terms` SNPs at a time in shared memory (t), one FP64 addition a genotype.  Consecutive individuals
// lie in consecutive threads, the loads of eight SNPs in flight.  An infinite effect, a job's codes: n = 300, p = 400:
// 38.6 us a call; n = 100,000, p = 2,000: 459 us (137 and 1185 us when each thread walked the values of its own sixteen).
static __device__ __noinline__ void dgv_terms(const double *xv, const double *freq, const int32_t *perm,
                                              const double *eff, int k, double *t)
{
    const double e = eff[perm ? perm[k] : k], eps = 2.220446049250313e-16;
    double x[3] = {0.0, 0.0, 0.0};
    if (xv) {
        for (int g = 0; g < 3; ++g) x[g] = xv[(size_t)k * 4 + g];
    } else {
        const double f = freq[k], twop = __dmul_rn(2.0, f);
        if (!(f < eps || (1.0 - f) < eps)) {
            const double sd = sqrt(__dmul_rn(twop, __dsub_rn(1.0, f)));
            for (int g = 0; g < 3; ++g) x[g] = __ddiv_rn(__dsub_rn((double)g, twop), sd);
        }
    }
    for (int g = 0; g < 3; ++g) t[g] = e == 0.0 ? 0.0 : x[g] * e;
}
template <int SRC>
static __device__ __noinline__ void dgv_plain(const uint8_t *src, size_t ld, const double *xv, const double *freq,
                                              const int32_t *perm, const double *eff, int k0, int cnt, int i0, int i1,
                                              double *t, int terms, bool first, double *out)
{
    for (int c0 = 0; c0 < cnt; c0 += terms) {
        const int m = min(terms, cnt - c0);
        __syncthreads();   // every use of what t holds is done, and so is every store of out
        for (int q = threadIdx.x; q < m; q += blockDim.x) dgv_terms(xv, freq, perm, eff, k0 + c0 + q, t + 4 * q);
        __syncthreads();
        for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
            const uint8_t *a = src + (size_t)(k0 + c0) * ld + (SRC == DGV_BED ? i >> 2 : i);
            double sum = first && c0 == 0 ? 0.0 : out[i];
#pragma unroll 8
            for (int k = 0; k < m; ++k) {
                int g = a[(size_t)k * ld];
                if (SRC == DGV_BED) {
                    g = g >> (2 * (i & 3)) & 3;
                    g -= g >> 1;
                }
                sum += t[4 * k + (g > 2 ? 1 : g)];
            }
            out[i] = sum;
        }
    }
}

// part[s * ldp + i] = sum over the SNPs of split s (per SNPs each) of x_ik effect_k.  A CTA of NT threads takes
// 4 * W * NT individuals; the loads of the next PF groups of SNPs are in flight while a group is looked up: one
// where a thread loads 16 bytes a SNP, more where it loads 4.
template <int SRC, int NT, int W>
__global__ void __launch_bounds__(NT, 512 / NT)
    k_dgv_tab(const uint8_t *src, size_t ld, const double *xv, const double *freq, const int32_t *perm,
              const double *eff, int n, int p, int per, double *part, size_t ldp)
{
    __shared__ double s_w[DGV_SUB];                         // w, then the same slot in fixed point
    __shared__ long long s_t[DGV_CHUNK][DGV_TAB];
    __shared__ double sh[NT / 32][2], s_c[3];
    __shared__ uint8_t s_near[DGV_SUB];                     // m
    __shared__ long long s_m[NT / 32];                      // the warps' sums of m w
    long long *s_f = reinterpret_cast<long long *>(s_w);
    constexpr int PF = SRC == DGV_BED ? 2 : (W == 1 ? 4 : 1);
    static_assert(DGV_CHUNK % PF == 0, "a chunk's tables serve whole rounds of the ring");
    const uint8_t *end = src + (size_t)(p - 1) * ld + (SRC == DGV_BED ? ld : (size_t)n);
    const int tid = threadIdx.x, t0 = blockIdx.x * (4 * W * NT);
    const int r0 = blockIdx.y * per, r1 = min(p, r0 + per);
    double *out = part + (size_t)blockIdx.y * ldp;
    // this lane's entries 27 b + lane of a warp's tables: digits of the group's first three SNPs
    const int lane = tid & 31, d0 = lane % 3, d1 = lane / 3 % 3, d2 = lane / 9;
    tc::pdl_trigger();

    for (int k0 = r0; k0 < r1; k0 += DGV_SUB) {
        const int cnt = min(DGV_SUB, r1 - k0);
        const int groups = (cnt + DGV_GROUP - 1) / DGV_GROUP;
        const int padded = (groups + DGV_CHUNK - 1) / DGV_CHUNK * (DGV_CHUNK * DGV_GROUP);
        double base = 0.0, mag = 0.0;
        // SNPs past the sub-range have w = 0: any valid codes do, and the first SNP's words are at hand
        DgvLoad<SRC, W> ring[PF][DGV_GROUP];
        auto fetch = [&](DgvLoad<SRC, W>(&r)[DGV_GROUP], int g) {
#pragma unroll
            for (int d = 0; d < DGV_GROUP; ++d) {
                const int k = k0 + DGV_GROUP * g + d;
                r[d] = dgv_load<SRC, NT, W>(src, end, ld, k < r1 ? k : k0, p, t0, n);
            }
        };
#pragma unroll
        for (int q = 0; q < PF; ++q) fetch(ring[q], q);
        // the sums of w's magnitude and of xme over the warps that hold SNPs, then one thread: every FP64
        // instruction of a warp takes the pipe 16 cycles
        __syncthreads();
        const int warps = min(NT, padded + 31) / 32;
        for (int q = tid; q < padded; q += NT) {
            double w = 0.0, xme = 0.0;
            unsigned m = 0;
            if (q < cnt) dgv_coef(xv, freq, perm, eff, k0 + q, w, xme, m);
            s_w[q] = w;
            s_near[q] = (uint8_t)m;
            base += xme;
            mag += fabs(w);
        }
        if ((tid >> 5) < warps) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                base += __shfl_xor_sync(0xffffffffu, base, o);
                mag += __shfl_xor_sync(0xffffffffu, mag, o);
            }
            if (lane == 0) {
                sh[tid >> 5][0] = base;
                sh[tid >> 5][1] = mag;
            }
        }
        __syncthreads();
        if (tid == 0) {
            double tb = 0.0, tm = 0.0;
            for (int w = 0; w < warps; ++w) {
                tb += sh[w][0];
                tm += sh[w][1];
            }
            // 4 tm = m 2^ex with m in [1/2, 1); a scale of 0 where the sums do not fit
            const bool fits = tm == 0.0 || (tm > 1e-280 && tm < 1e280);
            const int ex = tm == 0.0 ? 0 : ((__double2hiint(4.0 * tm) >> 20) & 0x7FF) - 1022;
            s_c[0] = tb;
            s_c[1] = fits ? __hiloint2double((1023 + 62 - ex) << 20, 0) : 0.0;
            s_c[2] = fits ? __hiloint2double((1023 - 62 + ex) << 20, 0) : 0.0;
        }
        __syncthreads();
        base = s_c[0];
        const double scale = s_c[1], unit = s_c[2];
        if (scale == 0.0) {
            // (its values in place of the tables)
            dgv_plain<SRC>(src, ld, xv, freq, perm, eff, k0, cnt, t0, min(n, t0 + 4 * W * NT),
                           reinterpret_cast<double *>(s_t), DGV_CHUNK * DGV_TAB / 4, k0 == r0, out);
            continue;
        }
        long long msum = 0;
        for (int q = tid; q < padded; q += NT) {
            const long long f = __double2ll_rn(s_w[q] * scale);
            const unsigned m = s_near[q];
            s_f[q] = f;
            msum += (m & 1u ? f : 0) + (m & 2u ? f << 1 : 0);
        }
        if ((tid >> 5) < warps) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) msum += __shfl_xor_sync(0xffffffffu, msum, o);
            if (lane == 0) s_m[tid >> 5] = msum;
        }
        __syncthreads();   // s_f and s_m are complete
        // the sums start at the constant: subtracted at the end, in registers that live through the loop, it cost the
        // 256-thread kernel a tenth
        long long centre = 0;
        for (int w = 0; w < warps; ++w) centre += s_m[w];
        long long acc[4 * W];
#pragma unroll
        for (int j = 0; j < 4 * W; ++j) acc[j] = -centre;
#pragma unroll 1
        for (int g0 = 0; g0 < groups; g0 += PF) {
            if (g0 % DGV_CHUNK == 0) {
                if (g0 > 0) __syncthreads();   // every lookup in the previous chunk's tables is done
#pragma unroll 1
                for (int h = tid >> 5; h < DGV_CHUNK; h += NT / 32) {
                    const long long *f = s_f + DGV_GROUP * (g0 + h);
                    long long a = (d0 ? f[0] : 0) + (d1 ? f[1] : 0) + (d2 ? f[2] : 0);
                    a += (d0 == 2 ? f[0] : 0) + (d1 == 2 ? f[1] : 0) + (d2 == 2 ? f[2] : 0);
                    const long long f3 = f[3], f4 = f[4];
                    if (lane < 27)
#pragma unroll
                        for (int b = 0; b < 9; ++b) s_t[h][27 * b + lane] = a + (b % 3) * f3 + (b / 3) * f4;
                }
                __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < PF; ++q) {
                const int g = g0 + q;
                uint32_t idx[W];
#pragma unroll
                for (int j = 0; j < W; ++j) idx[j] = 0u;
#pragma unroll
                for (int d = DGV_GROUP - 1; d >= 0; --d) {
                    const int k = k0 + DGV_GROUP * g + d;
                    const unsigned mis = SRC == DGV_PADDED ? 0u : dgv_mis(src, ld, k < r1 ? k : k0);
#pragma unroll
                    for (int j = 0; j < W; ++j) idx[j] = 3u * idx[j] + dgv_codes<SRC, W>(ring[q][d], j, mis);
                }
                if (g + PF < groups) fetch(ring[q], g + PF);
                const long long *tab = s_t[g % DGV_CHUNK];
#pragma unroll
                for (int j = 0; j < 4 * W; ++j) acc[j] += tab[(idx[j >> 2] >> (8 * (j & 3))) & 0xFFu];
            }
        }
#pragma unroll
        for (int j = 0; j < 4 * W; ++j) {
            const int i = t0 + dgv_at<SRC, NT, W>(j >> 2, j & 3);
            if (i < n) out[i] = (k0 > r0 ? out[i] : 0.0) + (base + (double)acc[j] * unit);
        }
    }
}

// pred = mu + the splits' sums: 32 individuals a CTA, eight threads each, whose sums are added in order.
__global__ void __launch_bounds__(256)
    k_dgv_sum(const double *part, size_t ldp, int n, int nsplit, double mu, double *pred)
{
    __shared__ double sh[8][32];
    tc::pdl_wait();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    double d = 0.0;
    if (i < n)
        for (int s = w; s < nsplit; s += 8) d += part[(size_t)s * ldp + i];
    sh[w][lane] = d;
    __syncthreads();
    if (w == 0 && i < n) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += sh[q][lane];
        pred[i] = mu + t;
    }
}

// Threads per CTA: small tiles where larger ones would be mostly padding, large ones where a table then serves more
// lookups.  dgv_enqueue gives a thread 16 individuals, but four to the small tiles of DGV_RAW, whose words take two
// loads each.
inline int dgv_tile(int n) { return n <= 1024 ? 1024 : (n <= 8192 ? 2048 : 4096); }

// Column splits: one wave of 512 threads an SM (152 of them), but at least one chunk of SNPs a split, so that a
// CTA's tables serve it whole.  The result's last bits depend on it.
inline int dgv_splits(int n, int p)
{
    const int tiles = (n + dgv_tile(n) - 1) / dgv_tile(n);
    const int most = (p + DGV_CHUNK * DGV_GROUP - 1) / (DGV_CHUNK * DGV_GROUP);
    const int want = 152 * (8192 / dgv_tile(n)) / tiles;
    return want < 1 ? 1 : (want < most ? want : most);
}

// Enqueues the splits' sums: part holds nsplit * ldp doubles, ldp >= n; fewer splits may be used (the return value
// says how many, or -1 for a failed launch).  cudaLaunchKernel* reports a failed launch in its own return value: an
// error that the caller left pending is neither reported nor cleared.
template <int SRC>
inline int dgv_enqueue_tab(const uint8_t *src, size_t ld, const double *xv, const double *freq, const int32_t *perm,
                           const double *eff, int n, int p, double *part, size_t ldp, int nsplit, cudaStream_t st)
{
    int per = (p + nsplit - 1) / nsplit;
    per = (per + DGV_GROUP - 1) / DGV_GROUP * DGV_GROUP;
    nsplit = (p + per - 1) / per;
    constexpr int W = SRC == DGV_RAW ? 1 : 4;   // words of a thread in the small tiles
    const int tile = dgv_tile(n), nt = tile == 1024 ? 256 / W : tile / 16;
    const dim3 grid((n + tile - 1) / tile, nsplit);
    void *args[] = {(void *)&src, (void *)&ld, (void *)&xv, (void *)&freq, (void *)&perm, (void *)&eff,
                    (void *)&n,   (void *)&p,  (void *)&per, (void *)&part, (void *)&ldp};
    const void *kern = tile == 1024   ? (const void *)k_dgv_tab<SRC, 256 / W, W>
                       : tile == 2048 ? (const void *)k_dgv_tab<SRC, 128, 4>
                                      : (const void *)k_dgv_tab<SRC, 256, 4>;
    return cudaLaunchKernel(kern, grid, dim3(nt), args, 0, st) == cudaSuccess ? nsplit : -1;
}

inline cudaError_t dgv_enqueue_sum(const double *part, size_t ldp, int n, int nsplit, double mu, double *pred,
                                   cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((n + 31) / 32);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void *args[] = {(void *)&part, (void *)&ldp, (void *)&n, (void *)&nsplit, (void *)&mu, (void *)&pred};
    return cudaLaunchKernelExC(&cfg, (const void *)k_dgv_sum, args);
}

template <int SRC>
inline cudaError_t dgv_enqueue(const uint8_t *src, size_t ld, const double *xv, const double *freq,
                               const int32_t *perm, const double *eff, int n, int p, double mu, double *part,
                               size_t ldp, int nsplit, double *pred, cudaStream_t st)
{
    nsplit = dgv_enqueue_tab<SRC>(src, ld, xv, freq, perm, eff, n, p, part, ldp, nsplit, st);
    return nsplit < 0 ? cudaErrorLaunchFailure : dgv_enqueue_sum(part, ldp, n, nsplit, mu, pred, st);
}

}  // namespace
}  // namespace soda

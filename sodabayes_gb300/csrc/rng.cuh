// rng.cuh — counter-based draws for the SODA sampler (device side).
//
// The reference gives every OpenMP thread its own xoroshiro128+ stream
// (parallelrng.f90:54-149), so a SNP's draws depend on which thread ran it.
// On the GPU each draw is instead keyed by (seed, chain, iteration, slot,
// purpose): Philox4x32-10 (Salmon, Moraes, Dror & Shaw, SC'11) turns that
// counter into 64-bit words, which are mapped to [0,1) exactly like
// rng_int64_to_real64 (parallelrng.f90:242-249).  The distributions below
// restate the reference's transforms:
//   normal         Box-Muller, sine branch, REAL-precision pi (parallelrng.f90:264-277)
//   gamma          Marsaglia & Tsang 2000, boost for shape<1  (parallelrng.f90:294-333)
//   inv. chi^2     1/gamma(dof/2, 2/(dof*scale))               (parallelrng.f90:348-362)
//   Dirichlet      normalised gammas                            (parallelrng.f90:445-455)
#pragma once
#include <stdint.h>
#include "../../include/sodagpu.h"

namespace soda {

// Purposes (third counter word); the CPU oracle uses the same numbering.
enum Purpose : uint32_t {
    P_SNP = 1, P_MU = 2, P_VARA = 3, P_VARE = 4, P_PI = 5, P_RA = 6,
    P_SKIP = 7, P_PERM = 8, P_POWER = 9
};

// parallelrng.f90:20 declares pi as a default REAL literal: float(pi) widened.
#define SODA_REF_PI 3.1415927410125732

// Device error code of a draw that overran its injected-draw tape record.
constexpr int CRNG_TAPE_OVERRUN = 19;

struct CRng {
    uint32_t k0, k1, c0, c1, c2, c3;
    uint32_t o0, o1, o2, o3;
    int have;   // cached outputs of the last block: 2 both halves, 1 the second, 0 none
    // injected draws: the uniforms of this draw site come from a tape record
    // of SODAGPU_TAPE_W values instead of Philox; tover is set on overrun
    const double *tape;
    int tpos;
    int *tover;
};

__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

__host__ __device__ __forceinline__ void philox4x32_10(uint32_t &c0, uint32_t &c1, uint32_t &c2,
                                                       uint32_t &c3, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
        const uint32_t lo0 = 0xD2511F53u * c0, hi0 = mulhi32(0xD2511F53u, c0);
        const uint32_t lo1 = 0xCD9E8D57u * c2, hi1 = mulhi32(0xCD9E8D57u, c2);
        const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    }
}

__host__ __device__ __forceinline__ void crng_init(CRng &s, uint64_t seed, int chain, int iter,
                                                   int slot, int purpose)
{
    s.k0 = (uint32_t)seed;
    s.k1 = (uint32_t)(seed >> 32);
    s.c0 = (uint32_t)iter;
    s.c1 = (uint32_t)slot;
    s.c2 = (uint32_t)purpose;
    s.c3 = (uint32_t)chain << 20;
    s.have = 0;
    s.tape = nullptr;
    s.tpos = 0;
    s.tover = nullptr;
}

__device__ __forceinline__ double crng_tape_next(CRng &s)
{
    double v = 0.5;
    if (s.tpos < SODAGPU_TAPE_W) v = s.tape[s.tpos];
    else if (s.tover) *s.tover = CRNG_TAPE_OVERRUN;
    ++s.tpos;
    return v;
}

// Computes the first Philox block of a draw site ahead of its first use (the
// counters do not depend on the data, so a kernel can do this before waiting
// for the kernel that produces them): crng_u64 then returns the same values.
__host__ __device__ __forceinline__ void crng_warm(CRng &s)
{
    if (s.have != 0 || s.tape) return;
    uint32_t a = s.c0, b = s.c1, c = s.c2, d = s.c3;
    philox4x32_10(a, b, c, d, s.k0, s.k1);
    s.c3++;
    s.o0 = a;
    s.o1 = b;
    s.o2 = c;
    s.o3 = d;
    s.have = 2;
}

__host__ __device__ __forceinline__ uint64_t crng_u64(CRng &s);

// Steps over the first n uniforms of a fresh stream.
__device__ __forceinline__ void crng_skip(CRng &s, int n)
{
    s.tpos += n;
    s.c3 += (uint32_t)(n >> 1);
    if (!s.tape && (n & 1)) crng_u64(s);
}

__host__ __device__ __forceinline__ uint64_t crng_u64(CRng &s)
{
    if (s.have == 2) {
        s.have = 1;
        return ((uint64_t)s.o1 << 32) | s.o0;
    }
    if (s.have == 0) {
        uint32_t a = s.c0, b = s.c1, c = s.c2, d = s.c3;
        philox4x32_10(a, b, c, d, s.k0, s.k1);
        s.c3++;
        s.o2 = c;
        s.o3 = d;
        s.have = 1;
        return ((uint64_t)b << 32) | a;
    }
    s.have = 0;
    return ((uint64_t)s.o3 << 32) | s.o2;
}

__host__ __device__ __forceinline__ double crng_unit(CRng &s)
{
#if defined(__CUDA_ARCH__)
    if (s.tape) return crng_tape_next(s);
#endif
    const uint64_t bits = 0x3FF0000000000000ULL | (crng_u64(s) >> 12);
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)bits) - 1.0;
#else
    double d;
    __builtin_memcpy(&d, &bits, sizeof d);
    return d - 1.0;
#endif
}

// ---------------------------------------------------------------------------
// FP32 uniforms of the reduced-precision sweeps (same counter streams): they
// take the top 24 bits of each word, offset by half a unit so they
// lie strictly inside (0,1): log(u) is always finite.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float crng_unit_f(CRng &s)
{
    if (s.tape) return (float)crng_tape_next(s);
    return ((float)(uint32_t)(crng_u64(s) >> 40) + 0.5f) * 5.9604644775390625e-8f;
}

// ---------------------------------------------------------------------------
// Distribution transforms, FP64 (the reference's) and FP32 with the same
// streams.  Each is in two parts, so that a kernel can take the uniforms and
// do the transcendental arithmetic before the mean, the standard deviation
// or the scale is known: the parts' values together are the plain draw's,
// bit for bit.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T crng_unit_t(CRng &s);
template <>
__device__ __forceinline__ double crng_unit_t<double>(CRng &s) { return crng_unit(s); }
template <>
__device__ __forceinline__ float crng_unit_t<float>(CRng &s) { return crng_unit_f(s); }

__device__ __forceinline__ double t_log(double x) { return log(x); }
__device__ __forceinline__ float t_log(float x) { return logf(x); }
__device__ __forceinline__ double t_exp(double x) { return exp(x); }
__device__ __forceinline__ float t_exp(float x) { return expf(x); }
__device__ __forceinline__ double t_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float t_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double t_sin(double x) { return sin(x); }
__device__ __forceinline__ float t_sin(float x) { return sinf(x); }
__device__ __forceinline__ double t_pow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float t_pow(float x, float y) { return powf(x, y); }

// rand_normal (parallelrng.f90:264-277): mean + sd * rr * sn; takes no
// uniforms when sd <= 0.
template <typename T>
struct NormalPre {
    T rr, sn;
};
template <typename T>
__device__ __forceinline__ NormalPre<T> normal_pre(CRng &s)
{
    const T u1 = crng_unit_t<T>(s), u2 = crng_unit_t<T>(s);
    NormalPre<T> z;
    z.rr = t_sqrt((T)-2.0 * t_log(u1));
    z.sn = t_sin((T)(2.0 * SODA_REF_PI) * u2);
    return z;
}
template <typename T>
__device__ __forceinline__ T normal_from(T mean, T sd, const NormalPre<T> &z)
{
    return mean + sd * z.rr * z.sn;
}
template <typename T>
__device__ __forceinline__ T t_rnorm(T mean, T sd, CRng &s)
{
    if (sd <= (T)0.0) return mean;
    return normal_from(mean, sd, normal_pre<T>(s));
}
__device__ __forceinline__ double d_rnorm(double mean, double sd, CRng &s) { return t_rnorm<double>(mean, sd, s); }

// rand_gamma (parallelrng.f90:294-333): scale * d * v, times w**(1/shape) for
// a shape below 1.  The rejection loop is bounded; on the (practically
// impossible) exhaustion *err is set and the last candidate kept.
template <typename T>
struct GammaPre {
    T d, v, wp;
    bool small;
    int taken;   // uniforms used: three when the first candidate is accepted and the shape is at least 1
};
template <typename T>
__device__ __forceinline__ GammaPre<T> gamma_pre(T shape, CRng &s, int *err)
{
    GammaPre<T> g;
    g.small = shape < (T)1.0;
    const T sh = g.small ? shape + (T)1.0 : shape;
    g.d = sh - (T)1.0 / (T)3.0;
    const T c = (T)1.0 / t_sqrt((T)9.0 * g.d);
    int tries = 0;
    g.taken = 0;
    for (;;) {
        T x = t_rnorm<T>((T)0.0, (T)1.0, s);
        T v = (T)1.0 + c * x;
        g.taken += 3;
        while (v <= (T)0.0 && tries < 100000) {
            x = t_rnorm<T>((T)0.0, (T)1.0, s);
            v = (T)1.0 + c * x;
            g.taken += 2;
            ++tries;
        }
        v = v * v * v;
        const T u = crng_unit_t<T>(s);
        const T xsq = x * x;
        g.v = v;
        if ((u < (T)1.0 - (T)0.0331 * xsq * xsq) ||
            (t_log(u) < (T)0.5 * xsq + g.d * ((T)1.0 - v + t_log(v))))
            break;
        if (++tries >= 100000) { if (err) *err = 1; break; }
    }
    g.wp = (T)1.0;
    if (g.small) {
        // shape < 1: g ~ gamma(shape+1, 1), then scale*g*w**(1/shape)
        const T w = crng_unit_t<T>(s);
        ++g.taken;
        g.wp = t_pow(w, (T)1.0 / shape);
    }
    return g;
}
template <typename T>
__device__ __forceinline__ T gamma_from(T scale, const GammaPre<T> &g)
{
    return g.small ? scale * (g.d * g.v) * g.wp : scale * g.d * g.v;
}
__device__ __forceinline__ double d_rgamma(double shape, double scale, CRng &s, int *err)
{
    return gamma_from(scale, gamma_pre<double>(shape, s, err));
}

// rand_scaled_inverse_chi_square (parallelrng.f90:348-362) from the gamma
// draw of shape dof / 2
template <typename T>
__device__ __forceinline__ T scinvchi2_from(T dof, T scale, const GammaPre<T> &g)
{
    const T sc = (T)0.5 * dof * scale;
    return (T)1.0 / gamma_from((T)1.0 / sc, g);
}
__device__ __forceinline__ double d_rscinvchi2(double dof, double scale, CRng &s, int *err)
{
    return scinvchi2_from(dof, scale, gamma_pre<double>(0.5 * dof, s, err));
}

}  // namespace soda

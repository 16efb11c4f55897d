// Device building blocks shared by the stochastic kernels.
//
// Random streams are Philox-4x32-10 (Salmon et al., SC'11), keyed by
// (seed, realisation) and counted by (draw, step seed, cell, phase|species|sweep),
// so every draw is a pure function of where it is used: the same results come out
// whatever the launch shape, tile size or batching (plain, wide or persistent).
//
// The elementary functions and samplers are written from the mathematics and
// evaluate a fixed sequence of IEEE single-precision operations (explicit fmaf,
// the file is compiled with -fmad=false), so a CPU replay gets the same bits:
//   log   x = m 2^e, log m = 2 atanh((m-1)/(m+1)), series to s^11
//   exp   x = k ln2 + r (two-part ln2), Taylor series to r^8
//   sin/cos(2 pi u)  quadrant reduction on u, Taylor series on [-pi/4, pi/4]
//   binomial  chunked inversion of the pmf recurrence, (1-q)^m by binary powering
//   Poisson   count of unit-rate exponential arrivals before lambda
#pragma once
#ifdef __CUDACC_RTC__
#include "gpgmp_rtc_prelude.h"    // run-time compilation: fixed-width types and limits
#else
#include <cstdint>
#include <climits>
#include <cuda_runtime.h>
#endif

namespace gpgmp {

constexpr uint32_t PH_INIT = 0x01000000u;
constexpr uint32_t PH_SSA = 0x02000000u;
constexpr uint32_t PH_DIFF = 0x03000000u;
constexpr uint32_t PH_SOURCE = 0x04000000u;
constexpr uint32_t PH_PART = 0x05000000u;
constexpr uint32_t PH_PAIR = 0x06000000u;
constexpr uint32_t PH_POP = 0x07000000u;    // population bookkeeping (individuals)

constexpr int SSA_EVENT_CAP = 1 << 22;
constexpr int SIM_EVENT_CAP = 1;
constexpr int SIM_OVERFLOW = 2;
constexpr int MAX_SPECIES = 32;
constexpr int MAX_REACTIONS = 128;

__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                       uint32_t k0, uint32_t k1, uint32_t out[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
#ifdef __CUDA_ARCH__
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
#else
        uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
#endif
        uint32_t n0 = hi1 ^ c1 ^ k0;
        uint32_t n2 = hi0 ^ c3 ^ k1;
        c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// A stream: key fixed, counter word 0 advances, four outputs buffered.
struct Stream {
    uint32_t k0, k1, c1, c2, c3, c0;
    uint32_t buf[4];
    int idx;
    __device__ __forceinline__ void init(uint32_t key0, uint32_t key1, uint32_t ctr1, uint32_t ctr2, uint32_t ctr3) {
        k0 = key0; k1 = key1; c1 = ctr1; c2 = ctr2; c3 = ctr3; c0 = 0u; idx = 4;
    }
    // the next four outputs at once; only where every draw so far came from block()
    __device__ __forceinline__ void block(uint32_t out[4]) {
        philox4x32_10(c0, c1, c2, c3, k0, k1, out);
        c0 += 1u;
    }
    __device__ __forceinline__ uint32_t next() {
        if (idx == 4) {
            philox4x32_10(c0, c1, c2, c3, k0, k1, buf);
            c0 += 1u;
            idx = 0;
        }
        uint32_t v;
        // constant-index selects keep buf in registers
        v = idx == 0 ? buf[0] : (idx == 1 ? buf[1] : (idx == 2 ? buf[2] : buf[3]));
        ++idx;
        return v;
    }
};

__device__ __forceinline__ float u01_open0(uint32_t x) { return (float)((x >> 8) + 1u) * 5.9604644775390625e-08f; }
__device__ __forceinline__ float u01(uint32_t x) { return (float)(x >> 8) * 5.9604644775390625e-08f; }

#define GPGMP_LN2_HI 0.693145751953125f
#define GPGMP_LN2_LO 1.4286068202862268e-06f

__device__ __forceinline__ float gp_logf(float x) {
    if (!(x > 0.0f)) return x == 0.0f ? -INFINITY : __int_as_float(0x7fc00000);
    if (isinf(x)) return x;
    uint32_t b = __float_as_uint(x);
    int e = 0;
    if ((b >> 23) == 0) {
        x = x * 16777216.0f;
        b = __float_as_uint(x);
        e = -24;
    }
    e += (int)((b >> 23) & 0xffu) - 127;
    float m = __uint_as_float((b & 0x007fffffu) | 0x3f800000u);
    if (m > 1.41421353816986083984375f) { m = m * 0.5f; e += 1; }
    float s = (m - 1.0f) / (m + 1.0f);
    float z = s * s;
    float p = fmaf(z, 2.0f / 11.0f, 2.0f / 9.0f);
    p = fmaf(z, p, 2.0f / 7.0f);
    p = fmaf(z, p, 2.0f / 5.0f);
    p = fmaf(z, p, 2.0f / 3.0f);
    p = fmaf(z, p, 2.0f);
    float lm = s * p;
    float fe = (float)e;
    return fmaf(fe, GPGMP_LN2_HI, fmaf(fe, GPGMP_LN2_LO, lm));
}

// a / b to the nearest, for a and b well inside the normal range (2^-60 < |b| < 2^60 and
// |a / b| > 2^-100 or a = 0): Newton's step on the approximate reciprocal gives the nearest
// reciprocal (compared for every significand of b; the instruction's error bound alone leaves
// a dozen in doubt), then Markstein's correction (1990, as div_small below) the nearest
// quotient.
__device__ __forceinline__ float div_mid(float a, float b) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    y = fmaf(fmaf(-b, y, 1.0f), y, y);
    const float q0 = a * y;
    return fmaf(fmaf(-q0, b, a), y, q0);
#else
    return a / b;
#endif
}

// gp_logf(u01_open0(x)), the same operations without the cases that a draw cannot reach
// (zero, subnormal, infinite): v = (x >> 8) + 1 in [1, 2^24] stands for v 2^-24, and one
// subtraction splits its bits into the exponent and a significand in (2^-1/2, 2^1/2].
// All 2^24 arguments give the bits of gp_logf.
__device__ __forceinline__ float log_draw(uint32_t x) {
    const uint32_t t = __float_as_uint((float)((x >> 8) + 1u)) - 0x3f3504f4u;
    const float m = __uint_as_float((t & 0x007fffffu) + 0x3f3504f4u);
    // (t >> 23) - 24 as a float, from the low bits of 1.5 2^23 + integer
    const float fe = __uint_as_float((t >> 23) + 0x4b400000u) - (12582912.0f + 24.0f);
    const float s = div_mid(m - 1.0f, m + 1.0f);
    const float z = s * s;
    float p = fmaf(z, 2.0f / 11.0f, 2.0f / 9.0f);
    p = fmaf(z, p, 2.0f / 7.0f);
    p = fmaf(z, p, 2.0f / 5.0f);
    p = fmaf(z, p, 2.0f / 3.0f);
    p = fmaf(z, p, 2.0f);
    const float lm = s * p;
    return fmaf(fe, GPGMP_LN2_HI, fmaf(fe, GPGMP_LN2_LO, lm));
}

__device__ __forceinline__ float gp_expf(float x) {
    if (x != x) return x;
    if (x > 88.5f) return INFINITY;
    if (x < -103.0f) return 0.0f;
    float kf = rintf(x * 1.4426950408889634f);
    float r = fmaf(-kf, GPGMP_LN2_HI, x);
    r = fmaf(-kf, GPGMP_LN2_LO, r);
    float p = fmaf(r, 1.0f / 40320.0f, 1.0f / 5040.0f);
    p = fmaf(r, p, 1.0f / 720.0f);
    p = fmaf(r, p, 1.0f / 120.0f);
    p = fmaf(r, p, 1.0f / 24.0f);
    p = fmaf(r, p, 1.0f / 6.0f);
    p = fmaf(r, p, 0.5f);
    p = fmaf(r, p, 1.0f);
    p = fmaf(r, p, 1.0f);
    int k = (int)kf;
    int k1 = k / 2, k2 = k - k1;
    float s1 = __uint_as_float((uint32_t)(k1 + 127) << 23);
    float s2 = __uint_as_float((uint32_t)(k2 + 127) << 23);
    return (p * s1) * s2;
}

__device__ __forceinline__ void gp_sincos2pi(float u, float* sn, float* cs) {
    float a = u * 4.0f;
    float qf = rintf(a);
    float d = a - qf;
    float y = d * 1.5707963267948966f;
    float z = y * y;
    float ps = fmaf(z, -1.0f / 39916800.0f, 1.0f / 362880.0f);
    ps = fmaf(z, ps, -1.0f / 5040.0f);
    ps = fmaf(z, ps, 1.0f / 120.0f);
    ps = fmaf(z, ps, -1.0f / 6.0f);
    float sy = fmaf(y * z, ps, y);
    float pc = fmaf(z, 1.0f / 479001600.0f, -1.0f / 3628800.0f);
    pc = fmaf(z, pc, 1.0f / 40320.0f);
    pc = fmaf(z, pc, -1.0f / 720.0f);
    pc = fmaf(z, pc, 1.0f / 24.0f);
    pc = fmaf(z, pc, -0.5f);
    float cy = fmaf(z, pc, 1.0f);
    // quadrant: odd ones swap sine and cosine, 2 and 3 negate the sine, 1 and 2 the cosine
    const uint32_t q = (uint32_t)(int)qf;
    const float s_ = q & 1u ? cy : sy, c_ = q & 1u ? sy : cy;
    *sn = __uint_as_float(__float_as_uint(s_) ^ ((q & 2u) << 30));
    *cs = __uint_as_float(__float_as_uint(c_) ^ (((q + 1u) & 2u) << 30));
}


// double-precision exp, same construction as gp_expf (two-part ln 2 with 21 trailing
// zero bits in the high part, Taylor series to r^13)
__device__ __forceinline__ double gp_exp_d(double x) {
    if (x != x) return x;
    if (x > 709.0) return INFINITY;
    if (x < -745.0) return 0.0;
    double kd = rint(x * 1.4426950408889634);
    double r = fma(-kd, 0.6931471803691238, x);
    r = fma(-kd, 1.9082149292705877e-10, r);
    double p = fma(r, 1.0 / 6227020800.0, 1.0 / 479001600.0);
    p = fma(r, p, 1.0 / 39916800.0);
    p = fma(r, p, 1.0 / 3628800.0);
    p = fma(r, p, 1.0 / 362880.0);
    p = fma(r, p, 1.0 / 40320.0);
    p = fma(r, p, 1.0 / 5040.0);
    p = fma(r, p, 1.0 / 720.0);
    p = fma(r, p, 1.0 / 120.0);
    p = fma(r, p, 1.0 / 24.0);
    p = fma(r, p, 1.0 / 6.0);
    p = fma(r, p, 0.5);
    p = fma(r, p, 1.0);
    p = fma(r, p, 1.0);
    int k = (int)kd;
    int k1 = k / 2, k2 = k - k1;
    double s1 = __longlong_as_double((long long)(k1 + 1023) << 52);
    double s2 = __longlong_as_double((long long)(k2 + 1023) << 52);
    return (p * s1) * s2;
}

__device__ __forceinline__ float gp_tanhf(float e) {
    float a = e < 0.0f ? -e : e;
    float t = gp_expf(-2.0f * a);
    float v = (1.0f - t) / (1.0f + t);
    return e < 0.0f ? -v : v;
}
__device__ __forceinline__ float gp_sinhf(float e) {
    float E = gp_expf(e);
    return (E - 1.0f / E) * 0.5f;
}

// Correctly rounded a / b for b = k + 1 = 1 .. kRecipMax, from the correctly rounded
// reciprocal y of b (Markstein 1990, "Computation of elementary functions on the IBM
// RISC System/6000 processor": with q0 = a y, the remainder a - q0 b is exact in one
// fused multiply-add and q0 + y (a - q0 b) rounds to a / b).  Checked against the
// division for every significand of a and every b of the table; it holds while the
// remainder does not underflow, |a| > 2^-100 (binomial_count says why that suffices).
constexpr int kRecipMax = 64, kRecipHead = 12;
#define GPGMP_RECIP4(i) 1.0f / (i), 1.0f / (i + 1), 1.0f / (i + 2), 1.0f / (i + 3)
#define GPGMP_RECIP16(i) GPGMP_RECIP4(i), GPGMP_RECIP4(i + 4), GPGMP_RECIP4(i + 8), GPGMP_RECIP4(i + 12)
static __constant__ float kRecip[kRecipMax] = {GPGMP_RECIP16(1.0f), GPGMP_RECIP16(17.0f), GPGMP_RECIP16(33.0f),
                                               GPGMP_RECIP16(49.0f)};
__device__ __forceinline__ float div_small(float a, float b, float y) {
    const float q0 = a * y;
    return fmaf(fmaf(-q0, b, a), y, q0);
}

// base^m by binary powering, least significant bit first
__device__ __forceinline__ float pow_int(float base, int m) {
    float f = (m & 1) ? base : 1.0f;
    int e = m >> 1;
    while (e) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {      // four bits per test; the bits past the top one are zero
            base = base * base;
            if (e & (1 << i)) f = f * base;
        }
        e >>= 4;
    }
    return f;
}

// The smallest k whose cumulative pmf of Binomial(m, q), m q <= 30, q <= 1/2, exceeds u
// (m where rounding leaves the sum at or below u): f = (1-q)^m, r = q / (1 - q), each
// term from the last by f (m - k) r / (k + 1).  The search was bound by the conversions
// of m - k and k + 1 and the reciprocal of the division, all three on the 16-lane
// special-function pipe (1M cells of Poisson(100) counts: 42 us for one species' jumps, 27
// now); here m - k counts down as a float (exact below 2^24) and the division by k + 1 is
// div_small.  f starts at or above 2^-61, grows to the mode and falls after it, so a
// term below 2^-100 only comes after cdf has passed 1/2 and changes neither cdf nor k:
// what div_small's remainder does there does not matter.
__device__ __forceinline__ int binomial_count(float u, int m, float f, float r) {
    int k = 0;
    float cdf = f;
    if (m < (1 << 24)) {
        float left = (float)m;
        // the first terms with their divisors as constants; past k = m the terms are zero,
        // so the test for it waits until after
#pragma unroll
        for (; k < kRecipHead; ++k) {
            if (u < cdf) break;
            f = div_small(f * (left * r), (float)(k + 1), 1.0f / (float)(k + 1));
            left -= 1.0f;
            cdf = cdf + f;
        }
        if (k == kRecipHead && m > kRecipHead) {
            const int kmax = m < kRecipMax ? m : kRecipMax;
            for (; k < kmax; ++k) {
                if (u < cdf) break;
                f = div_small(f * (left * r), (float)(k + 1), kRecip[k]);
                left -= 1.0f;
                cdf = cdf + f;
            }
        }
        k = k < m ? k : m;
    }
    while (u >= cdf && k < m) {
        f = f * ((float)(m - k) * r) / (float)(k + 1);
        k++;
        cdf = cdf + f;
    }
    return k;
}

// What a binomial draw needs from its probability p, worked out once where many draws
// share it: q / (1 - q), the counts per draw for q = min(p, 1 - p), and (1 - q)^(2^i) for
// the powers.
template <int BITS>
struct BinomialSetup {
    float sq[BITS], r;
    int chunk;
    int kind;      // 0: none (p <= 0 or NaN), 1: p <= 1/2, 2: p > 1/2 (counts those left), 3: all (p >= 1)
    __device__ __forceinline__ void init(float p) {
        kind = !(p > 0.0f) ? 0 : p >= 1.0f ? 3 : p > 0.5f ? 2 : 1;
        const float q = p > 0.5f ? 1.0f - p : p;
        sq[0] = 1.0f - q;
#pragma unroll
        for (int i = 1; i < BITS; ++i) sq[i] = sq[i - 1] * sq[i - 1];
        r = q / (1.0f - q);
        const float chunkf = 30.0f / q;
        chunk = chunkf >= 2147483520.0f ? INT_MAX : (int)chunkf;
        if (chunk < 1) chunk = 1;
    }
    // (1 - q)^m, the products of pow_int
    __device__ __forceinline__ float power(int m) const {
        if (m >= (1 << BITS)) return pow_int(sq[0], m);
        float f = (m & 1) ? sq[0] : 1.0f;
#pragma unroll
        for (int i = 1; i < BITS; ++i) f = f * ((m & (1 << i)) ? sq[i] : 1.0f);
        return f;
    }
    // n from one draw: whether n needs at most one, and its count (n > 0, kind 1 or 2)
    __device__ __forceinline__ bool single(int n) const { return n <= chunk && kind != 3; }
    __device__ __forceinline__ int count(uint32_t draw, int n) const {
        const int k = binomial_count(u01(draw), n, power(n), r);
        return kind == 2 ? n - k : k;
    }
};
// The same for one probability of a whole block, with the first powers in a table.
struct BinomialTable : BinomialSetup<1> {
    const float* table;      // (1 - q)^m for m < size, in shared memory
    int size;
    __device__ __forceinline__ float power(int m) const { return m < size ? table[m] : pow_int(sq[0], m); }
    __device__ __forceinline__ int count(uint32_t draw, int n) const {
        const int k = binomial_count(u01(draw), n, power(n), r);
        return kind == 2 ? n - k : k;
    }
};
template <int BITS>
__device__ __forceinline__ int binomial(Stream& st, int n, const BinomialSetup<BITS>& b) {
    if (n <= 0 || b.kind == 0) return 0;
    if (b.kind == 3) return n;
    int rem = n, total = 0;
    while (rem > 0) {
        const int m = rem < b.chunk ? rem : b.chunk;
        total += binomial_count(u01(st.next()), m, pow_int(b.sq[0], m), b.r);
        rem -= m;
    }
    return b.kind == 2 ? n - total : total;
}
__device__ __forceinline__ int binomial(Stream& st, int n, float p) {
    if (n <= 0 || !(p > 0.0f)) return 0;
    BinomialSetup<1> b;
    b.init(p);
    return binomial(st, n, b);
}

// Unit-rate arrivals before lam: the times are the running sums of -log_draw, each rounded,
// and the count is how many of them stay at or below lam.
__device__ __forceinline__ int poisson_exact(Stream& st, float lam) {
    int k = 0;
    float t = 0.0f;
    for (;;) {
        uint32_t w[4];
        st.block(w);
        float a[4];      // the logarithms are independent, only the sums are a chain
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = log_draw(w[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            t = t - a[i];
            if (t > lam) return k;
            k++;
            if (k == INT_MAX) return k;
        }
    }
}

__device__ __forceinline__ float log2_approx(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The same count with a bound instead of the sums: most blocks lie well below lam, and for
// them one approximate logarithm of the four draws' product tells that all four arrivals
// count.  `off` bounds how far the approximate time can be from the rounded running sum, in
// 2^-24: each running sum is rounded by at most its own size (4 a block, at most the block's
// last) and so is the approximate one (5 sum), log_draw and lg2.approx are off by at most 8
// and 4 of the time, and a block's product and an argument near 1 add 6; all of it doubled.
// An arrival within that of lam (one cell in a thousand at lam = 100) sends the cell to
// poisson_exact, and from lam = 256 on, where it would be one in a hundred, all cells.  Two
// species at lam = 100 on 1M cells: 400 us, now 257; at lam = 50 on 8.4M cells 1.68 ms, now
// 0.96.
__device__ __forceinline__ int poisson(Stream& st, float lam) {
    if (!(lam > 0.0f)) return 0;
    const Stream from = st;
    if (lam < 256.0f) {
        constexpr float kLn2 = 0.6931471806f, kScale = 5.9604644775390625e-08f;      // 2^-24
        float t = 0.0f, sum = 0.0f, blocks = 0.0f;
        int k = 0;
        for (;;) {
            uint32_t w[4];
            st.block(w);
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = (float)((w[i] >> 8) + 1u);
            const float p = ((v[0] * v[1]) * (v[2] * v[3])) * 1.262177448353619e-29f;      // 2^-96
            const float t4 = fmaf(-kLn2, log2_approx(p), t);
            sum += t4;
            blocks += 1.0f;
            const float off = 2.0f * kScale * fmaf(5.0f, sum, fmaf(12.0f, t4, fmaf(6.0f, blocks, 16.0f)));
            if (t4 + off <= lam) {
                t = t4;
                k += 4;
                continue;
            }
            bool sure = true;
            int more = -1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                t = fmaf(-kLn2, log2_approx(v[i] * kScale), t);
                if (more < 0) {
                    sure = sure && fabsf(t - lam) > off;
                    if (t > lam) more = i;
                }
            }
            if (sure && more >= 0) return k + more;
            break;
        }
    }
    st = from;
    return poisson_exact(st, lam);
}

// two normals from two draws (Box-Muller)
__device__ __forceinline__ void normal2(uint32_t w0, uint32_t w1, float* z0, float* z1) {
    float rad = sqrtf(-2.0f * log_draw(w0));
    float s, c;
    gp_sincos2pi(u01(w1), &s, &c);
    *z0 = rad * c;
    *z1 = rad * s;
}

}  // namespace gpgmp

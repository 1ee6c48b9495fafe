// lbm_noise.cuh -- seeded Gaussian perturbation of the initial populations.
//
// N(0,1) samples per (seed, site): Philox4x32-10 (Salmon, Moraes, Dror,
// Shaw, SC'11) on the counter (site_lo, site_hi, block, 0) gives four 32-bit
// words; each pair of words is one Box-Muller draw (Box and Muller, 1958):
// a radius sqrt(-2 ln u1) from 23 bits of the first word, an angle from 24
// bits of the second, and the pair (r cos theta, r sin theta).  Block g
// feeds sample pairs 2g and 2g+1; populations 2m and 2m+1 of a site take
// pair m.  The logarithm is summed from the atanh series, sine and cosine
// from their Taylor series on a quarter turn (Horner steps as fused
// multiply-adds).  Every floating-point step is an explicit single-precision
// operation or fma with the IEEE result (no contraction left to the compiler, no
// library transcendental; the division and the square root start from
// approximations and are corrected with exact remainders), so a CPU
// implementation of the same recipe gets the same bits.  Single precision because FP64 runs at a small fraction of the FP32
// rate on GB300 and the samples only perturb the initial state.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lbm {

__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[0], p1 = (uint64_t)0xCD9E8D57u * c[2];
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0;
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1;
        c[0] = n0;
        c[1] = (uint32_t)p1;
        c[2] = n2;
        c[3] = (uint32_t)p0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// The exponent / mantissa split of the logarithm of a normal x in (0, 1):
// x = m 2^e with m in [sqrt(1/2), sqrt(2)); returns m and the float of e
// (2^23 + 2^22 + e as a float's bits, then the 2^23 + 2^22 taken off: exact,
// and no conversion instruction, of which the GPU runs 16 lanes a cycle).
__device__ __forceinline__ void log_split(float x, float &m, float &fe)
{
    const unsigned bits = __float_as_uint(x);
    unsigned e = (bits >> 23) + (0x4b400000u - 127u);
    m = __uint_as_float((bits & 0x007fffffu) | 0x3f800000u);
    if (m > 1.41421354f) {
        m = __fmul_rn(m, 0.5f);
        e += 1;
    }
    fe = __fadd_rn(__uint_as_float(e), -12582912.0f);
}

// Both Box-Muller draws of a Philox block at once on packed FP32 pairs
// (lane .x from words 0, 1; lane .y from words 2, 3).  Every product that
// feeds a sum is an explicit fused multiply-add (one rounding, the CPU's
// fmaf), every other operation an IEEE add / multiply (lane-wise, as the
// scalar ones), division and square root correctly rounded: no step is left
// for the compiler to fuse, so the CPU recipe gives the same bits.
__device__ __forceinline__ float2 nz_f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 nz_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 nz_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 nz_fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Correctly rounded a / b (b in [1.7, 2.42], |a| < 1/2) and sqrt(a) (a in [2^-24,
// 34)): the hardware's approximate reciprocal (square root), one Newton step,
// and the quotient (root) corrected with its exact remainder (P. W. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Develop. 34 (1990)).  The arguments both take here are functions
// of the 2^23 values of u1: checked for every one of them against the IEEE
// division and square root.  Those, with their special cases, and the
// conversions of integers took a fifth of the kernel: 256^3 0.76 -> 0.60 ms (223
// instructions for four samples, issue slots 74% busy), 512^3 FP16
// initialisation 7.7 -> 6.7 ms.
__device__ __forceinline__ float2 nz_div(float2 a, float2 b)
{
    const float2 nb = make_float2(-b.x, -b.y);
    float2 y = make_float2(__fdividef(1.0f, b.x), __fdividef(1.0f, b.y));
    y = nz_fma(y, nz_fma(nb, y, nz_f2(1.0f)), y);
    const float2 q = nz_mul(a, y);
    return nz_fma(nz_fma(nb, q, a), y, q);
}
__device__ __forceinline__ float2 nz_sqrt(float2 a)
{
    float2 y = make_float2(rsqrtf(a.x), rsqrtf(a.y));
    const float2 s = nz_mul(a, y), h = nz_mul(nz_f2(0.5f), y);
    // r = 1/2 - h s: both halves of the coupled Newton step
    const float2 r = nz_fma(make_float2(-h.x, -h.y), s, nz_f2(0.5f));
    const float2 s1 = nz_fma(s, r, s), h1 = nz_fma(h, r, h);
    return nz_fma(nz_fma(make_float2(-s1.x, -s1.y), s1, a), h1, s1);
}

// ln x = e ln 2 + 2 s (1 + s^2/3 + ... + s^12/13), s = (m-1)/(m+1)
// (|s| <= 0.1716: truncation below 1e-9)
__device__ __forceinline__ float2 series_logf2(float2 x)
{
    float2 m, fe;
    log_split(x.x, m.x, fe.x);
    log_split(x.y, m.y, fe.y);
    const float2 num = nz_add(m, nz_f2(-1.0f)), den = nz_add(m, nz_f2(1.0f));
    const float2 s = nz_div(num, den);
    const float2 s2 = nz_mul(s, s);
    // 1 / (2k + 1), folded at compile time to the correctly rounded floats
    constexpr float inv_odd[7] = {1.0f / 1.0f, 1.0f / 3.0f, 1.0f / 5.0f,  1.0f / 7.0f,
                                  1.0f / 9.0f, 1.0f / 11.0f, 1.0f / 13.0f};
    float2 acc = nz_f2(inv_odd[6]);
#pragma unroll
    for (int k = 5; k >= 0; --k) acc = nz_fma(s2, acc, nz_f2(inv_odd[k]));
    const float ln2 = 0.693147182f;
    return nz_fma(nz_mul(nz_f2(2.0f), s), acc, nz_mul(fe, nz_f2(ln2)));
}

// cos and sin of the angle 2 pi (k / 4 + 1 / 8) + x, x in (-pi/4, pi/4), k in
// 0..3: the Taylor series of cos x (to x^10) and sin x (to x^9), the rotation
// by pi/4 to pi/4 + x, then the quarter turn k (per lane).
__device__ __forceinline__ void quarter_turn_cs2(uint32_t k0, uint32_t k1, float2 x, float2 &c, float2 &s)
{
    const float2 x2 = nz_mul(x, x);
    float2 sp = nz_f2(1.0f / 362880.0f);
    sp = nz_fma(x2, sp, nz_f2(-1.0f / 5040.0f));
    sp = nz_fma(x2, sp, nz_f2(1.0f / 120.0f));
    sp = nz_fma(x2, sp, nz_f2(-1.0f / 6.0f));
    const float2 sn = nz_fma(nz_mul(x, x2), sp, x);
    float2 cp = nz_f2(-1.0f / 3628800.0f);
    cp = nz_fma(x2, cp, nz_f2(1.0f / 40320.0f));
    cp = nz_fma(x2, cp, nz_f2(-1.0f / 720.0f));
    cp = nz_fma(x2, cp, nz_f2(1.0f / 24.0f));
    cp = nz_fma(x2, cp, nz_f2(-0.5f));
    const float2 cs = nz_fma(x2, cp, nz_f2(1.0f));
    const float2 h = nz_f2(0.707106781f);  // sqrt(1/2)
    const float2 c0 = nz_mul(h, nz_add(cs, make_float2(-sn.x, -sn.y))), s0 = nz_mul(h, nz_add(cs, sn));
    // the quarter turn: an odd k swaps the two, cos changes sign for k = 1, 2,
    // sin for k = 2, 3
    c.x = __uint_as_float(__float_as_uint(k0 & 1 ? s0.x : c0.x) ^ ((k0 + 1) & 2) << 30);
    s.x = __uint_as_float(__float_as_uint(k0 & 1 ? c0.x : s0.x) ^ (k0 & 2) << 30);
    c.y = __uint_as_float(__float_as_uint(k1 & 1 ? s0.y : c0.y) ^ ((k1 + 1) & 2) << 30);
    s.y = __uint_as_float(__float_as_uint(k1 & 1 ? c0.y : s0.y) ^ (k1 & 2) << 30);
}

// Two Box-Muller pairs from the four words: u1 = (w >> 9 + 1/2) / 2^23 in
// (0, 1) (exact), the angle's quarter turn from the top two bits of the
// partner word and its offset in the quarter from the next 22,
// (f + 1/2) / 2^22 (exact); r = sqrt(-2 ln u1), samples (r cos, r sin).
__device__ __forceinline__ void box_muller2(const uint32_t (&w)[4], float (&z)[4])
{
    // v + 1/2 of a 23- (22-) bit v: 2^23 + v as a float's bits, less 2^23 - 1/2
    const auto half_up = [](uint32_t v0, uint32_t v1) {
        return nz_add(make_float2(__uint_as_float(0x4b000000u | v0), __uint_as_float(0x4b000000u | v1)),
                      nz_f2(-8388607.5f));
    };
    const float2 u1 = nz_mul(half_up(w[0] >> 9, w[2] >> 9), nz_f2(1.0f / 8388608.0f));
    const float2 r = nz_sqrt(nz_mul(nz_f2(-2.0f), series_logf2(u1)));
    const float2 fq = nz_mul(half_up((w[1] >> 8) & 0x3fffffu, (w[3] >> 8) & 0x3fffffu), nz_f2(1.0f / 4194304.0f));
    const float2 x = nz_mul(nz_add(fq, nz_f2(-0.5f)), nz_f2(1.57079637f));  // (fq - 1/2) pi/2
    float2 c, s;
    quarter_turn_cs2(w[1] >> 30, w[3] >> 30, x, c, s);
    const float2 zc = nz_mul(r, c), zs = nz_mul(r, s);
    z[0] = zc.x;
    z[1] = zs.x;
    z[2] = zc.y;
    z[3] = zs.y;
}

// The four samples of block g of a site: pairs 2g (z[0], z[1]) and 2g + 1
// (z[2], z[3]).
__device__ __forceinline__ void gauss_block(uint64_t seed, uint64_t site, uint32_t g, float (&z)[4])
{
    uint32_t c[4] = {(uint32_t)site, (uint32_t)(site >> 32), g, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    box_muller2(c, z);
}

}  // namespace lbm

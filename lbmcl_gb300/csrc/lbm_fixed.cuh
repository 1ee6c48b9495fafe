// lbm_fixed.cuh -- the FP64 FLUID update with most of its additions (and the
// products by 3 and 4.5) in 64-bit integers, bit for bit the update in IEEE
// double operations (moments_exact, relax_exact).
//
// Bound: the FP64 pipe.  GB300 runs an FP64 operation for one warp in 16 to 20
// cycles per SM, and 64 to 128 lanes of integer adds, logic or products a
// cycle beside it; the update is 260 FP64 operations a site in IEEE operations,
// 80 here, and 4,500 integer instructions.  256^3: 7767 -> 3470 us per
// iteration (2110 -> 4722 MLUPS, 9% -> 21% of HBM), 64^3 133 -> 62.9, 32^3 19.6 ->
// 12.0 (ncu at 256^3: FP64 pipe 61% active, integer pipe 70%).  Left out, against
// 3777 before the warps left the windows together: the last sum of every
// population on the FP64 pipe too (19 operations more, a seventh of the integer
// instructions less) 4436; 254 registers, 8 warps per SM instead of 16, 4698; 80
// registers with spills 3779.
//
// Between values whose binary exponents are known to lie in a small
// window, an IEEE addition is an integer addition and one rounding to 53
// significant bits, ten or so integer instructions.  What stays on the FP64
// pipe: the products that need 106 bits, the six sums of velocity components,
// three differences of momenta and three divisions (one shared reciprocal).
//
// Fixed point: unit 2^-61 in an unsigned 64-bit word.  A double in [2^-8, 4) is
// an exact multiple of it with at least 54 bits, so at least one bit is dropped
// by every rounding below (t >= 1).  Smaller values enter with their lost bits
// jammed into the lowest one ("round to odd"): where they do, at least two bits
// are dropped, so the lowest one only has to say "not exact".
//
// The windows (f_0 in [2^-8, 1), f_i in [2^-8, 1/4), 2^-10 <= 1/tau < 64; then
// rho in [7/8, 2), |u_x|, |u_y|, |u_z| < 1/8; then feq - f a double, as it is within
// a factor of two, |feq - f| / tau < 1/2, new f in [2^-7, 2)) hold for flows well
// inside the low-Mach range of the scheme.  Beyond the first the update is IEEE
// operations (260), beyond the others its relaxation is (170 beside the 18 of
// the moments here), so that a site outside takes no longer than without all
// this: 256^3 with |u| = 0.15 everywhere 5933 us per iteration, rho = 2.5 5935,
// IEEE operations alone 8431 (both updates one after the other 9663, 9089).  The
// lanes of a warp leave together: some inside and some outside would run both.
#pragma once

#include "lbm_device.cuh"

namespace lbm {
namespace fx {

using u64 = unsigned long long;
constexpr u64 ONE = 1ull << 61;

__device__ __forceinline__ unsigned hi32(u64 x) { return (unsigned)(x >> 32); }
__device__ __forceinline__ unsigned lo32(u64 x) { return (unsigned)x; }
__device__ __forceinline__ u64 make64(unsigned hi, unsigned lo) { return ((u64)hi << 32) | lo; }
__device__ __forceinline__ u64 bits(double v) { return (u64)__double_as_longlong(v); }
__device__ __forceinline__ double value(u64 b) { return __longlong_as_double((long long)b); }

// bits dropped when S >= 2^53 is rounded to 53 significant ones
__device__ __forceinline__ int drop(u64 S) { return 11 - __clz((int)hi32(S)); }

// S plus what makes truncation of its t lowest bits round to nearest, ties to
// even (t >= 1)
__device__ __forceinline__ u64 nearest(u64 S, int t)
{
    return S + (u64)((1u << (t - 1)) - 1u + ((lo32(S) >> t) & 1u));
}

// S rounded to 53 significant bits
__device__ __forceinline__ u64 round53(u64 S)
{
    const int t = drop(S);
    const u64 R = nearest(S, t);
    return make64(hi32(R), lo32(R) & (~0u << t));
}

// the double nearest to S 2^-61 (a carry out of the mantissa lands in the
// exponent, as it should)
__device__ __forceinline__ double to_double(u64 S)
{
    const int t = drop(S);
    const u64 m = nearest(S, t) >> t;
    return value(make64(hi32(m) + ((unsigned)(t + 1013) << 20), lo32(m)));
}

// x 2^k, k < 32: multiplications, whose pipe the other integer operations
// leave idle
__device__ __forceinline__ u64 shl(u64 x, unsigned k)
{
    const unsigned p = 1u << k;
    const u64 l = (u64)lo32(x) * p;
    return make64(hi32(x) * p + hi32(l), lo32(l));
}

// v in [2^-8, 4): exact
__device__ __forceinline__ u64 exact(double v)
{
    const u64 b = bits(v);
    const u64 m = make64((hi32(b) & 0xfffffu) | 0x100000u, lo32(b));
    return shl(m, (hi32(b) >> 20) - 1014u);
}

// m 2^(e - 1075) (m < 2^53 or 2^53 itself, e <= 1022), truncated, lost bits
// jammed into the lowest
__device__ __forceinline__ u64 jam(u64 m, int e)
{
    const u64 M = shl(m, 10);
    const int s = min(1024 - e, 63);
    const u64 X = M >> s;
    return X | (u64)((X << s) != M);
}
// |v| < 1/2, not subnormal (v = 0 is fine)
__device__ __forceinline__ u64 jam(double v)
{
    const u64 b = bits(v);
    const unsigned e = (hi32(b) >> 20) & 0x7ffu;
    return jam(make64((hi32(b) & 0xfffffu) | (e ? 0x100000u : 0u), lo32(b)), (int)e);
}

// Over the populations of a site so far, for one check of the windows: the bits
// that a difference feq - f has beyond 53 (its 11 lowest ones), the largest
// change and the smallest and largest new population (high words)
struct Extremes {
    unsigned lost = 0, change = 0, least = 0xffffffffu, most = 0;
};

// Correctly rounded x / r, y / r, z / r for r in [2^-4, 8), |x|, |y|, |z| zero
// or in [2^-64, 8), from one reciprocal: a single-precision seed, three Newton
// steps, then q = x c and q + (x - r q) c with exact remainders.  After the
// third step c is the reciprocal correctly rounded, unless r's mantissa is all
// ones (its reciprocal lies an ulp above the power of two the step returns),
// and the corrected quotient then is the correctly rounded one (P. W.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Develop. 34 (1990)).  15 FP64 operations; three IEEE
// divisions take about 42.
__device__ __forceinline__ void quotients(double x, double y, double z, double r, double &qx, double &qy, double &qz)
{
    const u64 b = bits(r);
    // r truncated to single precision and the seed back to double: both exact
    // in the exponent range of r, as integer operations
    const unsigned fb = ((hi32(b) - (896u << 20)) << 3) | (lo32(b) >> 29);
    const unsigned gb = __float_as_uint(__frcp_rn(__uint_as_float(fb)));
    double c = value(make64((gb >> 3) + (896u << 20), gb << 29));
    c = __fma_rn(c, __fma_rn(-r, c, 1.0), c);  // 2^-22 -> 2^-44
    c = __fma_rn(c, __fma_rn(-r, c, 1.0), c);  // within an ulp
    c = __fma_rn(c, __fma_rn(-r, c, 1.0), c);  // correctly rounded, unless r's mantissa is all ones
    if (lo32(b) == 0xffffffffu && (hi32(b) & 0xfffffu) == 0xfffffu) c = value(make64((2045u - (hi32(b) >> 20)) << 20, 1));
    const double px = __dmul_rn(x, c), py = __dmul_rn(y, c), pz = __dmul_rn(z, c);
    qx = __fma_rn(__fma_rn(-r, px, x), c, px);
    qy = __fma_rn(__fma_rn(-r, py, y), c, py);
    qz = __fma_rn(__fma_rn(-r, pz, z), c, pz);
}

// f + inv_tau (feq - f), f as F in fixed point, feq in [2^-8, 4)
__device__ __forceinline__ double relaxed(double feq, u64 F, double inv_tau, Extremes &x)
{
    const long long D = (long long)(exact(feq) - F);  // exact
    const bool neg = D < 0;
    const u64 A = neg ? (u64)-D : (u64)D;
    // A as a double
    const int z = hi32(A) ? __clz((int)hi32(A)) : 32 + __clz((int)lo32(A));
    const u64 n = A << (z & 63);
    x.lost |= lo32(n);
    const u64 m = n >> 11;
    const u64 d = A ? make64(hi32(m) + ((unsigned)(1024 - z) << 20), lo32(m)) : 0ull;
    const double g = __dmul_rn(inv_tau, value(d));
    x.change = max(x.change, hi32(bits(g)));
    const u64 M = jam(g);
    const u64 S = neg ? F - M : F + M;
    x.least = min(x.least, hi32(S));
    x.most = max(x.most, hi32(S));
    return to_double(S);
}

// What fluid did: nothing (f as it was), the moments (f not valid), or the
// moments and the update.
enum Done { NOTHING, MOMENTS, UPDATE };

// Does any lane of the warp (of those here) say so?
__device__ __forceinline__ bool any(bool p) { return __any_sync(__activemask(), p); }

// The BGK update of a FLUID site (f in and out) and its moments, as far as the
// windows let it.
__device__ __forceinline__ Done fluid(double (&f)[Q], double inv_tau, const Weights<double> &W, double &r_, double &ux_,
                                      double &uy_, double &uz_)
{
    unsigned least = hi32(bits(f[1])), most = least;
#pragma unroll
    for (int i = 2; i < Q; ++i) {
        least = min(least, hi32(bits(f[i])));
        most = max(most, hi32(bits(f[i])));
    }
    // (a set sign makes a high word larger than any of these bounds)
    if (any(least < (1015u << 20) || most >= (1021u << 20) || hi32(bits(f[0])) - (1015u << 20) >= (8u << 20) ||
            hi32(bits(inv_tau)) - (1013u << 20) >= (16u << 20)))
        return NOTHING;
    u64 F[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) F[i] = exact(f[i]);
    // moments in moments_exact's order
    u64 R = F[0];
#pragma unroll
    for (int i = 1; i < Q - 1; ++i) R = round53(R + F[i]);
    const double r = to_double(R + F[Q - 1]);
    const double px = to_double(round53(round53(round53(F[1] + F[7]) + F[10]) + F[11]) + F[15]);
    const double mx = to_double(round53(round53(round53(F[3] + F[8]) + F[9]) + F[13]) + F[17]);
    const double py = to_double(round53(round53(round53(F[2] + F[7]) + F[8]) + F[12]) + F[16]);
    const double my = to_double(round53(round53(round53(F[4] + F[9]) + F[10]) + F[14]) + F[18]);
    const double pz = to_double(round53(round53(round53(F[6] + F[15]) + F[16]) + F[17]) + F[18]);
    const double mz = to_double(round53(round53(round53(F[5] + F[11]) + F[12]) + F[13]) + F[14]);
    double ux, uy, uz;
    // (r is at least 19 2^-8 and below 5.5; a difference is a multiple of 2^-61)
    quotients(__dsub_rn(px, mx), __dsub_rn(py, my), __dsub_rn(pz, mz), r, ux, uy, uz);
    r_ = r;
    ux_ = ux;
    uy_ = uy;
    uz_ = uz;
    const unsigned top = 1020u << 20;  // 1/8
    // rho in [7/8, 2): with |u_i| < 1/8 every bracket is at least 0.46 and
    // every feq at least 0.011
    if (any((hi32(bits(ux)) & 0x7fffffffu) >= top || (hi32(bits(uy)) & 0x7fffffffu) >= top ||
            (hi32(bits(uz)) & 0x7fffffffu) >= top || hi32(bits(r)) - 0x3fec0000u >= 0x40000000u - 0x3fec0000u))
        return MOMENTS;
    Extremes x;
    const double u2 = __dadd_rn(__dadd_rn(__dmul_rn(ux, ux), __dmul_rn(uy, uy)), __dmul_rn(uz, uz));
    const u64 C = jam(__dmul_rn(1.5, u2));
    const double rw[3] = {__dmul_rn(r, W.w[0]), __dmul_rn(r, W.w[1]), __dmul_rn(r, W.w[2])};
    f[0] = relaxed(__dmul_rn(rw[0], to_double(ONE - C)), F[0], inv_tau, x);
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        const int j = opp_of(i);
        if (j < i) continue;
        const double eu = proj_exact(i, ux, uy, uz);
        const u64 b = bits(eu);
        const unsigned sign = hi32(b) & 0x80000000u, e = (hi32(b) >> 20) & 0x7ffu;
        const u64 m = make64((hi32(b) & 0xfffffu) | 0x100000u, lo32(b));
        // (a subnormal eu gives what zero gives)
        // |3 eu|: 3 m has 54 or 55 bits
        const u64 m3 = 3 * m;
        const int t3 = 1 + (int)(hi32(m3) >> 22);
        const u64 T = e ? jam(nearest(m3, t3) >> t3, (int)e + t3) : 0ull;
        // 4.5 eu: 9 m has 56 or 57 bits
        const u64 m9 = 9 * m;
        const int t9 = 3 + (int)(hi32(m9) >> 24);
        const u64 n9 = nearest(m9, t9) >> t9;
        const u64 h = e ? make64((hi32(n9) + ((e + t9 - 2) << 20)) | sign, lo32(n9)) : make64(sign, 0);
        const u64 SQ = jam(__dmul_rn(value(h), eu));
        const double plus = to_double(round53(round53(ONE + T) + SQ) - C);
        const double minus = to_double(round53(round53(ONE - T) + SQ) - C);
        const double w = rw[wclass_of(i)];
        f[i] = relaxed(__dmul_rn(w, sign ? minus : plus), F[i], inv_tau, x);
        f[j] = relaxed(__dmul_rn(w, sign ? plus : minus), F[j], inv_tau, x);
        // (most sites that fail below fail here)
        if (any((x.lost & 0x7ffu) != 0)) return MOMENTS;
    }
    // every feq - f a double, every change below 1/2, 2^-7 <= new f (two bits
    // dropped) < 2
    const bool ok = x.change < (1022u << 20) && x.least >= (1u << 22) && x.most < (1u << 30);
    return any(!ok) ? MOMENTS : UPDATE;
}

}  // namespace fx
}  // namespace lbm

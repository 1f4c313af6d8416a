// ieee64.cuh — correctly rounded FP64 division and square root with most of the
// work on the FP32 and integer pipes.
//
// An FP64 instruction of a warp takes 64 cycles on this GPU, and a / b is about
// seven of them, sqrt(x) seven and a half.  Here the operands' mantissas are cut
// into pairs of FP32 numbers, the quotient (root) is formed from an FP32
// reciprocal (reciprocal root) and one correction to about 2^-44, and three FP64
// instructions do the rest: the residual of that estimate, its correction, and
// the residual r of the corrected value q.  q is the correctly rounded quotient
// exactly when |a - q b| is at most half a unit in q's last place times b, and r
// is that difference without rounding error, so the test is an integer
// comparison; the few operands that fail it (about one in ten thousand), that lie
// outside 2^-500 .. 2^500, or whose result is a power of two (where the spacing
// changes) are left to the instruction sequence of the language's operators.  So
// every result has the bits of a / b and sqrt(x).
//
// Measured, cycles per warp and SM sub-partition with 16 warps on an SM: div64
// 295, a / b 566; sqrt64 and an addition 354, sqrt(x) and an addition 650.  A
// single warp: 419 / 562 and 501 / 688.
#pragma once

#include <cuda_runtime.h>

namespace mafm {
namespace {

__device__ __noinline__ double div64_any(double a, double b) { return a / b; }
__device__ __noinline__ double sqrt64_any(double x) { return sqrt(x); }

// The mantissa of a double in [1, 2) as an FP32 pair: 24 leading bits and the
// next 23 (what is left is below 2^-46).
__device__ __forceinline__ void mantissa32(int hi, int lo, float& h, float& l) {
    h = __int_as_float(0x3f800000 | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29));
    l = __fmul_rn(__fsub_rn(__int_as_float(0x3f800000 | ((lo & 0x1fffffff) >> 6)), 1.0f), 1.1920928955078125e-7f);
}

// A positive normal float as a double.
__device__ __forceinline__ double widen(float x) {
    const int b = __float_as_int(x);
    return __hiloint2double((b >> 3) + (896 << 20), b << 29);
}

// h + l as a double for h in [0.5, 4) and |l| < 2^-20 h: l in units of h's last
// place as a double, added to its bits.
__device__ __forceinline__ double join(float h, float l) {
    const int b = __float_as_int(h);
    const int units = __float2int_rn(__fmul_rn(l, __int_as_float(((127 + 52 + 127) << 23) - (b & 0x7f800000))));
    const long long w = (((long long)((b >> 3) + (896 << 20)) << 32) | (unsigned)(b << 29)) + units;
    return __longlong_as_double(w);
}

// Exponent field within 500 of the bias.
__device__ __forceinline__ bool middling(int hi) { return (unsigned)(((hi >> 20) & 0x7ff) - 523) <= 1000u; }

// a / b
__device__ __forceinline__ double div64(double a, double b) {
    const int ah = __double2hiint(a), al = __double2loint(a), bh = __double2hiint(b), bl = __double2loint(b);
    float am, an, bm, bn;
    mantissa32(ah, al, am, an);
    mantissa32(bh, bl, bm, bn);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(bm));
    const float e = __fmaf_rn(-bn, y, __fmaf_rn(-bm, y, 1.0f));
    const float ph = __fmul_rn(am, y);
    float pl = __fmaf_rn(am, y, -ph);
    pl = __fmaf_rn(am, __fmul_rn(y, e), pl);
    pl = __fmaf_rn(an, y, pl);
    const double A = __hiloint2double((ah & 0xfffff) | 0x3ff00000, al), B = __hiloint2double((bh & 0xfffff) | 0x3ff00000, bl);
    const double q0 = join(ph, pl);
    const double q = __fma_rn(__fma_rn(-q0, B, A), widen(y), q0);
    const double r = __fma_rn(-q, B, A);
    // half a unit in the last place of q, times B
    const int qh = __double2hiint(q), ql = __double2loint(q);
    const long long bound = __double_as_longlong(B) + ((long long)((qh & 0x7ff00000) - ((1023 + 53) << 20)) << 32);
    const bool ok = middling(ah) && middling(bh) && (__double_as_longlong(r) & 0x7fffffffffffffffll) <= bound &&
                    ((qh & 0xfffff) | ql) != 0;
    if (!ok) return div64_any(a, b);
    // exponent difference and sign
    return __hiloint2double(qh + ((ah & 0x7ff00000) - (bh & 0x7ff00000)) ^ ((ah ^ bh) & 0x80000000), ql);
}

// sqrt(x)
__device__ __forceinline__ double sqrt64(double x) {
    const int xh = __double2hiint(x), xl = __double2loint(x);
    // mantissa in [1, 4): an odd exponent leaves one factor 2 in it
    const int odd = ~(xh >> 20) & 1;           // the bias 1023 is odd
    float m, n;
    mantissa32(xh, xl, m, n);
    const float two = odd ? 2.0f : 1.0f;
    m = __fmul_rn(m, two);
    n = __fmul_rn(n, two);
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(m));
    const float sh = __fmul_rn(m, y), hy = __fmul_rn(y, 0.5f);
    const float sl = __fmul_rn(__fadd_rn(__fmaf_rn(-sh, sh, m), n), hy);
    const double X = __hiloint2double((xh & 0xfffff) | (odd ? 0x40000000 : 0x3ff00000), xl);
    const double s0 = join(sh, sl);
    const double s = __fma_rn(__fma_rn(-s0, s0, X), widen(hy), s0);
    const double r = __fma_rn(-s, s, X);
    // (s - u / 2)^2 < X < (s + u / 2)^2 with u = 2^-52, s in (1, 2): -s u < r <= s u
    const int hs = __double2hiint(s), ls = __double2loint(s);
    const long long bound = __double_as_longlong(s) - (52ll << 52), rb = __double_as_longlong(r);
    const long long mag = rb & 0x7fffffffffffffffll;
    const bool ok = xh >= 0 && middling(xh) && (rb < 0 ? mag < bound : mag <= bound) && (hs >> 20) == 1023 &&
                    ((hs & 0xfffff) | ls) != 0;
    if (!ok) return sqrt64_any(x);
    // (exponent of x - exponent of X) / 2
    return __hiloint2double(hs + ((((xh >> 20) - 1023 - odd) >> 1) << 20), ls);
}

}  // namespace
}  // namespace mafm

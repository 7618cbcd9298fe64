// ieee_int.cuh -- IEEE double products and quotients on the integer pipe.
//
// GB300 issues one FP64 warp instruction per ~62 cycles and SM sub-partition,
// while its integer pipe and wide multipliers run beside FP64 work.  A
// correctly rounded product is 25 instructions (4 wide multiplies), a quotient
// 40 from its divisor's reciprocal, which takes another 20.  Measured (24
// warps per SM, 8 independent chains per thread, in units of one FP64
// product): integer product 0.55 alone; one FP64 and one integer product
// together 1.00; __ddiv_rn 7.3; integer quotient with its reciprocal 1.08
// alone, 1.13 together with an FP64 product.
//
// Every function returns the round-to-nearest-even result IEEE 754 prescribes
// for operands inside its guard (normal operands whose result is normal or
// overflows by rounding); the callers send other operands to the FP64 pipe.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PCRP_FN __host__ __device__ __forceinline__
#else
#include <cstring>
#define PCRP_FN inline
#endif

namespace pcrp {
namespace ieee {

PCRP_FN uint32_t hi(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    __builtin_memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
PCRP_FN uint32_t lo(double x)
{
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    __builtin_memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}
PCRP_FN double make(uint32_t h, uint32_t l)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)h, (int)l);
#else
    const uint64_t u = ((uint64_t)h << 32) | l;
    double d;
    __builtin_memcpy(&d, &u, 8);
    return d;
#endif
}
// high word of (h:l) << n, n < 32
PCRP_FN uint32_t shl(uint32_t l, uint32_t h, uint32_t n)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(l, h, n);
#else
    return n ? (h << n) | (l >> (32 - n)) : h;
#endif
}
PCRP_FN uint32_t mant_hi(uint32_t h) { return (h & 0xFFFFFu) | 0x100000u; }

// ---------------------------------------------------------------------------
// products x*y, several y per factor x
// ---------------------------------------------------------------------------
struct Factor {
    uint32_t l, m;          // mantissa: low word, high 21 bits
    uint32_t se;            // sign and exponent fields, less the bias and one
};

PCRP_FN Factor factor(double x)
{
    const uint32_t h = hi(x);
    return {lo(x), mant_hi(h), (h & 0xFFF00000u) - (1024u << 20)};
}

// Both exponent fields in [513, 1533]: the product's is in [3, 2044].  (`mul`
// takes any two normal factors whose fields sum to between 1024 and 3068: the
// product's field is in [1, 2046], or it overflows by rounding.)
PCRP_FN bool mid(double x) { return (hi(x) << 1) - (513u << 21) < (1021u << 21); }

// Guard of many operands at once: `off(x)` is below 2^30 iff x's exponent
// field is in [623, 1134] (2^-400 <= |x| < 2^112), so `fits` of the or of
// several tests them all.  Quotients of such operands are normal, their
// exponent field in [511, 1535] (2^-512 < |q| <= 2^512), and so are products of
// a quotient with one, [111, 1647]: inside what `div` and `mul` take, though a
// quotient at either end is outside `mid`.  The window reaches further down than up because the couplings
// of diagonally dominant systems square with every stride.
PCRP_FN uint32_t off(double x) { return hi(x) * 2u - (623u << 21); }
PCRP_FN bool fits(uint32_t offs) { return offs < (1u << 30); }

// x*y for normal x, y with a normal product (see `mid`).  The 105- or 106-bit product of the
// mantissas is formed in 32-bit words w3:w2:w1:w0, shifted left by 12 or 11
// so that its upper words hold the 53 result bits and the next one the rest,
// and rounded to nearest even: up iff the rest, with "odd, or more below"
// or-ed into its last bit (its low 11 bits are zero), exceeds one half.  The
// carry runs through the mantissa into the exponent field.
PCRP_FN double mul(const Factor& f, double y)
{
    const uint32_t h = hi(y), l = lo(y), m = mant_hi(h);
    const uint64_t t0 = (uint64_t)f.l * l, t3 = (uint64_t)f.m * m;
    const uint64_t s = (uint64_t)f.m * l + (uint64_t)f.l * m;   // < 2^54
    uint32_t w1, w2, w3;
#ifdef __CUDA_ARCH__
    asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, %6;\n\taddc.u32 %2, %7, 0;"
        : "=&r"(w1), "=&r"(w2), "=r"(w3)
        : "r"((uint32_t)s), "r"((uint32_t)(t0 >> 32)), "r"((uint32_t)(s >> 32)), "r"((uint32_t)t3),
          "r"((uint32_t)(t3 >> 32)));
#else
    const uint64_t u = s + (t0 >> 32), v = t3 + (u >> 32);
    w1 = (uint32_t)u; w2 = (uint32_t)v; w3 = (uint32_t)(v >> 32);
#endif
    const uint32_t top = w3 >> 9, n = 12u - top;
    const uint32_t below = (uint32_t)t0 < 1u ? (uint32_t)t0 : 1u;
    uint32_t rh = shl(w2, w3, n), rl = shl(w1, w2, n);
    const uint32_t rest = (w1 << n) | ((rl & 1u) | below);
    const uint32_t se = (h & 0xFFF00000u) + (top << 20) + f.se;
#ifdef __CUDA_ARCH__
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, 0x7FFFFFFF;\n\taddc.cc.u32 %0, %0, 0;\n\taddc.u32 %1, %1, %3;\n\t}"
        : "+r"(rl), "+r"(rh) : "r"(rest), "r"(se));
#else
    const uint64_t r = (((uint64_t)rh << 32) | rl) + (rest > 0x80000000u ? 1u : 0u);
    rl = (uint32_t)r; rh = (uint32_t)(r >> 32) + se;
#endif
    return make(rh, rl);
}

// ---------------------------------------------------------------------------
// quotients x/y from a reciprocal of y
// ---------------------------------------------------------------------------

// About 2^63 / Y, Y the top 32 bits of y's mantissa shifted to 64: never
// above 2^95 / (mantissa of y << 11), at most 5 below it.  A single-precision
// reciprocal of the top 24 bits and one Newton step; any bits for y that is
// not normal (the caller's guard keeps them unused).
PCRP_FN uint32_t recip(double y)
{
    const uint32_t Y = shl(lo(y), mant_hi(hi(y)), 11);
    uint32_t b = ((Y >> 8) & 0x7FFFFFu) | 0x3F800000u;          // in [1, 2)
#ifdef __CUDA_ARCH__
    float g;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"(__uint_as_float(b)));
    b = min(__float_as_uint(g), 0x3F7FFFFFu);                   // in [1/2, 1)
#else
    float g;
    __builtin_memcpy(&g, &b, 4);
    g = 1.0f / g;
    __builtin_memcpy(&b, &g, 4);
    if (b > 0x3F7FFFFFu) b = 0x3F7FFFFFu;
#endif
    const uint32_t G = b * 256u + 0x80000000u;                  // 2^63 / Y to ~2^-22.5
    const int64_t e = (int64_t)((uint64_t(1) << 63) - (uint64_t)G * Y);
    const int64_t c = (int64_t)(int32_t)(e >> 10) * (int64_t)(G >> 1);   // G e / 2^63, times 2^52
    return G + (uint32_t)((int32_t)(c >> 32) >> 20) - 3u;
}

// Both operands inside `mid`, or else exponent fields in [100, 1946] and
// within 900 of each other: everything the quotient below touches is normal.
PCRP_FN bool div_guard(double x, double y)
{
    if (mid(x) && mid(y)) return true;
    const int ex = (int)((hi(x) >> 20) & 0x7FFu), ey = (int)((hi(y) >> 20) & 0x7FFu);
    return (unsigned)(ex - 100) <= 1846u && (unsigned)(ey - 100) <= 1846u && (unsigned)(ex - ey + 900) <= 1800u;
}

// x/y inside div_guard, G = recip(y): with X, Y the mantissas (X doubled if
// below Y), q1 = the first 31 bits of X/Y (short by at most 7), the exact
// remainder, q2 = the next 22 bits (short by at most 1), twice the exact
// remainder again, and one comparison with Y that rounds to nearest.  (A
// quotient of two 53-bit mantissas is never a midpoint, so nearest-even needs
// no tie rule.)  Remainders are sums with -Y modulo 2^64.
PCRP_FN double div(double x, double y, uint32_t G)
{
    const uint32_t xh = hi(x), yh = hi(y);
    uint64_t X = ((uint64_t)mant_hi(xh) << 32) | lo(x);
    const uint64_t Y = ((uint64_t)mant_hi(yh) << 32) | lo(y), N = 0 - Y;
    uint32_t se = (xh & 0xFFF00000u) - (yh & 0xFFF00000u) + (1022u << 20);
    if (X < Y) { X <<= 1; se -= 1u << 20; }
    const uint32_t nl = (uint32_t)N, nh = (uint32_t)(N >> 32);
    const uint32_t q1 = (uint32_t)(((uint64_t)(uint32_t)(X >> 22) * G) >> 32);
    uint64_t r = (uint64_t)q1 * nl + (X << 30);                 // X 2^30 - q1 Y < 8 Y
    r += (uint64_t)(q1 * nh) << 32;
    const uint32_t q2 = (uint32_t)(((uint64_t)(uint32_t)(r >> 25) * G) >> 32) >> 5;
    uint64_t d = (uint64_t)(2u * q2) * nl + (r << 23);          // 2 (r 2^22 - q2 Y) < 2.4 Y
    d += (uint64_t)(2u * q2 * nh) << 32;
    uint32_t rl = q1 << 22, rh = q1 >> 10;
#ifdef __CUDA_ARCH__
    // (2 * remainder >= Y: the sum with -Y carries out)
    asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 t, %4, %5;\n\t"
        "addc.cc.u32 %0, %0, %6;\n\taddc.u32 %1, %1, %7;\n\t}"
        : "+r"(rl), "+r"(rh)
        : "r"((uint32_t)d), "r"(nl), "r"((uint32_t)(d >> 32)), "r"(nh), "r"(q2), "r"(se));
#else
    const uint64_t q = (((uint64_t)rh << 32) | rl) + q2 + (d >= Y ? 1u : 0u);
    rl = (uint32_t)q; rh = (uint32_t)(q >> 32) + se;
#endif
    return make(rh, rl);
}

// x/y of any size: x finite and not zero, y normal; false if the result
// overflows or an operand is outside that.  The quotient above with its
// remainder, rounded at the place its exponent gives (subnormal results
// included).  For the few quotients outside div_guard.
PCRP_FN bool div_any(double x, double y, double& q)
{
    const uint32_t xh = hi(x), yh = hi(y);
    int ex = (int)((xh >> 20) & 0x7FFu);
    const int ey = (int)((yh >> 20) & 0x7FFu);
    uint64_t X = ((uint64_t)(xh & 0xFFFFFu) << 32) | lo(x);
    const uint64_t Y = ((uint64_t)mant_hi(yh) << 32) | lo(y);
    if (ex == 0x7FF || ey == 0 || ey == 0x7FF) return false;
    if (ex == 0) {
        if (X == 0) return false;
#ifdef __CUDA_ARCH__
        const int n = __clzll((long long)X) - 11;
#else
        const int n = __builtin_clzll(X) - 11;
#endif
        X <<= n;
        ex = 1 - n;
    } else {
        X |= uint64_t(1) << 52;
    }
    const uint32_t lt = X < Y;
    X <<= lt;
    const uint32_t G = recip(y);
    const uint32_t q1 = (uint32_t)(((uint64_t)(uint32_t)(X >> 22) * G) >> 32);
    uint64_t r = (X << 30) - (uint64_t)q1 * Y;
    const uint32_t q2 = (uint32_t)(((uint64_t)(uint32_t)(r >> 25) * G) >> 32) >> 5;
    r = (r << 22) - (uint64_t)q2 * Y;
    uint64_t Q = ((uint64_t)q1 << 22) + q2;                     // floor of the quotient, or one less
    if (r >= Y) { r -= Y; Q++; }
    const int E = ex - ey + 1023 - (int)lt;
    uint64_t bits;
    if (E >= 1) {
        if (E > 2046) return false;
        bits = ((uint64_t)(E - 1) << 52) + Q + (2 * r > Y ? 1u : 0u);
    } else if (E < -53) {
        bits = 0;
    } else {
        const int n = 1 - E;                                    // 1 .. 54
        const uint64_t rest = Q & ((uint64_t(1) << n) - 1), half = uint64_t(1) << (n - 1);
        bits = Q >> n;
        bits += rest > half || (rest == half && (r != 0 || (bits & 1)));
    }
    q = make((uint32_t)(bits >> 32) | ((xh ^ yh) & 0x80000000u), (uint32_t)bits);
    return true;
}

}  // namespace ieee
}  // namespace pcrp

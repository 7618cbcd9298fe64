// pcr_tile.cuh -- the faithful FP64 PCR-Penta work of one CTA (shared by the
// uniform-batch kernels of pcr_f64.cu and the persistent ragged kernel).
// The arithmetic and its correspondence with the reference are described at
// the top of pcr_f64.cu.
#pragma once
#include "ieee_int.cuh"
#include "pcrp_internal.h"
#include "tma.cuh"

namespace pcrp {

__device__ __forceinline__ double mul(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ double add(double x, double y) { return __dadd_rn(x, y); }
__device__ __forceinline__ double sub(double x, double y) { return __dsub_rn(x, y); }
// Bits of x other than the sign, OR-folded into one word: zero exactly for
// +-0.  Written in PTX on the two 32-bit halves so that it stays on the
// integer pipe (the equivalent C bit test can be turned into an FP64 compare,
// which here takes a slot of the FP64 pipe).
__device__ __forceinline__ unsigned magbits(double x) {
    unsigned r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\tshl.b32 hi, hi, 1;\n\tor.b32 %0, hi, lo;\n\t}"
        : "=r"(r) : "d"(x));
    return r;
}
// x != 0.0 (false for +-0, true for everything else including NaN)
__device__ __forceinline__ bool nz(double x) { return magbits(x) != 0u; }
// -x by flipping the sign bit on the integer pipe (bit-identical to unary
// minus), in PTX for the same reason as magbits
__device__ __forceinline__ double neg(double x) {
    double r;
    asm("{\n\t.reg .b32 lo, hi;\n\tmov.b64 {lo, hi}, %1;\n\txor.b32 hi, hi, 0x80000000;\n\tmov.b64 %0, {lo, hi};\n\t}"
        : "=d"(r) : "d"(x));
    return r;
}

// Exact IEEE results of operations with a zero operand, formed on the
// integer pipe (an FP64 operation costs ~40 integer operations of pipe time
// here), for the strides after the outer coefficients have decayed to zero.
__device__ __forceinline__ unsigned hiw(double x) { return (unsigned)__double2hiint(x); }
// the zero whose sign is bit 31 of s
__device__ __forceinline__ double szero(unsigned s) { return __hiloint2double((int)(s & 0x80000000u), 0); }
// x + z for a zero z with sign bit zs, x not NaN: x itself, unless x is a
// zero too (then -0 only if both are -0: round-to-nearest)
__device__ __forceinline__ double add_z(double x, unsigned zs) { return nz(x) ? x : szero(hiw(x) & zs); }
// x / y, IEEE round-to-nearest, off the main path: a zero x over a nonzero
// finite y is the signed zero IEEE 754 prescribes; then the integer quotient
// of any size; the FP64 division for the rest (infinities, nans, zero and
// subnormal divisors, overflow).
static __device__ __noinline__ double dvd(double x, double y) {
    if (!nz(x) && nz(y) && (hiw(y) & 0x7FF00000u) != 0x7FF00000u) return szero(hiw(x) ^ hiw(y));
    double q;
    if (ieee::div_any(x, y, q)) return q;
    return __ddiv_rn(x, y);
}
// x / y from G = ieee::recip(y) on the integer pipe where both operands are
// inside its guard; other operands take dvd.
__device__ __forceinline__ double quot(double x, double y, uint32_t G) {
    if (ieee::div_guard(x, y)) return ieee::div(x, y, G);
    return dvd(x, y);
}
__device__ __forceinline__ double quot(double x, double y) { return quot(x, y, ieee::recip(y)); }

// z - x for a zero z with sign bit zs, x not NaN
__device__ __forceinline__ double sub_z(unsigned zs, double x) { return nz(x) ? neg(x) : szero(zs & ~hiw(x)); }
// every one of the values +-0 / finite
__device__ __forceinline__ bool zeros(double x, double y, double z) {
    return (magbits(x) | magbits(y) | magbits(z)) == 0u;
}
__device__ __forceinline__ unsigned expw(double x) { return hiw(x) & 0x7FF00000u; }
__device__ __forceinline__ bool finite6(double p, double q, double r, double s, double t, double u) {
    return max(max(max(expw(p), expw(q)), max(expw(r), expw(s))), max(expw(t), expw(u))) < 0x7FF00000u;
}
__device__ __forceinline__ bool finite4(double p, double q, double r, double s) {
    return max(max(expw(p), expw(q)), max(expw(r), expw(s))) < 0x7FF00000u;
}

constexpr int kMaxThreads = 256;
constexpr int kMaxRowsPerThread = 8;
// Lanes of a warp whose rows take different cases run one after the other, and
// a row that no case takes runs the general form after its tests.  Where such
// rows lie among others away from the ends (scattered zeros, rows scaled far
// apart, exact zero pivots), the general form for all rows of the warp is
// cheaper than the cases and then that.  So a warp that met one away from the
// ends sends all its rows there in the next kGeneralStrides strides of the
// phase, and then tries the cases again (1: a third of the gain lost; for the
// rest of a pass: 2 % more lost where outer coefficients underflow unevenly).
// In phase A the rows without a case wait for a loop of their own, so that
// those of a thread's two rows run together (inline 1-2 % slower); in phase B
// that loop cost weakly dominant batches 1-2 % (m=64 n=2^20 34.2 against 33.75
// ms, m=256 n=65536 8.80 against 8.61).  us, without any of this and now:
// 2 % zeros among a, b, d, e and y, m=300 n=2049 945 -> 493, m=256 n=4096 1408
// -> 740; small integers with exact zero pivots, m=256 n=4096 1189 -> 753; rows
// scaled by up to 2^+-400 1306 -> 959; dense rows m=300 n=2049 457 -> 437,
// m=64 n=2^20 33.9 -> 33.75 ms, 20000 ragged systems of 8 to 64 rows 1.53 -> 1.21.
constexpr int kGeneralStrides = 3;

// ---------------------------------------------------------------------------
// One row of a stride, straight-line per case
// ---------------------------------------------------------------------------
// The row updates below give the bits of the reference's operations
// (Reductions I-III, kernel.cu:63-140) for one case of operands each; they
// return false, with nothing written, for rows outside their case, and those
// rows take the general form in pcr_tile.  In every case the quotients and
// most products run on the integer pipe (ieee_int.cuh), the sums and phase
// B's rhs products on the FP64 pipe: per row and stride 36 products and sums
// and 4 quotients, of which 16 sums and 2 products stay FP64.  A rhs is often
// zero, which is outside the integer product's guard: phase A's dense case
// decides for its two (m=256 n=65536 7.92 -> 7.82 ms); for phase B's as well
// the same decision gains on one-sided batches what it costs on dense ones.
// No other branch inside a case: with a branch per operation the chains of a
// row serialise (measured: 14.0 against 13.2 ms for m=16 n=2^20).
//
// A multiplier of a side (left: row - dl, right: row + dl) is "active" when
// it is a nonzero quotient inside the guard.  Otherwise it is a zero (its
// numerator is zero, or the row two steps out does not exist) or the side
// itself is missing; then every product with it is a zero whose sign is the
// factors' sign xor, adding it leaves a nonzero term alone, and no FP64
// operation is issued for that side.  This covers the ends of a (sub)system
// (in a whole-system tile the last two strides consist of them), one-sided
// and tridiagonal batches (a or e zero), and the late strides of diagonally
// dominant systems, whose outer coefficients underflow to zero.
template <int CAP>
struct TileRows {
    double a[CAP], b[CAP], c[CAP], d[CAP], e[CAP], y[CAP];            // state
    double Ta[CAP], Tb[CAP], Tc[CAP], Td[CAP], Te[CAP], Ty[CAP];      // T(m)
    uint32_t Tr[CAP];                                                 // ieee::recip of Tc
};

// signs (bit 31) of the products of a zero multiplier of sign s with a row
struct Signs { unsigned a, b, c, d, e, y; };

// Phase A, both multipliers active.  The rhs first, the reciprocal last: the
// other order 1 % slower (m=16 n=2^20 8.67 against 8.59 ms).
template <int CAP>
__device__ __forceinline__ bool row_a_both(TileRows<CAP>& t, int k, int dl, double& cT)
{
    const int l = k - dl, r = k + dl;
    const double am = t.a[k], em = t.e[k];
    const double aL = t.a[l], bL = t.b[l], cL = t.c[l], dL = t.d[l], eL = t.e[l];
    const double aR = t.a[r], bR = t.b[r], cR = t.c[r], dR = t.d[r], eR = t.e[r];
    const unsigned w = ieee::off(am) | ieee::off(em) | ieee::off(aL) | ieee::off(bL) | ieee::off(cL) | ieee::off(dL) |
                       ieee::off(eL) | ieee::off(aR) | ieee::off(bR) | ieee::off(cR) | ieee::off(dR) | ieee::off(eR);
    if (!ieee::fits(w)) return false;
    const double al1 = ieee::div(neg(am), bL, ieee::recip(bL)), al2 = ieee::div(neg(em), dR, ieee::recip(dR));
    const ieee::Factor f1 = ieee::factor(al1), f2 = ieee::factor(al2);
    const double yl = t.y[l], yr = t.y[r];
    double y1, y2;
    if (ieee::fits(ieee::off(yl) | ieee::off(yr))) { y1 = ieee::mul(f1, yl); y2 = ieee::mul(f2, yr); }
    else { y1 = mul(al1, yl); y2 = mul(al2, yr); }
    t.Ty[k] = add(add(y1, t.y[k]), y2);
    cT = add(add(ieee::mul(f1, dL), t.c[k]), ieee::mul(f2, bR));
    t.Tc[k] = cT;
    t.Tb[k] = add(add(ieee::mul(f1, cL), t.b[k]), ieee::mul(f2, aR));
    t.Td[k] = add(add(ieee::mul(f1, eL), t.d[k]), ieee::mul(f2, cR));
    t.Ta[k] = ieee::mul(f1, aL);
    t.Te[k] = ieee::mul(f2, eR);
    t.Tr[k] = ieee::recip(cT);
    return true;
}

// A multiplier num/piv of any size; false for a zero pivot.
__device__ __forceinline__ bool tiny_quotient(double num, double piv, uint32_t G, double& f)
{
    if (!nz(piv)) return false;
    f = quot(num, piv, G);
    return true;
}
// f*x cannot change a sum with c (|f*x| < 2^-54 |c|, or f*x a zero and c
// not): from the exponent fields, x finite, c inside `mid`
__device__ __forceinline__ bool absorbed(double f, double x, double c)
{
    return expw(x) < 0x7FF00000u && expw(f) < (1100u << 20) && ieee::mid(c) && expw(f) + expw(x) + (55u << 20) <= expw(c) + (1022u << 20);
}

// Phase A once the couplings are tiny (al1*dL, al2*bR and the rhs products
// too small to change the row's c and y): the quotients as above, cT and the
// rhs are the row's own, the other products and sums on the FP64 pipe, whose
// subnormal and zero results need no case of their own.  A missing side adds
// -0, which changes nothing.
template <int CAP>
__device__ __forceinline__ bool row_a_tiny(TileRows<CAP>& t, int k, int dl, bool hasL, bool has2L, bool hasR, bool has2R, double& cT)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double cm = t.c[k], ym = t.y[k];
    double al1 = 0.0, al2 = 0.0;
    if (has2L && !tiny_quotient(neg(t.a[k]), t.b[l], ieee::recip(t.b[l]), al1)) return false;
    if (has2R && !tiny_quotient(neg(t.e[k]), t.d[r], ieee::recip(t.d[r]), al2)) return false;
    if (!(absorbed(al1, t.d[l], cm) && absorbed(al1, t.y[l], ym) && absorbed(al2, t.b[r], cm) &&
          absorbed(al2, t.y[r], ym))) return false;
    const double m0 = szero(~0u);
    t.Tb[k] = hasL ? add(add(mul(al1, t.c[l]), t.b[k]), hasR ? mul(al2, t.a[r]) : m0) : 0.0;
    t.Td[k] = hasR ? add(add(hasL ? mul(al1, t.e[l]) : m0, t.d[k]), mul(al2, t.c[r])) : 0.0;
    t.Ta[k] = hasL ? mul(al1, t.a[l]) : 0.0;
    t.Te[k] = hasR ? mul(al2, t.e[r]) : 0.0;
    cT = cm;
    t.Tc[k] = cm; t.Ty[k] = ym;
    t.Tr[k] = ieee::recip(cm);
    return true;
}

// Zero multiplier of phase A towards row q (l or r): its sign, and the signs
// of its products with that row; false if it is not a zero or a factor is not
// finite.  num: the row's numerator, piv: row q's pivot, has2: the row two
// steps out exists (else the multiplier is +0).
template <int CAP>
__device__ __forceinline__ bool zero_side(TileRows<CAP>& t, int q, bool has2, double num, double piv, unsigned& s,
                                          Signs& g)
{
    if (has2 && nz(num)) return false;
    const double qa = t.a[q], qb = t.b[q], qc = t.c[q], qd = t.d[q], qe = t.e[q], qy = t.y[q];
    if (!finite6(qa, qb, qc, qd, qe, qy)) return false;
    s = has2 && nz(piv) ? hiw(num) ^ hiw(piv) ^ 0x80000000u : 0u;
    g = {s ^ hiw(qa), s ^ hiw(qb), s ^ hiw(qc), s ^ hiw(qd), s ^ hiw(qe), s ^ hiw(qy)};
    return true;
}

// A missing side adds nothing, which is what adding -0 does.
__device__ __forceinline__ Signs absent() { return {~0u, ~0u, ~0u, ~0u, ~0u, ~0u}; }

// Phase A of a row with both sides, one multiplier active and the other one a
// zero: the right one active, or the mirror image in the same code (a and e,
// b and d exchanged; the zero terms may be added in any order).  One-sided
// batches (a = 0 from upwind differences, for instance).
template <int CAP>
__device__ __forceinline__ bool row_a_one(TileRows<CAP>& t, int k, int dl, bool right, double& cT)
{
    const int q = right ? k + dl : k - dl, o = right ? k - dl : k + dl;
    // inner and outer coefficients of the active side (in, out) and the other (io, oo)
    const double* in = right ? t.d : t.b;
    const double* io = right ? t.b : t.d;
    const double* out = right ? t.e : t.a;
    const double* oo = right ? t.a : t.e;
    const double num = out[k], piv = in[q], p1 = io[q], p2 = t.c[q], p4 = out[q];
    if (!ieee::fits(ieee::off(num) | ieee::off(piv) | ieee::off(p1) | ieee::off(p2) | ieee::off(p4))) return false;
    unsigned s;
    Signs g;
    if (!zero_side(t, o, true, oo[k], io[o], s, g)) return false;
    const double al = ieee::div(neg(num), piv, ieee::recip(piv));
    const ieee::Factor f = ieee::factor(al);
    cT = add(add_z(t.c[k], right ? g.d : g.b), ieee::mul(f, p1));
    const double inner = add(add_z(in[k], right ? g.e : g.a), ieee::mul(f, p2));   // dT (bT)
    const double across = add(add_z(io[k], g.c), mul(al, oo[q]));                  // bT (dT)
    const double far = ieee::mul(f, p4), near = szero(right ? g.a : g.e);          // eT, aT (aT, eT)
    t.Tc[k] = cT;
    t.Tr[k] = ieee::recip(cT);
    t.Ty[k] = add(add_z(t.y[k], g.y), mul(al, t.y[q]));
    t.Tb[k] = right ? across : inner; t.Td[k] = right ? inner : across;
    t.Ta[k] = right ? near : far;     t.Te[k] = right ? far : near;
    return true;
}

// Phase A, neither multiplier active (at least one side present): no FP64
// operation at all.
template <int CAP>
__device__ __forceinline__ bool row_a_none(TileRows<CAP>& t, int k, int dl, bool hasL, bool has2L, bool hasR, bool has2R, double& cT)
{
    unsigned s1 = 0u, s2 = 0u;
    Signs g1 = absent(), g2 = absent();
    if (hasL && !zero_side(t, k - dl, has2L, t.a[k], t.b[k - dl], s1, g1)) return false;
    if (hasR && !zero_side(t, k + dl, has2R, t.e[k], t.d[k + dl], s2, g2)) return false;
    cT = add_z(add_z(t.c[k], g1.d), g2.b);
    t.Tc[k] = cT;
    t.Tr[k] = ieee::recip(cT);
    t.Tb[k] = hasL ? add_z(add_z(t.b[k], g1.c), g2.a) : 0.0;
    t.Td[k] = hasR ? add_z(add_z(t.d[k], g1.e), g2.c) : 0.0;
    t.Ty[k] = add_z(add_z(t.y[k], g1.y), g2.y);
    t.Ta[k] = hasL ? szero(g1.a) : 0.0;
    t.Te[k] = hasR ? szero(g2.e) : 0.0;
    return true;
}

// The same for a row with both sides whose b, c, d and y are not zero, in a
// tile without infinities and nans: T(m) is the row itself, and of the
// neighbours only the signs that a and e inherit are read (12 reads and 6
// tests of the neighbours less).
template <int CAP>
__device__ __forceinline__ bool row_a_self(TileRows<CAP>& t, int k, int dl, bool has2L, bool has2R, double& cT)
{
    const double b = t.b[k], c = t.c[k], d = t.d[k], y = t.y[k], bL = t.b[k - dl], dR = t.d[k + dl];
    if (!(nz(b) && nz(c) && nz(d) && nz(y))) return false;
    const unsigned s1 = has2L && nz(bL) ? hiw(t.a[k]) ^ hiw(bL) ^ 0x80000000u : 0u;
    const unsigned s2 = has2R && nz(dR) ? hiw(t.e[k]) ^ hiw(dR) ^ 0x80000000u : 0u;
    cT = c;
    t.Tc[k] = c;
    t.Tr[k] = ieee::recip(c);
    t.Tb[k] = b; t.Td[k] = d; t.Ty[k] = y;
    t.Ta[k] = szero(s1 ^ hiw(t.a[k - dl]));
    t.Te[k] = szero(s2 ^ hiw(t.e[k + dl]));
    return true;
}

// The same with zeros among b, c, d and y (the ends of the system, sparse
// right-hand sides), or a side missing: a zero takes its sign from the products
// added to it.  Zeros of c and y used to take row_a_none with its tests of both
// neighbours (us, one nonzero right-hand side value per system, 777 systems of
// 3001 rows 706 -> 634).
template <int CAP>
__device__ __forceinline__ bool row_a_tri(TileRows<CAP>& t, int k, int dl, bool hasL, bool has2L, bool hasR, bool has2R, double& cT)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double b = t.b[k], c = t.c[k], d = t.d[k], y = t.y[k], bL = t.b[l], dR = t.d[r];
    const unsigned s1 = has2L && nz(bL) ? hiw(t.a[k]) ^ hiw(bL) ^ 0x80000000u : 0u;
    const unsigned s2 = has2R && nz(dR) ? hiw(t.e[k]) ^ hiw(dR) ^ 0x80000000u : 0u;
    // (a missing side adds -0)
    const unsigned zb = (hasL ? s1 ^ hiw(t.c[l]) : ~0u) & (hasR ? s2 ^ hiw(t.a[r]) : ~0u);
    const unsigned zd = (hasL ? s1 ^ hiw(t.e[l]) : ~0u) & (hasR ? s2 ^ hiw(t.c[r]) : ~0u);
    cT = nz(c) ? c : szero(hiw(c) & (hasL ? s1 ^ hiw(t.d[l]) : ~0u) & (hasR ? s2 ^ hiw(t.b[r]) : ~0u));
    t.Tc[k] = cT;
    t.Tr[k] = ieee::recip(cT);
    t.Ty[k] = nz(y) ? y : szero(hiw(y) & (hasL ? s1 ^ hiw(t.y[l]) : ~0u) & (hasR ? s2 ^ hiw(t.y[r]) : ~0u));
    t.Tb[k] = hasL ? add_z(b, zb) : 0.0;
    t.Td[k] = hasR ? add_z(d, zd) : 0.0;
    t.Ta[k] = hasL ? szero(s1 ^ hiw(t.a[l])) : 0.0;
    t.Te[k] = hasR ? szero(s2 ^ hiw(t.e[r])) : 0.0;
    return true;
}

// Phase B, both multipliers active (f1 = b/cT(l), f2 = d/cT(r)); kA, kE: the
// coefficients a and e of the row and of T are zeros (only their signs
// matter).
template <bool kA, bool kE, int CAP>
__device__ __forceinline__ bool row_b_both(TileRows<CAP>& t, int k, int dl, double& f1, double& f2)
{
    const int l = k - dl, r = k + dl;
    const double bi = t.b[k], di = t.d[k], cL = t.Tc[l], cR = t.Tc[r];
    const double aL = t.Ta[l], bL = t.Tb[l], dL = t.Td[l], eL = t.Te[l];
    const double aR = t.Ta[r], bR = t.Tb[r], dR = t.Td[r], eR = t.Te[r];
    unsigned w = ieee::off(bi) | ieee::off(di) | ieee::off(cL) | ieee::off(cR) | ieee::off(bL) | ieee::off(dL) |
                 ieee::off(bR) | ieee::off(dR);
    if (!kA) w |= ieee::off(aL) | ieee::off(aR);
    if (!kE) w |= ieee::off(eL) | ieee::off(eR);
    if (!ieee::fits(w)) return false;
    if (kA && !zeros(t.a[k], aL, aR)) return false;
    if (kE && !zeros(t.e[k], eL, eR)) return false;
    f1 = ieee::div(bi, cL, t.Tr[l]); f2 = ieee::div(di, cR, t.Tr[r]);
    const ieee::Factor g1 = ieee::factor(f1), g2 = ieee::factor(f2);
    const double ny = add(sub(mul(f1, t.Ty[l]), t.y[k]), mul(f2, t.Ty[r]));
    const double nc = add(sub(ieee::mul(g1, dL), t.c[k]), ieee::mul(g2, bR));
    const double b1 = ieee::mul(g1, bL), d2 = ieee::mul(g2, dR);        // nonzero
    const double nb = kA ? b1 : add(sub(b1, t.a[k]), ieee::mul(g2, aR));
    const double nd = kE ? d2 : add(sub(ieee::mul(g1, eL), t.e[k]), d2);
    t.y[k] = ny; t.c[k] = nc; t.b[k] = nb; t.d[k] = nd;
    t.a[k] = kA ? szero(hiw(f1) ^ hiw(aL)) : ieee::mul(g1, aL);
    t.e[k] = kE ? szero(hiw(f2) ^ hiw(eR)) : ieee::mul(g2, eR);
    return true;
}

// Phase B once the couplings are tiny: c and y change sign, the rest on the
// FP64 pipe (a missing side's products are +0).
template <int CAP>
__device__ __forceinline__ bool row_b_tiny(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1,
                                           double& f2)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double ci = t.c[k], yi = t.y[k];
    double g1 = 0.0, g2 = 0.0;
    if (hasL && !(tiny_quotient(t.b[k], t.Tc[l], t.Tr[l], g1) && absorbed(g1, t.Td[l], ci) &&
                  absorbed(g1, t.Ty[l], yi))) return false;
    if (hasR && !(tiny_quotient(t.d[k], t.Tc[r], t.Tr[r], g2) && absorbed(g2, t.Tb[r], ci) &&
                  absorbed(g2, t.Ty[r], yi))) return false;
    t.b[k] = add(sub(hasL ? mul(g1, t.Tb[l]) : 0.0, t.a[k]), hasR ? mul(g2, t.Ta[r]) : 0.0);
    t.d[k] = add(sub(hasL ? mul(g1, t.Te[l]) : 0.0, t.e[k]), hasR ? mul(g2, t.Td[r]) : 0.0);
    t.a[k] = hasL ? mul(g1, t.Ta[l]) : 0.0;
    t.e[k] = hasR ? mul(g2, t.Te[r]) : 0.0;
    t.c[k] = neg(ci); t.y[k] = neg(yi);
    if (hasL) f1 = g1;
    if (hasR) f2 = g2;
    return true;
}

// Zero multiplier num/cT(q) of phase B; false if it is not a zero or a factor
// is not finite.
template <int CAP>
__device__ __forceinline__ bool zero_quotient(TileRows<CAP>& t, int q, double num, double& f, Signs& g)
{
    const double qc = t.Tc[q];
    if (nz(num) || !nz(qc)) return false;
    const double qa = t.Ta[q], qb = t.Tb[q], qd = t.Td[q], qe = t.Te[q], qy = t.Ty[q];
    if (!finite6(qa, qb, qc, qd, qe, qy)) return false;
    const unsigned s = hiw(num) ^ hiw(qc);
    f = szero(s);
    g = {s ^ hiw(qa), s ^ hiw(qb), s ^ hiw(qc), s ^ hiw(qd), s ^ hiw(qe), s ^ hiw(qy)};
    return true;
}

// Phase B, neither multiplier active: the row changes sign.
template <int CAP>
__device__ __forceinline__ bool row_b_none(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1, double& f2)
{
    Signs g1{0u, 0u, 0u, 0u, 0u, 0u}, g2{0u, 0u, 0u, 0u, 0u, 0u};
    const double ai = t.a[k], ci = t.c[k], ei = t.e[k], yi = t.y[k];
    if (!finite6(ai, ci, ei, yi, ci, yi)) return false;
    if (hasL && !zero_quotient(t, k - dl, t.b[k], f1, g1)) return false;
    if (hasR && !zero_quotient(t, k + dl, t.d[k], f2, g2)) return false;
    t.b[k] = add_z(sub_z(g1.b, ai), g2.a);
    t.c[k] = add_z(sub_z(g1.d, ci), g2.b);
    t.d[k] = add_z(sub_z(g1.e, ei), g2.d);
    t.y[k] = add_z(sub_z(g1.y, yi), g2.y);
    t.a[k] = szero(g1.a);
    t.e[k] = szero(g2.e);
    return true;
}

// The same for a tridiagonal row in a tile without infinities and nans: a and e
// of the row and of T are zeros, and a zero pivot leaves its multiplier (f1, f2
// on entry) in place, a zero too but in the last stride.  Batches of small
// integers, whose rows decouple in a few strides while a tenth of the pivots are
// exactly zero, took the general form in every warp (figures at row_b_wide).
template <int CAP>
__device__ __forceinline__ bool row_b_self(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1, double& f2)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double cL = hasL ? t.Tc[l] : 1.0, cR = hasR ? t.Tc[r] : 1.0;
    if (!nz(cL) && nz(f1) || !nz(cR) && nz(f2)) return false;
    const double g1 = nz(cL) ? szero(hiw(t.b[k]) ^ hiw(cL)) : f1, g2 = nz(cR) ? szero(hiw(t.d[k]) ^ hiw(cR)) : f2;
    const unsigned s1 = hiw(g1), s2 = hiw(g2);
    const double ci = t.c[k], yi = t.y[k];
    // (a missing side's products are +0)
    const unsigned zb = (hasL ? s1 ^ hiw(t.Tb[l]) : 0u) & ~hiw(t.a[k]) & (hasR ? s2 ^ hiw(t.Ta[r]) : 0u);
    const unsigned zd = (hasL ? s1 ^ hiw(t.Te[l]) : 0u) & ~hiw(t.e[k]) & (hasR ? s2 ^ hiw(t.Td[r]) : 0u);
    t.c[k] = add_z(sub_z(hasL ? s1 ^ hiw(t.Td[l]) : 0u, ci), hasR ? s2 ^ hiw(t.Tb[r]) : 0u);
    t.y[k] = add_z(sub_z(hasL ? s1 ^ hiw(t.Ty[l]) : 0u, yi), hasR ? s2 ^ hiw(t.Ty[r]) : 0u);
    t.b[k] = szero(zb);
    t.d[k] = szero(zd);
    t.a[k] = szero(hasL ? s1 ^ hiw(t.Ta[l]) : 0u);
    t.e[k] = szero(hasR ? s2 ^ hiw(t.Te[r]) : 0u);
    f1 = g1; f2 = g2;
    return true;
}

// Rows near the ends of a (sub)system, where sides are missing and the
// neighbouring rows hold structural zeros: any operand may be a zero, the
// others are inside the window; integer quotients and products with the zeros
// selected, sums on the FP64 pipe.
// The lanes that test together (any set of a warp's lanes) take this case or
// the general form together: the general form alone is cheaper than this case
// for some lanes and then that for the others (rows scaled by up to 2^+-400,
// us, 8 systems of 512 rows 112 -> 81, 4000 of 128 401 -> 263; dominant rows
// 179 / 179).
__device__ __forceinline__ bool all_fit(uint32_t offs) { return __all_sync(__activemask(), ieee::fits(offs)); }
struct Multiplier {
    ieee::Factor f;
    double x;
    bool active;                        // nonzero: products by ieee::mul
};
__device__ __forceinline__ unsigned off_or_zero(double x) { return nz(x) ? ieee::off(x) : 0u; }
__device__ __forceinline__ Multiplier multiplier(double num, double piv, uint32_t G, bool active, bool zero)
{
    Multiplier m;
    m.x = ieee::div(num, piv, G);
    m.active = active;
    if (!active) m.x = zero ? szero(hiw(num) ^ hiw(piv)) : 0.0;
    m.f = ieee::factor(m.x);
    return m;
}
__device__ __forceinline__ double times(const Multiplier& m, double y)
{
    const double p = ieee::mul(m.f, y);
    return m.active && nz(y) ? p : szero(hiw(m.x) ^ hiw(y));
}

template <int CAP>
__device__ __forceinline__ bool row_a_zeros(TileRows<CAP>& t, int k, int dl, bool hasL, bool has2L, bool hasR,
                                            bool has2R, double& cT)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double am = neg(t.a[k]), em = neg(t.e[k]);
    const double aL = t.a[l], bL = t.b[l], cL = t.c[l], dL = t.d[l], eL = t.e[l];
    const double aR = t.a[r], bR = t.b[r], cR = t.c[r], dR = t.d[r], eR = t.e[r];
    if (!all_fit(off_or_zero(am) | off_or_zero(em) | off_or_zero(aL) | off_or_zero(bL) | off_or_zero(cL) |
                 off_or_zero(dL) | off_or_zero(eL) | off_or_zero(aR) | off_or_zero(bR) | off_or_zero(cR) |
                 off_or_zero(dR) | off_or_zero(eR))) return false;
    const bool piv1 = has2L && nz(bL), piv2 = has2R && nz(dR);
    const Multiplier m1 = multiplier(am, bL, ieee::recip(bL), piv1 && nz(am), piv1);
    const Multiplier m2 = multiplier(em, dR, ieee::recip(dR), piv2 && nz(em), piv2);
    const double m0 = szero(~0u);                 // (a missing side adds -0, which changes nothing)
    cT = add(add(hasL ? times(m1, dL) : m0, t.c[k]), hasR ? times(m2, bR) : m0);
    t.Tc[k] = cT;
    t.Tr[k] = ieee::recip(cT);
    t.Tb[k] = hasL ? add(add(times(m1, cL), t.b[k]), hasR ? times(m2, aR) : m0) : 0.0;
    t.Td[k] = hasR ? add(add(hasL ? times(m1, eL) : m0, t.d[k]), times(m2, cR)) : 0.0;
    t.Ty[k] = add(add(hasL ? mul(m1.x, t.y[l]) : m0, t.y[k]), hasR ? mul(m2.x, t.y[r]) : m0);
    t.Ta[k] = hasL ? times(m1, aL) : 0.0;
    t.Te[k] = hasR ? times(m2, eR) : 0.0;
    return true;
}

template <int CAP>
__device__ __forceinline__ bool row_b_zeros(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1, double& f2)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double bi = t.b[k], di = t.d[k], cL = hasL ? t.Tc[l] : 1.0, cR = hasR ? t.Tc[r] : 1.0;
    const double aL = hasL ? t.Ta[l] : 0.0, bL = hasL ? t.Tb[l] : 0.0, dL = hasL ? t.Td[l] : 0.0, eL = hasL ? t.Te[l] : 0.0;
    const double aR = hasR ? t.Ta[r] : 0.0, bR = hasR ? t.Tb[r] : 0.0, dR = hasR ? t.Td[r] : 0.0, eR = hasR ? t.Te[r] : 0.0;
    if (!all_fit(off_or_zero(bi) | off_or_zero(di) | ieee::off(cL) | ieee::off(cR) | off_or_zero(aL) | off_or_zero(bL) |
                 off_or_zero(dL) | off_or_zero(eL) | off_or_zero(aR) | off_or_zero(bR) | off_or_zero(dR) |
                 off_or_zero(eR))) return false;
    const Multiplier m1 = multiplier(bi, cL, t.Tr[l], hasL && nz(bi), hasL);
    const Multiplier m2 = multiplier(di, cR, t.Tr[r], hasR && nz(di), hasR);
    // (a missing side's products are +0: its factors are)
    const double ny = add(sub(hasL ? mul(m1.x, t.Ty[l]) : 0.0, t.y[k]), hasR ? mul(m2.x, t.Ty[r]) : 0.0);
    const double nb = add(sub(times(m1, bL), t.a[k]), times(m2, aR));
    const double nc = add(sub(times(m1, dL), t.c[k]), times(m2, bR));
    const double nd = add(sub(times(m1, eL), t.e[k]), times(m2, dR));
    t.y[k] = ny; t.b[k] = nb; t.c[k] = nc; t.d[k] = nd;
    t.a[k] = times(m1, aL);
    t.e[k] = times(m2, eR);
    f1 = m1.x; f2 = m2.x;
    return true;
}

// The zeros case of a tridiagonal row in a tile without infinities and nans:
// a and e of the row and of T are zeros, of which only the signs are read.
// Rows near an end used to take the general form here, in short systems most
// rows of the late strides (with row_a_tri and a kernel of their own, us: 35733
// systems of 90 rows 794 -> 580, 4000 of 128 143 -> 102, 777 of 3001 634 -> 585,
// 256 of 16384 1093 -> 1064).
template <int CAP>
__device__ __forceinline__ bool row_b_tri(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1, double& f2)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double bi = t.b[k], di = t.d[k], cL = hasL ? t.Tc[l] : 1.0, cR = hasR ? t.Tc[r] : 1.0;
    const double bL = hasL ? t.Tb[l] : 0.0, dL = hasL ? t.Td[l] : 0.0;
    const double bR = hasR ? t.Tb[r] : 0.0, dR = hasR ? t.Td[r] : 0.0;
    if (!all_fit(off_or_zero(bi) | off_or_zero(di) | ieee::off(cL) | ieee::off(cR) | off_or_zero(bL) |
                 off_or_zero(dL) | off_or_zero(bR) | off_or_zero(dR))) return false;
    const Multiplier m1 = multiplier(bi, cL, t.Tr[l], hasL && nz(bi), hasL);
    const Multiplier m2 = multiplier(di, cR, t.Tr[r], hasR && nz(di), hasR);
    const unsigned s1 = hiw(m1.x), s2 = hiw(m2.x);
    const double ny = add(sub(hasL ? mul(m1.x, t.Ty[l]) : 0.0, t.y[k]), hasR ? mul(m2.x, t.Ty[r]) : 0.0);
    const double nc = add(sub(times(m1, dL), t.c[k]), times(m2, bR));
    const double b1 = times(m1, bL), d2 = times(m2, dR);
    // b1 - a + m2 * Ta(r), m1 * Te(l) - e + d2, the zeros by their signs
    const unsigned zb = hasR ? s2 ^ hiw(t.Ta[r]) : 0u, zd = (hasL ? s1 ^ hiw(t.Te[l]) : 0u) & ~hiw(t.e[k]);
    const double nb = add_z(nz(b1) ? b1 : szero(hiw(b1) & ~hiw(t.a[k])), zb);
    const double nd = add_z(d2, zd);
    const double na = szero(hasL ? s1 ^ hiw(t.Ta[l]) : 0u), ne = szero(hasR ? s2 ^ hiw(t.Te[r]) : 0u);
    t.y[k] = ny; t.c[k] = nc; t.b[k] = nb; t.d[k] = nd; t.a[k] = na; t.e[k] = ne;
    f1 = m1.x; f2 = m2.x;
    return true;
}

// The same for operands outside the integer forms' window, with the products
// on the FP64 pipe (10 FP64 operations instead of the general form's 18, and no
// second try), and for zero pivots: f1, f2 enter as the multipliers those leave
// in place.  The lanes of a warp take row_b_tri or this form together.  us, the
// general form / this one lane by lane / together: rows scaled by up to
// 2^+-400, 4000 systems of 128 rows 215 / 152 / 105, 777 of 3001 1362 / 983 /
// 852; every row scaled by 1e40 145 / 104 / 104 and 818 / 617 / 619.  Small
// integers with exact zero pivots (also by row_b_self, row_a_tri and zero_left),
// the general form against now: 253 -> 145 and 1612 -> 909.
template <int CAP>
__device__ __forceinline__ bool row_b_wide(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double& f1, double& f2)
{
    const int l = hasL ? k - dl : k, r = hasR ? k + dl : k;
    const double cL = hasL ? t.Tc[l] : 1.0, cR = hasR ? t.Tc[r] : 1.0;
    double g1 = 0.0, g2 = 0.0;
    if (hasL) g1 = nz(cL) ? quot(t.b[k], cL, t.Tr[l]) : f1;
    if (hasR) g2 = nz(cR) ? quot(t.d[k], cR, t.Tr[r]) : f2;
    if (max(expw(g1), expw(g2)) >= 0x7FF00000u) return false;
    const unsigned s1 = hiw(g1), s2 = hiw(g2);
    const double ny = add(sub(hasL ? mul(g1, t.Ty[l]) : 0.0, t.y[k]), hasR ? mul(g2, t.Ty[r]) : 0.0);
    const double nc = add(sub(hasL ? mul(g1, t.Td[l]) : 0.0, t.c[k]), hasR ? mul(g2, t.Tb[r]) : 0.0);
    const double b1 = hasL ? mul(g1, t.Tb[l]) : 0.0, d2 = hasR ? mul(g2, t.Td[r]) : 0.0;
    const unsigned zb = hasR ? s2 ^ hiw(t.Ta[r]) : 0u, zd = (hasL ? s1 ^ hiw(t.Te[l]) : 0u) & ~hiw(t.e[k]);
    t.b[k] = add_z(nz(b1) ? b1 : szero(hiw(b1) & ~hiw(t.a[k])), zb);
    t.d[k] = add_z(d2, zd);
    t.a[k] = szero(hasL ? s1 ^ hiw(t.Ta[l]) : 0u);
    t.e[k] = szero(hasR ? s2 ^ hiw(t.Te[r]) : 0u);
    t.c[k] = nc; t.y[k] = ny;
    f1 = g1; f2 = g2;
    return true;
}

// The general forms: every operation on the FP64 pipe but the quotients whose
// operands are inside the integer quotient's guard.
template <int CAP>
__device__ __forceinline__ double row_a_general(TileRows<CAP>& t, int k, int dl, bool hasL, bool has2L, bool hasR, bool has2R)
{
    const int lc = hasL ? k - dl : k, rc = hasR ? k + dl : k;
    // both integer quotients first, whatever the operands: one dependent
    // chain beside the other
    const double am = neg(t.a[k]), em = neg(t.e[k]), bL = t.b[lc], dR = t.d[rc];
    double al1 = ieee::div(am, bL, ieee::recip(bL)), al2 = ieee::div(em, dR, ieee::recip(dR));
    if (!has2L) al1 = 0.0;
    else if (!ieee::div_guard(am, bL)) al1 = nz(bL) ? dvd(am, bL) : 0.0;
    if (!has2R) al2 = 0.0;
    else if (!ieee::div_guard(em, dR)) al2 = nz(dR) ? dvd(em, dR) : 0.0;
    // (a missing side adds -0, which changes nothing: kernel.cu:82-91,108-117)
    const double m0 = szero(~0u);
    const double cT = add(add(hasL ? mul(al1, t.d[lc]) : m0, t.c[k]), hasR ? mul(al2, t.b[rc]) : m0);
    const double kT = add(add(hasL ? mul(al1, t.y[lc]) : m0, t.y[k]), hasR ? mul(al2, t.y[rc]) : m0);
    const double bT = hasL ? add(add(mul(al1, t.c[lc]), t.b[k]), hasR ? mul(al2, t.a[rc]) : m0) : 0.0;
    const double dT = hasR ? add(add(hasL ? mul(al1, t.e[lc]) : m0, t.d[k]), mul(al2, t.c[rc])) : 0.0;
    const double aT = hasL ? mul(al1, t.a[lc]) : 0.0, eT = hasR ? mul(al2, t.e[rc]) : 0.0;
    t.Ta[k] = aT; t.Tb[k] = bT; t.Tc[k] = cT; t.Td[k] = dT; t.Te[k] = eT; t.Ty[k] = kT;
    t.Tr[k] = ieee::recip(cT);
    return cT;
}

// f1, f2 enter as the multipliers a zero pivot leaves in place (kernel.cu:122,129)
template <int CAP>
__device__ __forceinline__ double2 row_b_general(TileRows<CAP>& t, int k, int dl, bool hasL, bool hasR, double f1, double f2)
{
    const int lc = hasL ? k - dl : k, rc = hasR ? k + dl : k;
    const double bi = t.b[k], di = t.d[k], cL = t.Tc[lc], cR = t.Tc[rc];
    const double q1 = ieee::div(bi, cL, t.Tr[lc]), q2 = ieee::div(di, cR, t.Tr[rc]);
    if (hasL && nz(cL)) f1 = ieee::div_guard(bi, cL) ? q1 : dvd(bi, cL);
    if (hasR && nz(cR)) f2 = ieee::div_guard(di, cR) ? q2 : dvd(di, cR);
    const double a1 = hasL ? mul(f1, t.Ta[lc]) : 0.0, b1 = hasL ? mul(f1, t.Tb[lc]) : 0.0;   // kernel.cu:120-125
    const double c1 = hasL ? mul(f1, t.Td[lc]) : 0.0, d1 = hasL ? mul(f1, t.Te[lc]) : 0.0;
    const double k1 = hasL ? mul(f1, t.Ty[lc]) : 0.0;
    const double c2 = hasR ? mul(f2, t.Tb[rc]) : 0.0, b2 = hasR ? mul(f2, t.Ta[rc]) : 0.0;   // kernel.cu:127-132
    const double d2 = hasR ? mul(f2, t.Td[rc]) : 0.0, e2 = hasR ? mul(f2, t.Te[rc]) : 0.0;
    const double k2 = hasR ? mul(f2, t.Ty[rc]) : 0.0;
    t.b[k] = add(sub(b1, t.a[k]), b2);     // kernel.cu:138-140
    t.c[k] = add(sub(c1, t.c[k]), c2);
    t.d[k] = add(sub(d1, t.e[k]), d2);
    t.y[k] = add(sub(k1, t.y[k]), k2);
    t.a[k] = a1; t.e[k] = e2;
    return make_double2(f1, f2);
}

// Phase A's multipliers of row m (T(m) = left*row(m-d) + row(m) +
// right*row(m+d)), formed again
template <int CAP>
__device__ __noinline__ double multiplier_left(TileRows<CAP>& t, int m, int dl, int kfirst)
{
    return m - 2 * dl >= kfirst && nz(t.b[m - dl]) ? quot(neg(t.a[m]), t.b[m - dl]) : 0.0;
}
template <int CAP>
__device__ __noinline__ double multiplier_right(TileRows<CAP>& t, int m, int dl, int klast)
{
    return m + 2 * dl <= klast && nz(t.d[m + dl]) ? quot(neg(t.e[m]), t.d[m + dl]) : 0.0;
}
// The same of a tridiagonal row in a tile without infinities and nans, where a
// and e are zeros
template <int CAP>
__device__ __forceinline__ double zero_left(TileRows<CAP>& t, int m, int dl, int kfirst)
{
    return m - 2 * dl >= kfirst && nz(t.b[m - dl]) ? szero(~(hiw(t.a[m]) ^ hiw(t.b[m - dl]))) : 0.0;
}
template <int CAP>
__device__ __forceinline__ double zero_right(TileRows<CAP>& t, int m, int dl, int klast)
{
    return m + 2 * dl <= klast && nz(t.d[m + dl]) ? szero(~(hiw(t.e[m]) ^ hiw(t.d[m + dl]))) : 0.0;
}

// Row k couples to no other row, and no product of its c and y with another
// such row's can leave the normal range.
template <int CAP>
__device__ __forceinline__ bool decoupled(TileRows<CAP>& t, int k)
{
    return zeros(t.a[k], t.b[k], t.d[k]) && !nz(t.e[k]) && ieee::mid(t.c[k]) && ieee::mid(t.y[k]);
}

// Global loads of the state; kL2Only reads through L2 only (ld.global.cg), for
// persistent kernels that read data other CTAs wrote earlier in the same launch.
template <bool kL2Only>
__device__ __forceinline__ double gload(const double* p) {
    if (kL2Only) return __ldcg(p);
    return *p;
}

// One CTA's work: window w of subsystem r of system j (whole subsystem when
// p.final_step).  Every thread of the CTA must call it with the same (j, r, w).
// kFew: one case for all rows (row_a_zeros, row_b_zeros), then the general
// form; else a case per kind of row (launch_cap chooses).  kTri: a tridiagonal
// batch (null outer bands), whose rows have cases of their own; in a kernel of
// their own, since in the pentadiagonal one they cost it 2-3 %.  kWindow: the
// pass is a window pass (not p.final_step), known when compiled, which leaves
// the finish and its tests out of the kernel that long systems spend most of
// their time in (m=64 n=2^20 34.5 -> 34.3 ms, m=256 n=65536 7.86 -> 7.81).
template <int CAP, bool kL2Only = false, bool kFew = false, bool kTri = false, bool kWindow = false>
__device__ __forceinline__ void pcr_tile(const PcrPassArgs& p, int64_t j, uint32_t r, uint32_t w, TileRows<CAP>& T)
{
    // row numbers inside a system fit 32 bits (n <= 2^31), and G = 2^lg: a
    // 64-bit division is ~80 instructions, and every thread runs this code for
    // two rows of a tile
    const int lg = p.lg;
    const bool final_step = !kWindow && p.final_step != 0;
    const int64_t sbase = p.offsets ? p.offsets[j] : j * p.src_ss;
    const int64_t dbase = p.offsets ? p.offsets[j] : j * p.dst_ss;
    const uint32_t nsys = (uint32_t)(p.offsets ? (p.offsets[j + 1] - p.offsets[j]) : p.n);
    if (r >= nsys) return;
    const uint32_t nr = ((nsys - 1 - r) >> lg) + 1;          // rows of subsystem r
    const uint32_t wlo = w * (uint32_t)p.L;
    if (wlo >= nr) return;
    const uint32_t whi = min(wlo + (uint32_t)p.L, nr);
    const uint32_t t0 = wlo - min(wlo, (uint32_t)p.H), t1 = min(whi + (uint32_t)p.H, nr);
    const int TR = (int)(t1 - t0);
    const int tid = threadIdx.x, bd = blockDim.x;
    // distance of local rows t, t+1 and local row 0 of the source
    const int64_t sstep = p.src_sub ? 1 : p.G * p.src_rs;
    const int64_t soff = p.src_sub ? sbase + r * (nsys >> lg) + min(r, nsys & ((1u << lg) - 1)) : sbase + r * p.src_rs;
    const int64_t dstep = p.G * p.dst_rs;
    const int64_t doff = dbase + r * p.dst_rs;
    // a null outer band (a tridiagonal batch, first pass only) is +0.0
    const bool has_a = p.src[A_] != nullptr, has_e = p.src[E_] != nullptr;
    const double* __restrict__ ga = has_a ? p.src[A_] + soff : nullptr;
    const double* __restrict__ gb = p.src[B_] + soff;
    const double* __restrict__ gc = p.src[C_] + soff;
    const double* __restrict__ gd = p.src[D_] + soff;
    const double* __restrict__ ge = has_e ? p.src[E_] + soff : nullptr;
    const double* __restrict__ gy = p.src[Y_] + soff;

    // The multipliers of phase B that the reference keeps from one stride to
    // the next (kernel.cu:60) are read in one case only: in the last stride of
    // a whole subsystem, by a row whose pivot cT is exactly zero and that has
    // no other multiplier of that stride (kernel.cu:122,129): fewer than 3*dl
    // rows are left then, and a subsystem with p.rem strides to go has at least
    // 2^p.rem rows.  So they are kept (in local memory) by the last stride but
    // one, and pass through global memory only if a global pass ends with it.
    double kept1[kMaxRowsPerThread], kept2[kMaxRowsPerThread];
    if (!kWindow && p.bulk) {
        // The whole system is the tile (t0 = 0, TR = n, even): thread 0
        // stages each array with one bulk asynchronous copy straight into its
        // shared-memory row array (16-byte aligned: contiguous layout, even
        // n, aligned arrays -- the host checks), completing on an mbarrier.
        // A wait that gives up (2 s; copies do not take that long) leaves
        // x = NaN for this system, so the failure shows in the result.
        __shared__ __align__(8) uint64_t bulk_bar;
        if (tid == 0) {
            tma::mbar_init(&bulk_bar, 1);
            tma::fence_mbarrier_init();
        }
        __syncthreads();
        if (tid == 0) {
            const uint32_t bytes = (uint32_t)TR * (uint32_t)sizeof(double);
            const uint64_t pol = tma::policy_evict_first();
            tma::mbar_expect_tx(&bulk_bar, (4u + (has_a ? 1u : 0u) + (has_e ? 1u : 0u)) * bytes);
            if (has_a) tma::bulk_g2s(T.a, ga, bytes, &bulk_bar, pol);
            tma::bulk_g2s(T.b, gb, bytes, &bulk_bar, pol);
            tma::bulk_g2s(T.c, gc, bytes, &bulk_bar, pol);
            tma::bulk_g2s(T.d, gd, bytes, &bulk_bar, pol);
            if (has_e) tma::bulk_g2s(T.e, ge, bytes, &bulk_bar, pol);
            tma::bulk_g2s(T.y, gy, bytes, &bulk_bar, pol);
        }
        const bool got = tma::mbar_wait_bounded(&bulk_bar, 0, 2000000000ull);
        if (__syncthreads_or(!got)) {
            if (tid == 0) tma::mbar_wait_bounded(&bulk_bar, 0, 2000000000ull);   // (copies in flight)
            __syncthreads();
            double* __restrict__ gx = p.x + doff;
            for (int k = tid; k < TR; k += bd) gx[k * dstep] = __longlong_as_double(0x7FF8000000000000LL);
            return;
        }
        for (int k = tid; k < TR; k += bd) {
            if (!has_a) T.a[k] = 0.0;
            if (!has_e) T.e[k] = 0.0;
        }
    } else {
#pragma unroll 2
        for (int k = tid; k < TR; k += bd) {
            const int64_t gi = (int64_t)(t0 + k) * sstep;
            const double a = has_a ? gload<kL2Only>(ga + gi) : 0.0;
            const double e = has_e ? gload<kL2Only>(ge + gi) : 0.0;
            const double b = gload<kL2Only>(gb + gi), c = gload<kL2Only>(gc + gi);
            const double d = gload<kL2Only>(gd + gi), y = gload<kL2Only>(gy + gi);
            T.a[k] = a; T.b[k] = b; T.c[k] = c; T.d[k] = d; T.e[k] = e; T.y[k] = y;
        }
    }
    if (p.rem == 1)
        for (int k = tid, q = 0; k < TR; k += bd, q++) {
            const int64_t gi = soff + (int64_t)(t0 + k) * sstep;
            kept1[q] = p.src[AL1_] ? gload<kL2Only>(p.src[AL1_] + gi) : 0.0;
            kept2[q] = p.src[AL1_] ? gload<kL2Only>(p.src[AL2_] + gi) : 0.0;
        }
    // local rows of the subsystem's ends: row k of the tile has a neighbour at
    // distance x iff k - x >= kfirst / k + x <= klast (32-bit: ends further
    // away than any distance of the tile are moved in to 2^14 rows)
    const int kfirst = -(int)min(t0, 16384u), klast = (int)min(nr - 1 - t0, 16384u);

    // A whole subsystem whose rows are all decoupled (a = b = d = e = 0, c and
    // y away from the ends of the exponent range): every further stride only
    // changes the signs of c and y of every row, which the final step's
    // products and quotients cancel, so the remaining strides are skipped.
    bool apart = final_step;
    if (apart)
        for (int k = tid; k < TR; k += bd) apart = apart && decoupled(T, k);
    // tridiagonal batches: no row of the tile holds an infinity or a nan (kept
    // up by phase B)
    __shared__ int s_odd;
    if (kTri) {
        bool odd = false;
        for (int k = tid; k < TR; k += bd) odd = odd || !finite4(T.b[k], T.c[k], T.d[k], T.y[k]);
        const bool any = __syncthreads_or(odd);
        if (tid == 0) s_odd = any;
    }
    const int strides = __syncthreads_and(apart) ? 0 : p.K;

    // the first strides in which this warp's rows try the cases of phase A and
    // of phase B (kGeneralStrides): not the first ones if rows with and without
    // zeros mix (the warp's first rows are looked at)
    int casesA = 0, casesB = 0;
    if (!kFew && !kTri) {
        const bool z = tid < TR && !(nz(T.a[tid]) && nz(T.b[tid]) && nz(T.d[tid]) && nz(T.e[tid]));
        const unsigned zm = __ballot_sync(~0u, z);
        if (zm != ~0u && __popc(zm) >= 2) casesA = casesB = kGeneralStrides;
    }
    for (int s = 0; s < strides; s++) {
        const int dl = 1 << s;
        // rows this stride must produce: the window widened by the halo the
        // remaining strides of the pass still consume (everything if final).
        int klo = 0, khi = TR;
        if (!final_step) {
            const int rem = 2 * ((1 << p.K) - (2 << s));
            klo = max((int)(wlo - t0) - rem, kfirst); khi = min((int)(whi - t0) + rem, klast + 1);
        }
        // the rows whose T(m) those need, all in the tile
        const int Alo = max(klo - dl, 0), Ahi = min(khi + dl, TR);

        // ---- phase A: T(m) = a1*row(m-d) + row(m) + a2*row(m+d) ----------
        bool zero_pivot = false;
        const bool tame = kTri && s_odd == 0;
        bool odd = false;                         // a row away from the ends without a case
        unsigned rest = 0u;                       // rows no case took: bit q for row tid + q*bd
#pragma unroll 1
        for (int k = tid, q = 0; k < TR; k += bd, q++) {
            if (k < Alo || k >= Ahi) continue;
            const bool hasL = k - dl >= kfirst, hasR = k + dl <= klast;
            const bool has2L = k - 2 * dl >= kfirst, has2R = k + 2 * dl <= klast;
            if (!(hasL || hasR)) continue;
            const bool left = has2L && nz(T.a[k]), right = has2R && nz(T.e[k]);   // nonzero multipliers
            double cT;
            bool done = false;
            if (kFew) {
                done = row_a_zeros(T, k, dl, hasL, has2L, hasR, has2R, cT);
                if (!done) cT = row_a_general(T, k, dl, hasL, has2L, hasR, has2R);
                done = true;
            } else if (!left && !right) {
                if (tame && hasL && hasR) done = row_a_self(T, k, dl, has2L, has2R, cT);
                if (tame && !done) done = row_a_tri(T, k, dl, hasL, has2L, hasR, has2R, cT);
                if (!done) done = row_a_none(T, k, dl, hasL, has2L, hasR, has2R, cT);
            } else if (!kTri && s >= casesA && has2L && has2R) {
                if (left && right) done = row_a_both(T, k, dl, cT);
                else done = row_a_one(T, k, dl, right, cT);
                if (!done) done = row_a_tiny(T, k, dl, hasL, has2L, hasR, has2R, cT);
            }
            // (rows near the subsystem's ends, where neighbouring rows hold
            // structural zeros, have no case)
            if (done) zero_pivot = zero_pivot || !nz(cT);
            else rest |= 1u << q;
        }
        if (!kFew && __any_sync(~0u, rest != 0u)) {
#pragma unroll 1
            for (; rest != 0u; rest &= rest - 1u) {
                const int k = tid + (__ffs(rest) - 1) * bd;
                const bool hasL = k - dl >= kfirst, hasR = k + dl <= klast;
                const bool has2L = k - 2 * dl >= kfirst, has2R = k + 2 * dl <= klast;
                const double cT = row_a_general(T, k, dl, hasL, has2L, hasR, has2R);
                if (!kTri) odd = odd || (k - 3 * dl >= kfirst && k + 3 * dl <= klast);
                zero_pivot = zero_pivot || !nz(cT);
            }
            if (!kTri && __any_sync(~0u, odd) && s >= casesA) casesA = s + 1 + kGeneralStrides;
        }
        double pre1[kMaxRowsPerThread], pre2[kMaxRowsPerThread];
        const bool zeros_left = __syncthreads_or(zero_pivot);   // (read again by tridiagonal tiles)
        if (zeros_left) {
            // some pivot cT of the tile is exactly zero: the multipliers the
            // reference then uses (kernel.cu:96-112), from the state before
            // phase B changes it (where one case serves all rows and in
            // tridiagonal tiles, only of the rows that divide by it: the test in
            // the per-case kernel costs dense batches 0.5-0.8 %)
            for (int k = tid, q = 0; k < TR; k += bd, q++) {
                const bool hasL = k - dl >= kfirst, hasR = k + dl <= klast;
                const bool has2L = k - 2 * dl >= kfirst, has2R = k + 2 * dl <= klast;
                if (k < klo || k >= khi) continue;
                if (kFew || kTri) {
                    const int ml = hasR ? k + dl : k - dl, mr = has2R ? k + dl : k - dl;
                    if (hasL && !nz(T.Tc[k - dl]))
                        pre1[q] = !hasR && !has2L ? kept1[q]
                                  : tame ? zero_left(T, ml, dl, kfirst) : multiplier_left(T, ml, dl, kfirst);
                    if (hasR && !nz(T.Tc[k + dl]))
                        pre2[q] = !has2R && !hasL ? kept2[q]
                                  : tame ? zero_right(T, mr, dl, klast) : multiplier_right(T, mr, dl, klast);
                } else {
                    pre1[q] = hasR ? multiplier_left(T, k + dl, dl, kfirst)
                                   : has2L ? multiplier_left(T, k - dl, dl, kfirst) : kept1[q];
                    pre2[q] = has2R ? multiplier_right(T, k + dl, dl, klast)
                                    : hasL ? multiplier_right(T, k - dl, dl, klast) : kept2[q];
                }
            }
            __syncthreads();
        }

        // ---- phase B: new row = b/cT(i-d)*T(i-d) - row(i) + d/cT(i+d)*T(i+d)
        // (in place: phase B reads no other row's state)
        apart = final_step;
        const bool keep = s == p.rem - 2;
        odd = false;
#pragma unroll 1
        for (int k = tid, q = 0; k < TR; k += bd, q++) {
            if (k < klo || k >= khi) continue;
            const bool hasL = k - dl >= kfirst, hasR = k + dl <= klast;
            const bool left = hasL && nz(T.b[k]), right = hasR && nz(T.d[k]);
            double f1 = 0.0, f2 = 0.0;
            bool done = false;
            if (kFew) {
                done = row_b_zeros(T, k, dl, hasL, hasR, f1, f2);
                if (!done) {
                    const double2 f = row_b_general(T, k, dl, hasL, hasR, pre1[q], pre2[q]);
                    f1 = f.x; f2 = f.y;
                    done = true;
                }
            } else if (!left && !right) {
                if (tame) {
                    if (zeros_left) { f1 = pre1[q]; f2 = pre2[q]; }
                    done = row_b_self(T, k, dl, hasL, hasR, f1, f2);
                } else {
                    done = row_b_none(T, k, dl, hasL, hasR, f1, f2);
                }
            } else if (kTri) {
                // the dense form of inner rows in a window, one form for all in
                // a whole subsystem, where most rows are near an end
                const bool inner = k - 3 * dl >= kfirst && k + 3 * dl <= klast;
                if (inner && !final_step && left && right && !nz(T.a[k]) && !nz(T.e[k]))
                    done = row_b_both<true, true>(T, k, dl, f1, f2);
                else if (tame) done = row_b_tri(T, k, dl, hasL, hasR, f1, f2);
            } else if (s >= casesB && k - 3 * dl >= kfirst && k + 3 * dl <= klast) {
                if (left && right) {
                    const bool za = !nz(T.a[k]), ze = !nz(T.e[k]);
                    if (za && ze) done = row_b_both<true, true>(T, k, dl, f1, f2);
                    else if (za) done = row_b_both<true, false>(T, k, dl, f1, f2);
                    else done = row_b_both<false, false>(T, k, dl, f1, f2);
                }
                if (!done) done = row_b_tiny(T, k, dl, hasL, hasR, f1, f2);
            }
            if (done) {
                apart = apart && !left && !right && decoupled(T, k);
                if (kTri && !finite4(T.b[k], T.c[k], T.d[k], T.y[k])) s_odd = 1;
                if (keep) { kept1[q] = f1; kept2[q] = f2; }
            } else {
                double2 f;
                if (kTri) f = make_double2(pre1[q], pre2[q]);
                if (!(tame && row_b_wide(T, k, dl, hasL, hasR, f.x, f.y)))
                    f = row_b_general(T, k, dl, hasL, hasR, pre1[q], pre2[q]);
                if (!kTri) odd = odd || (k - 4 * dl >= kfirst && k + 4 * dl <= klast);
                apart = apart && !left && !right && decoupled(T, k);
                if (kTri && !finite4(T.b[k], T.c[k], T.d[k], T.y[k])) s_odd = 1;
                if (keep) { kept1[q] = f.x; kept2[q] = f.y; }
            }
        }
        if (!kFew && !kTri && __any_sync(~0u, odd) && s >= casesB) casesB = s + 1 + kGeneralStrides;
        if (__syncthreads_and(apart)) break;
    }

    if (final_step) {
        // kernel.cu:145-153: pairs (i, i+delta) by Cramer's rule, singles x = y/c
        const int df = 1 << p.K;
        double* __restrict__ gx = p.x + doff;
        for (int k = tid; k < TR; k += bd) {       // whole subsystem: t0 == 0, TR == nr
            if (k < TR - df) {
                const int kk = k + df;
                const double deno = sub(mul(T.c[k], T.c[kk]), mul(T.b[kk], T.d[k]));
                gx[k * dstep] = quot(sub(mul(T.c[kk], T.y[k]), mul(T.d[k], T.y[kk])), deno);
                gx[kk * dstep] = quot(sub(mul(T.c[k], T.y[kk]), mul(T.b[kk], T.y[k])), deno);
            }
            if (k >= TR - df && k < df) gx[k * dstep] = quot(T.y[k], T.c[k]);
        }
    } else {
        // subsystem-major output: row t of subsystem r is row t >> K of
        // subsystem r + (t mod 2^K) G at the next level's stride G 2^K
        const int lg2 = lg + p.K;
        const uint32_t q2 = nsys >> lg2, rem2 = nsys & ((1u << lg2) - 1), kmask = (1u << p.K) - 1;
        for (int k = tid, q = 0; k < TR; k += bd, q++) {
            const uint32_t t = t0 + k;
            if (t >= wlo && t < whi) {
                int64_t gi;
                if (p.dst_sub) {
                    const uint32_t r2 = r + ((t & kmask) << lg);
                    gi = dbase + (r2 * q2 + min(r2, rem2) + (t >> p.K));    // (r2 * q2 <= nsys)
                } else {
                    gi = doff + t * dstep;
                }
                p.dst[A_][gi] = T.a[k]; p.dst[B_][gi] = T.b[k]; p.dst[C_][gi] = T.c[k];
                p.dst[D_][gi] = T.d[k]; p.dst[E_][gi] = T.e[k]; p.dst[Y_][gi] = T.y[k];
                if (p.rem == p.K + 1) { p.dst[AL1_][gi] = kept1[q]; p.dst[AL2_][gi] = kept2[q]; }
            }
        }
    }
}

}  // namespace pcrp

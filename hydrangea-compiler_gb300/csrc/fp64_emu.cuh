// fp64_emu.cuh -- binary64 additions and whole stencil sums on the integer pipe.
//
// GB300 does 5.29e11 FP64 operations per second, 1.68 per clock and SM, so an FP64
// stencil is bound by that pipe long before HBM.  The integer pipe is idle there; moving
// some of the stencil's additions onto it raises throughput while the results
// stay bit-identical to IEEE-754 round-to-nearest-even.
//
// dadd_pos() takes the textbook route for two non-negative normal operands
// whose exponents differ by at most 10 (the usual case of a stencil's sums):
//   1. order the operands by magnitude (for non-negative doubles the bit
//      patterns order like the values);
//   2. widen both significands (hidden bit set) by 10 guard bits; the smaller
//      one is aligned by shifting it left by 10 - gap, which is exact;
//   3. add, and renormalise by one place if the sum carried out, keeping the
//      bit shifted out as a sticky bit;
//   4. round to nearest, ties to even, on the 10 discarded bits, and
//      renormalise once more if rounding carried into bit 53.
// Any other case -- an operand that is zero, subnormal, negative, infinite or
// NaN, a larger exponent gap, or a result that overflows the exponent range --
// takes __dadd_rn on the FP64 unit, so the function is exact for every input.
#pragma once

#include <stdint.h>

namespace hyd {

// The fallback lives behind a call so that the compiler cannot if-convert it
// into an unconditional FP64 add on every lane: warps whose operands are all
// on the fast path branch over it and issue nothing on the FP64 pipe.
static __device__ __noinline__ double dadd_fallback(double x, double y) { return __dadd_rn(x, y); }

__device__ __forceinline__ double dadd_pos(double x, double y) {
    const unsigned long long X = (unsigned long long)__double_as_longlong(x);
    const unsigned long long Y = (unsigned long long)__double_as_longlong(y);
    const unsigned long long hi = X > Y ? X : Y, lo = X > Y ? Y : X;
    const unsigned eh = (unsigned)(hi >> 52), el = (unsigned)(lo >> 52);
    const unsigned d = eh - el;
    // fast path: both exponent fields in [1, 2046] with the sign bit clear (a
    // set sign bit makes the field >= 2048; hi >= lo, so testing el >= 1 and
    // eh <= 2046 covers both operands) and an exponent gap of at most 10, so
    // that aligning the smaller significand below 10 guard bits drops no bit
    bool ok = el >= 1u && eh <= 2046u && d <= 10u;
    constexpr unsigned long long kM52 = (1ULL << 52) - 1ULL, kH = 1ULL << 52;
    const unsigned long long mh = ((hi & kM52) | kH) << 10;                 // in [2^62, 2^63)
    const unsigned long long al = ((lo & kM52) | kH) << ((10u - d) & 15u);  // exact
    unsigned long long s = mh + al;                                          // < 2^64
    unsigned e = eh;
    if (s >> 63) {  // carry out: one place right, keeping the lost bit as sticky
        s = (s >> 1) | (s & 1ULL);
        e += 1u;
    }
    unsigned long long mant = s >> 10;  // in [2^52, 2^53)
    const unsigned rem = (unsigned)s & 0x3FFu;
    mant += (unsigned long long)((rem > 0x200u) | ((rem == 0x200u) & ((unsigned)mant & 1u)));
    if (mant >> 53) {  // rounded up to 2^53: exactly 2^52 one exponent higher
        mant >>= 1;
        e += 1u;
    }
    ok &= e <= 2046u;
    if (!ok) return dadd_fallback(x, y);
    return __longlong_as_double((long long)(((unsigned long long)e << 52) + (mant - kH)));
}

// ddiv_small_rn<D>(x) = x / D rounded to nearest even, for D = 3 or 5, in one
// multiply and two FMAs instead of a full IEEE division (the published
// correction scheme for division by a constant: Markstein, IBM J. R&D 1990;
// Brisebarre, Muller, Raina, IEEE Trans. Computers 53(8), 2004):
//   q0 = RN(x * z)            z = RN(1/D)
//   r  = x - D * q0           exact (one FMA): |r| <= D/2 ulp(q0) plus a hair,
//                             a multiple of ulp(q0) well inside 53 bits
//   q  = RN(q0 + r * z)       one FMA
// Why q is RN(x / D) for every finite x: q0 + r/D equals x/D exactly, and
// replacing 1/D by z moves the FMA's exact argument by |r| * |z - 1/D|, under
// 2^-54 ulp(q0).  x/D is either exact (then r = 0) or, since D is odd, lies k/D
// of an ulp past a representable value (0 < k < D), at least 1/(2D) ulp away
// from any rounding midpoint -- with subnormal results too, whose ulp is fixed.
// A tiny shift cannot cross such a midpoint, so the single rounding of the FMA
// gives the correctly rounded quotient.  A zero remainder (x/D exact, x = +-0
// keeping its sign) and a non-finite q0 (x infinite or NaN) return q0 itself.
template <int D>
__device__ __forceinline__ double ddiv_small_rn(double x) {
    static_assert(D == 3 || D == 5, "the correction is proved here for odd D = 3, 5");
    constexpr double z = 1.0 / D;  // RN(1/D)
    const double q0 = __dmul_rn(x, z);
    const double r = __fma_rn(-(double)D, q0, x);
    const unsigned long long qb = (unsigned long long)__double_as_longlong(q0);
    const unsigned long long rb = (unsigned long long)__double_as_longlong(r);
    if (((qb >> 52) & 0x7FFULL) == 0x7FFULL || (rb << 1) == 0ULL) return q0;
    return __fma_rn(r, z, q0);
}

// ---- whole stencil sums on the integer pipe -----------------------------------
// (x0 + x1) + x2 + ..., every addition rounded to nearest even as the FP64 unit
// does it, and what follows the sum in the stencil bodies: nothing, / 4, / 3,
// / 5, or - 4e.  Where dadd_pos unpacks, aligns, rounds and packs each addition
// on its own (about 80 instructions), all operands here are put once on one
// fixed-point grid and only the sums are rounded:
//   1. E = the largest exponent field; an operand with field e becomes its
//      53-bit significand times 2^(e - E + S), for E - e < S: an exact integer
//      on the grid 2^(E - 1023 - 52 - S).  S is such that the sum of all stays
//      below 2^64;
//   2. each partial sum T (>= 2^53, so that p >= 1 bits hang below its 53
//      leading ones) is rounded in place: add half of 2^p, clear the p low
//      bits, and on a tie the bit above them too;
//   3. the last one is shifted back and packed.  Rounding up to the next power
//      of two needs no case: the significand 2^53 carries into the exponent.
// The alignment shifts and the additions are multiply-adds by powers of two
// (IMAD, a pipe that is idle here), so the ALU pipe does only the fields and
// the rounding.  Operands that are zero, subnormal, negative, infinite, NaN or
// further apart, and exponents near the ends of the range, take the FP64 unit
// (behind a call, as in dadd_pos).  Measured: HEAT at 8192^2 517 us per step with
// two additions through dadd_pos, 391 with dsum4_pos (the FP64 pipe then 97%
// busy with the other three operations); jacobi_1d at 2^25 365 -> 191 us with
// dmean3_pos; HEAT_EXAMPLE 895 -> 415 us with dmean5_pos.
struct GridSum {
    unsigned tl, th;  // the rounded sum
    unsigned E, p;    // the largest field; the sum's lowest significant bit
};

// T += x * pw, x = a 53-bit significand (xh: its high word)
__device__ __forceinline__ void grid_add(unsigned& tl, unsigned& th, unsigned xl, unsigned xh, unsigned pw) {
    asm("{\n\t.reg .u64 t;\n\t.reg .u32 h;\n\t"
        "mov.b64 t, {%0, %1};\n\t"
        "mad.wide.u32 t, %2, %4, t;\n\t"
        "mov.b64 {%0, h}, t;\n\t"
        "mad.lo.u32 %1, %3, %4, h;\n\t}"
        : "+r"(tl), "+r"(th)
        : "r"(xl), "r"(xh), "r"(pw));
}
// Rounds T to its 53 leading bits (nearest, ties to even); returns their lowest
// bit's position p.
__device__ __forceinline__ unsigned grid_round(unsigned& tl, unsigned& th) {
    const unsigned q = 31u - (unsigned)__clz((int)th);  // 21 .. 31
    const unsigned half = 1u << ((q + 11u) & 31u);      // 2^(p - 1), p = q - 20
    asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, 0;" : "+r"(tl), "+r"(th) : "r"(half));
    const unsigned low = 2u * half - 1u;
    tl &= ~((tl & low) ? low : 4u * half - 1u);
    return q - 20u;
}
__device__ __forceinline__ unsigned field_of(double x) { return (unsigned)__double2hiint(x) >> 20; }  // >= 2048: negative
__device__ __forceinline__ unsigned sig_hi(double x) {
    return ((unsigned)__double2hiint(x) & 0xFFFFFu) | 0x100000u;
}

// The sum of x[0 .. N-1]; false when an operand is outside what the grid
// takes.  `e` only widens the grid (it is on it too).
template <int N, int S>
__device__ __forceinline__ bool grid_sum(const double (&x)[N], double e, GridSum& g) {
    static_assert(N >= 2 && N <= 5 && S >= 2 && ((unsigned long long)N << (53 + S - 3)) <= (1ull << 61), "T < 2^64");
    unsigned f[N], E = field_of(e), m = E;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        f[k] = field_of(x[k]);
        E = max(E, f[k]);
        m = min(m, f[k]);
    }
    // [80, 2043]: all operands normal, no overflow, no result below the normals
    if (E - 80u > 1963u || E - m >= (unsigned)S) return false;
    const unsigned t = (unsigned)S - E;
    g.E = E;
    g.tl = g.th = 0u;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        grid_add(g.tl, g.th, (unsigned)__double2loint(x[k]), sig_hi(x[k]), 1u << ((f[k] + t) & 31u));
        if (k > 0) g.p = grid_round(g.tl, g.th);
    }
    return true;
}
// The double T >> p with field E - S + p, times 2^-kDown (the hidden bit adds
// the field's last 1).
template <int S, int kDown>
__device__ __forceinline__ double grid_pack(const GridSum& g) {
    return __hiloint2double((int)((g.th >> g.p) + ((g.E + g.p - (unsigned)(S + 1 + kDown)) << 20)),
                            (int)__funnelshift_r(g.tl, g.th, g.p));
}
// The same divided by D = 3 or 5, rounded to nearest.  With the sum's
// significand m at the top of a word, X = 2^11 m, y = the high half of
// X * M, M = (2^(64 + k) + 1) / D with k = 1 or 2, is floor(2^k X / D): the
// product exceeds 2^k X / D by less than 1/D, and that quotient's fraction is a
// multiple of 1/D.  y has its leading bit at 63 or 62; cut to 53 bits, what is cut off
// is never half a unit (a power of two times m / D, D odd), so adding half and
// truncating is round to nearest.
template <int S, int D>
__device__ __forceinline__ double grid_pack_div(const GridSum& g) {
    static_assert(D == 3 || D == 5, "odd divisors only");
    constexpr unsigned long long M = D == 3 ? 0xAAAAAAAAAAAAAAABull : 0xCCCCCCCCCCCCCCCDull;
    constexpr unsigned kUp = D == 3 ? 1 : 2;  // y = 2^kUp X / D
    // the sum's leading bit is at 52 + p, or at 53 + p when it was rounded up
    // to a power of two: put it at bit 63
    const unsigned n = (unsigned)__clz((int)g.th);  // 0 .. 10
    const unsigned long long T = (unsigned long long)g.th << 32 | g.tl;
    const unsigned long long y = __umul64hi(T << n, M);
    const unsigned up = (unsigned)(y >> 63);            // leading bit at 63, or at 62
    const unsigned long long r = y + (up ? 0x400ull : 0x200ull);
    const unsigned long long mant = r >> (10u + up);
    // sum = (T << n) 2^(E - 1075 - S - n), so the quotient is mant 2^(10 + up - kUp + E - 1075 - S - n)
    const unsigned field = g.E + 10u + up - (unsigned)S - n - kUp;
    return __longlong_as_double((long long)(mant + ((unsigned long long)(field - 1u) << 52)));
}
// The sum minus 4e, rounded to nearest even: one exact subtraction on the
// grid, normalised and rounded.
template <int S>
__device__ __forceinline__ double grid_pack_minus_4(const GridSum& g, double e) {
    unsigned el = 0u, eh = 0u;
    grid_add(el, eh, (unsigned)__double2loint(e), sig_hi(e), 4u << ((field_of(e) + (unsigned)S - g.E) & 31u));
    unsigned dl = g.tl, dh = g.th;
    asm("sub.cc.u32 %0, %0, %2;\n\tsubc.u32 %1, %1, %3;" : "+r"(dl), "+r"(dh) : "r"(el), "r"(eh));
    const unsigned s = (unsigned)((int)dh >> 31);  // all ones when negative
    dl ^= s;
    dh ^= s;
    asm("sub.cc.u32 %0, %0, %2;\n\tsubc.u32 %1, %1, %2;" : "+r"(dl), "+r"(dh) : "r"(s));
    // the leading bit to bit 63
    unsigned field = g.E + 63u - 52u - (unsigned)S;  // of a magnitude with its leading bit there
    if (dh == 0u) {
        dh = dl;
        dl = 0u;
        field -= 32u;
    }
    if (dh == 0u) return 0.0;
    const unsigned n = (unsigned)__clz((int)dh);
    dh = __funnelshift_l(dl, dh, n);
    dl <<= n;
    field -= n;
    unsigned c;
    asm("add.cc.u32 %0, %0, 0x400;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, 0, 0;" : "+r"(dl), "+r"(dh), "=r"(c));
    dl &= (dl & 0x7FFu) ? ~0x7FFu : ~0xFFFu;
    const unsigned hi = (dh >> 11) + (c << 21) + ((field - 1u) << 20);
    return __hiloint2double((int)(hi | (s & 0x80000000u)), (int)__funnelshift_r(dl, dh, 11));
}

static __device__ __noinline__ double dsum4_fallback(double a, double b, double c, double d) {
    return __dadd_rn(__dadd_rn(__dadd_rn(a, b), c), d);
}
// ((a + b) + c) + d
__device__ __forceinline__ double dsum4_pos(double a, double b, double c, double d) {
    const double x[4] = {a, b, c, d};
    GridSum g;
    if (!grid_sum<4, 9>(x, a, g)) return dsum4_fallback(a, b, c, d);
    return grid_pack<9, 0>(g);
}
// (((a + b) + c) + d) / 4
__device__ __forceinline__ double dmean4_pos(double a, double b, double c, double d) {
    const double x[4] = {a, b, c, d};
    GridSum g;
    if (!grid_sum<4, 9>(x, a, g)) return __dmul_rn(dsum4_fallback(a, b, c, d), 0.25);
    return grid_pack<9, 2>(g);
}
// (((a + b) + c) + d) - 4e
__device__ __forceinline__ double dlap4_pos(double a, double b, double c, double d, double e) {
    const double x[4] = {a, b, c, d};
    GridSum g;
    if (!grid_sum<4, 8>(x, e, g)) return __fma_rn(-4.0, e, dsum4_fallback(a, b, c, d));
    return grid_pack_minus_4<8>(g, e);
}

static __device__ __noinline__ double dmean3_fallback(double a, double b, double c) {
    return ddiv_small_rn<3>(__dadd_rn(__dadd_rn(a, b), c));
}
static __device__ __noinline__ double dmean5_fallback(double a, double b, double c, double d, double e) {
    return ddiv_small_rn<5>(__dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(a, b), c), d), e));
}
// ((a + b) + c) / 3
__device__ __forceinline__ double dmean3_pos(double a, double b, double c) {
    const double x[3] = {a, b, c};
    GridSum g;
    if (!grid_sum<3, 9>(x, a, g)) return dmean3_fallback(a, b, c);
    return grid_pack_div<9, 3>(g);
}
// ((((a + b) + c) + d) + e) / 5
__device__ __forceinline__ double dmean5_pos(double a, double b, double c, double d, double e) {
    const double x[5] = {a, b, c, d, e};
    GridSum g;
    if (!grid_sum<5, 8>(x, a, g)) return dmean5_fallback(a, b, c, d, e);
    return grid_pack_div<8, 5>(g);
}

}  // namespace hyd

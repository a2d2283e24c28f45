// softfp.cuh -- exact IEEE-754 binary64 operations on the integer and FP32 pipes.
//
// GB300 executes FP64 arithmetic at 1/64 of its FP32 rate (2 DFMA per SM per clock), and an IEEE
// double division costs about 9 DFMA slots there, while the integer and FP32 pipes of the fused
// pass are almost idle.  The helpers below compute bit-identical results to the FP64 instructions
// they replace, for the operands the fast paths accept, using integer arithmetic:
//
//   lt(x, y)      x < y  (false when either is NaN; -0 == +0)
//   gt0(x)        x > 0
//   lt_pos(x, c)  x < c for a positive constant c
//   neg_if(x, c)  c ? -x : x  (a sign flip: what multiplying by -1 gives for non-NaN x)
//   scale(x, k)   x * 2^k, exact (half(x) = x * 0.5, twice(x) = x * 2)
//   absval(x)     |x|
//   div(a, b)     the correctly rounded quotient (round to nearest, ties to even)
//   sqrt(x)       the correctly rounded square root
//   mul(a, b)     the correctly rounded product
//   add(a, b)     the correctly rounded sum (add_bits: the same on bit patterns, host or device)
//
// Division (my own construction from the arithmetic, not a library's sequence).  With significands
// ma, mb in [2^52, 2^53) and ma doubled when ma < mb, the result significand is ma 2^52 / mb rounded to
// nearest.  A 32-bit reciprocal of mb (an FP32 seed and one Newton step in 32-bit fixed point, from
// below) gives the quotient in two digits, each followed by its exact remainder, and the last
// remainder decides the rounding: see quot_estimate for the bounds.  32-bit products only, about 60
// instructions with the exponent handling (two Newton steps in 64-bit fixed point and a correction
// step took about 100).  Zero dividends are handled; subnormal, infinite and NaN operands and
// quotients outside the normal range go to the hardware division.
#pragma once

#include <cstdint>

namespace armon {
namespace sfp {

// The bit pattern is taken in inline PTX so that the compiler cannot see the integer tests that
// follow as floating-point class tests (zero, NaN, normal), which it would otherwise fold back into
// FP64 compares on the FP64 pipe.
__device__ __forceinline__ uint64_t bits(double x)
{
    uint64_t u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
    return u;
}
__device__ __forceinline__ double from_bits(uint64_t u) { return __longlong_as_double((long long)u); }

constexpr uint64_t kAbs = 0x7FFFFFFFFFFFFFFFull;
constexpr uint64_t kInf = 0x7FF0000000000000ull;
constexpr uint64_t kMant = 0x000FFFFFFFFFFFFFull;
constexpr uint64_t kHidden = 0x0010000000000000ull;

// Monotone key of a non-NaN double: -x and +x map to -k and +k, and -0, +0 both to 0.
__device__ __forceinline__ int64_t key(uint64_t u)
{
    const int64_t a = (int64_t)(u & kAbs);
    return (int64_t)u < 0 ? -a : a;
}

__device__ __forceinline__ bool lt(double x, double y)
{
    const uint64_t ux = bits(x), uy = bits(y);
    const bool nan = ((ux & kAbs) > kInf) | ((uy & kAbs) > kInf);
    return !nan && key(ux) < key(uy);
}

__device__ __forceinline__ bool gt0(double x)
{
    const int64_t u = (int64_t)bits(x);
    return u > 0 && (uint64_t)u <= kInf;
}

// x < c for a constant c > 0 given by its bit pattern: the signed order of the patterns is the
// IEEE order against a positive value, except for NaNs with the sign bit set.
__device__ __forceinline__ bool lt_pos(double x, uint64_t c)
{
    const uint64_t u = bits(x);
    return (int64_t)u < (int64_t)c && (u & kAbs) <= kInf;
}

// The sign-bit operations are written on the high word in inline PTX: a plain xor / and of the
// bit pattern is recognised as an FP negation / absolute value, which can be materialised on the
// FP64 pipe.
__device__ __forceinline__ double neg_if(double x, bool c)
{
    const uint32_t m = (uint32_t)c << 31;
    uint32_t hi;
    asm("xor.b32 %0, %1, %2;" : "=r"(hi) : "r"((uint32_t)__double2hiint(x)), "r"(m));
    return __hiloint2double((int)hi, __double2loint(x));
}

__device__ __forceinline__ double absval(double x)
{
    uint32_t hi;
    asm("and.b32 %0, %1, 0x7FFFFFFF;" : "=r"(hi) : "r"((uint32_t)__double2hiint(x)));
    return __hiloint2double((int)hi, __double2loint(x));
}

// x * 2^k for |k| < 2046: exact whenever x and the result are normal, so the exponent field moves
// by k; zeros are returned as they are; everything else (subnormal operand or result, overflow,
// infinities, NaN) takes the FP64 multiply by the power of two `p2` (== 2^k).
__device__ __forceinline__ double scale(double x, int k, double p2)
{
    const uint64_t u = bits(x);
    const int e = (int)((u >> 52) & 0x7FFu);
    if ((unsigned)(e - 1) < 2046u && (unsigned)(e + k - 1) < 2046u)
        return from_bits(u + ((uint64_t)(int64_t)k << 52));
    if ((u << 1) == 0) return x;
    return x * p2;
}
__device__ __forceinline__ double half(double x) { return scale(x, -1, 0.5); }
__device__ __forceinline__ double twice(double x) { return scale(x, 1, 2.0); }

// A 32-bit reciprocal of a divisor significand mb in [2^52, 2^53): y <= 2^84 / mb < 2^32, within 2^-30
// of it (relative).  The seed is rcp.approx (one ulp) of mb's top 24 bits, made odd so that it stays
// above 2^23 and its reciprocal below 2^-23; with 1/x for x = mb / 2^53 in units of 2^-31, the
// truncation (2^9), the odd bit (2^9) and the seed's ulp (2^8) leave it within [-0x300, 0x300] of
// the true value, so that less 0x400 it lies in [-0x700, -0x100].  One Newton step y += y (1 - x y)
// in 32 bits, with x rounded up, keeps it below and leaves 2^-40 (the step), 2^-31 (x) and 2^-31 (the
// truncation).
__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b)
{
    return (uint32_t)(((uint64_t)a * b) >> 32);
}
__host__ __device__ __forceinline__ uint32_t recip_step(uint32_t dhi, uint32_t seed_bits)
{
    const uint32_t y0 = ((seed_bits << 8) | 0x80000000u) - 0x400u;
    const uint64_t e = (1ull << 63) - ((uint64_t)dhi * y0 + y0);        // 1 - x y0 in Q63, below 2^43
    return y0 + (mulhi32(y0, (uint32_t)(e >> 11)) >> 20);
}
__device__ __forceinline__ uint32_t recip_y(uint64_t mb)
{
    const uint32_t dhi = (uint32_t)(mb >> 21);
    const float fd = __uint_as_float(0x4B000001u | ((dhi >> 8) & 0x7FFFFFu));
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(fd));
    return recip_step(dhi, __float_as_uint(rf));
}

// The quotient ma 2^52 / mb of significands ma in [mb, 2 mb) from mb's reciprocal y, in two digits of
// 27 and 26 bits: q1 falls short of ma 2^26 / mb by less than 1.25 (half a quarter each for ma's and
// y's truncation, one for the floor), so r1 = ma 2^26 - q1 mb < 1.25 mb; q2 of r1 2^26 / mb by less
// than 1.14 in the same way.  The result q is then floor(ma 2^52 / mb) or one less, and r = ma 2^52 -
// q mb, exact in 64 bits, lies in [0, 1.14 mb).
__host__ __device__ __forceinline__ uint64_t quot_estimate(uint64_t ma, uint64_t mb, uint32_t y, uint64_t& r)
{
    const uint32_t q1 = mulhi32((uint32_t)(ma >> 22), y) >> 4;
    const uint64_t r1 = (ma << 26) - (uint64_t)q1 * mb;
    const uint32_t q2 = mulhi32((uint32_t)(r1 >> 22), y) >> 4;
    r = (r1 << 26) - (uint64_t)q2 * mb;
    return ((uint64_t)q1 << 26) + q2;
}

// The FP64 division of the operands that the integer path leaves, out of line: inlined at every
// division it would be a fifth of a pass's code.
static __device__ __noinline__ double div_hw(double a, double b) { return a / b; }

// a / b; the reciprocal comes from get_y(mb), called only on the integer path.
template <class GetY>
__device__ __forceinline__ double div_core(double a, double b, uint64_t ub, GetY get_y)
{
    const uint64_t ua = bits(a);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7FFu;
    const uint32_t eb = (uint32_t)(ub >> 52) & 0x7FFu;
    const uint64_t sign = (ua ^ ub) & ~kAbs;
    const int e0 = (int)ea - (int)eb;
    const bool b_normal = (eb - 1u) < 2046u;
    if (!(b_normal && (ea - 1u) < 2046u && (unsigned)(e0 + 1021) <= 2043u)) {
        if (b_normal && (ua << 1) == 0) return from_bits(sign);   // +-0 / normal
        return div_hw(a, b);
    }
    uint64_t ma = (ua & kMant) | kHidden;
    const uint64_t mb = (ub & kMant) | kHidden;
    const uint32_t less = ma < mb ? 1u : 0u;
    ma <<= less;
    uint64_t r;
    uint64_t q = quot_estimate(ma, mb, get_y(mb), r);
    // Round to nearest.  A quotient of doubles is never halfway between two doubles, so with
    // r in [0, 1.14 mb) the rounded significand is q + 1 when 2 r > mb and q otherwise: for r >= mb
    // the quotient is q + 1 and what is left of r is below half of mb.
    q += (r << 1) > mb ? 1ull : 0ull;
    return from_bits(sign + ((uint64_t)(uint32_t)(e0 + 1022 - (int)less) << 52) + q);
}

// Out of line in the translation units that define ARMON_SFP_CALLS: the tile pass (sweep_tile.cuh), whose
// warps run every stage on few positions each, waits on instruction fetch when its code is larger
// (4096x4096 circular Sod, 200 cycles: 210 ms inline, 201 ms out of line; a 2048x2048 moving flow 47.9
// and 47.4 ms).  The marches keep it inline.
#ifdef ARMON_SFP_CALLS
#define ARMON_SFP_DIV __noinline__
#else
#define ARMON_SFP_DIV __forceinline__
#endif
static __device__ ARMON_SFP_DIV double div(double a, double b)
{
    return div_core(a, b, bits(b), [](uint64_t mb) { return recip_y(mb); });
}

// A divisor's reciprocal computed once for several quotients (of a normal divisor; div(a, R, b) is
// exact whatever R holds for other divisors).
struct Recip {
    uint64_t ub;
    uint32_t y;
};

__device__ __forceinline__ Recip recip(double b)
{
    Recip R;
    R.ub = bits(b);
    R.y = recip_y((R.ub & kMant) | kHidden);
    return R;
}

__device__ __forceinline__ double div(double a, const Recip& R, double b)
{
    return div_core(a, b, R.ub, [&](uint64_t) { return R.y; });
}

// Multiplication (my own construction).  For normal operands with significands ma, mb in
// [2^52, 2^53), both shifted to bit 63, the product lies in [2^126, 2^128); shifted to bit 127, its
// high word holds the result significand over 11 bits of rest, the lowest of which also stands for
// everything below (a sticky bit); round to nearest, ties to even.  Zero operands give signed zeros;
// subnormal, infinite and NaN operands and results near or outside the ends of the normal range
// take the FP64 multiply.
// the other operands, out of line
static __device__ __noinline__ double mul_rest(double a, double b)
{
    const uint64_t ua = bits(a), ub = bits(b);
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7FFu, eb = (uint32_t)(ub >> 52) & 0x7FFu;
    const uint64_t sign = (ua ^ ub) & ~kAbs;
    if (((ua << 1) == 0 && (eb - 1u) < 2046u) || ((ub << 1) == 0 && (ea - 1u) < 2046u) ||
        ((ua << 1) == 0 && (ub << 1) == 0))
        return from_bits(sign);                                  // +-0 * normal or zero
    return a * b;
}
__device__ __forceinline__ double mul(double a, double b)
{
    const uint64_t ua = bits(a), ub = bits(b);
    const uint32_t ah = (uint32_t)(ua >> 32), bh = (uint32_t)(ub >> 32), al = (uint32_t)ua, bl = (uint32_t)ub;
    const uint32_t ea = (ah >> 20) & 0x7FFu, eb = (bh >> 20) & 0x7FFu;
    const uint32_t sign = (ah ^ bh) & 0x80000000u;
    const uint32_t e = ea + eb - 1024u;      // the result's biased exponent less one, before normalisation
    if ((ea - 1u) < 2046u && (eb - 1u) < 2046u && e < 2044u) {
        const uint32_t xh = (ah << 11 | al >> 21) | 0x80000000u, xl = al << 11;
        const uint32_t yh = (bh << 11 | bl >> 21) | 0x80000000u, yl = bl << 11;
        const uint64_t p0 = (uint64_t)xl * yl;
        const uint64_t p1 = (uint64_t)xl * yh + (p0 >> 32);
        const uint64_t p2 = (uint64_t)xh * yl + (uint32_t)p1;
        const uint64_t p3 = (uint64_t)xh * yh + (p1 >> 32) + (p2 >> 32);
        const uint32_t top = (uint32_t)(p3 >> 63);
        uint32_t wh = (uint32_t)(p3 >> 32), wl = (uint32_t)p3;
        const uint32_t low = (uint32_t)p2;
        wh = __funnelshift_l(wl, wh, 1u - top);
        wl = __funnelshift_l(low, wl, 1u - top) | ((low | (uint32_t)p0) != 0 ? 1u : 0u);
        const uint32_t ml = __funnelshift_r(wl, wh, 11);
        const uint32_t up = (wl & 0x7FFu) + (ml & 1u) > 0x400u ? 1u : 0u;
        const uint64_t m = ((uint64_t)(sign + ((e + top) << 20) + (wh >> 11)) << 32 | ml) + up;
        return from_bits(m);
    }
    return mul_rest(a, b);
}

// Addition (my own construction).  For normal operands, x the one of larger magnitude and y the
// other, the significands are placed at bits 62..10 of 64-bit words (ten guard bits) and y's is
// shifted right by the exponent difference d, what falls off kept as a sticky bit.  Same signs:
// the sum, renormalised by one place when it carries into bit 63.  Opposite signs: the
// difference, minus one more unit when the sticky bit is set (the true value then lies strictly
// between that integer and the next), renormalised to bit 62; a sticky bit only arises for
// d >= 11, where at most one place of renormalisation is needed and the guard bits still decide
// the rounding.  Round to nearest, ties to even, on the ten guard bits and the sticky bit.  x - x
// gives +0; a zero operand gives the other operand (-0 only for -0 + -0); subnormal, infinite and
// NaN operands, subnormal results and overflow take the FP64 addition (ok = false).
__host__ __device__ __forceinline__ int clz64(uint64_t x)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return __builtin_clzll(x);
#endif
}

__host__ __device__ __forceinline__ uint64_t add_bits(uint64_t ua, uint64_t ub, bool& ok)
{
    const uint32_t ea = (uint32_t)(ua >> 52) & 0x7FFu, eb = (uint32_t)(ub >> 52) & 0x7FFu;
    ok = false;
    if (!((ea - 1u) < 2046u && (eb - 1u) < 2046u)) {
        const bool za = (ua << 1) == 0, zb = (ub << 1) == 0;
        if (za && zb) { ok = true; return ua & ub; }
        if (zb && (ea - 1u) < 2046u) { ok = true; return ua; }
        if (za && (eb - 1u) < 2046u) { ok = true; return ub; }
        return 0;
    }
    const bool swap = (ub & kAbs) > (ua & kAbs);
    const uint64_t ux = swap ? ub : ua, uy = swap ? ua : ub;
    const uint32_t d = swap ? eb - ea : ea - eb;
    int e = (int)(swap ? eb : ea);
    const uint64_t mx = ((ux & kMant) | kHidden) << 10;     // [2^62, 2^63)
    const uint64_t my = ((uy & kMant) | kHidden) << 10;
    uint64_t ys;
    bool sticky;
    if (d >= 64) {
        ys = 0;
        sticky = true;
    } else {
        ys = my >> d;
        sticky = d != 0 && (my << (64 - d)) != 0;
    }
    uint64_t sum;
    if (((ux ^ uy) >> 63) == 0) {
        sum = mx + ys;                                       // < 2^64
        if (sum >> 63) {
            sticky = sticky || (sum & 1) != 0;
            sum >>= 1;
            e += 1;
        }
    } else {
        sum = mx - ys - (sticky ? 1u : 0u);
        if (sum == 0) { ok = true; return 0; }               // x - x = +0
        const int sh = clz64(sum) - 1;
        sum <<= sh;
        e -= sh;
        if (e < 1) return 0;                                 // subnormal result
    }
    if (e > 2046) return 0;                                  // overflow
    const uint64_t m = sum >> 10, rem = sum & 0x3FFu;
    const bool up = rem > 0x200u || (rem == 0x200u && (sticky || (m & 1)));
    ok = true;
    return (ux & ~kAbs) + ((uint64_t)(e - 1) << 52) + m + (up ? 1u : 0u);
}

__device__ __forceinline__ double add(double a, double b)
{
    bool ok;
    const uint64_t r = add_bits(bits(a), bits(b), ok);
    return ok ? from_bits(r) : a + b;
}

// Square root (my own construction, in the manner of the division above).  A positive normal
// x = m 2^(e-1075), m in [2^52, 2^53), has its significand doubled when e - 1075 is odd, giving
// M = m 2^odd in [2^52, 2^54) over an even exponent.  The result significand is
// Q = floor(sqrt(M 2^52)) in [2^52, 2^53), rounded up when the remainder R = M 2^52 - Q^2 exceeds
// Q (a square root is never exactly halfway between two doubles, so there are no ties).  Q is
// estimated from y ~ 1/sqrt(a), a = M / 2^52 in [1, 4): an FP32 seed (rsqrt.approx of the top
// 24 bits of a), two Newton steps y <- y + y (1 - a y^2) / 2 in 64-bit fixed point, then
// g = a y.  The estimate, lowered by one, is corrected on the exact remainder (computed modulo
// 2^64, exact because |R| < 2^58 for an estimate within a few units); if R is still outside
// [0, 2Q] the hardware square root is used.  Zeros are returned as they are; negative, subnormal,
// infinite and NaN operands take the hardware square root.
static __device__ __noinline__ double sqrt_hw(double x) { return ::sqrt(x); }

__device__ __forceinline__ double sqrt(double x)
{
    const uint64_t u = bits(x);
    const uint32_t e = (uint32_t)(u >> 52);                  // sign and exponent
    if (e - 1u >= 2046u) return (u << 1) == 0 ? x : sqrt_hw(x);
    const uint32_t odd = (e & 1u) ^ 1u;                      // e - 1075 is odd
    const uint64_t M = ((u & kMant) | kHidden) << odd;       // [2^52, 2^54)
    const uint64_t A = M << 10;                              // a in Q62
    const uint32_t fa = ((127u + odd) << 23) | ((uint32_t)(M >> (29 + odd)) & 0x7FFFFFu);   // a, truncated
    float rf;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float(fa)));
    const uint32_t ur = __float_as_uint(rf);
    const uint32_t er = ur >> 23;
    int64_t Y;                                               // y in Q62, in [2^61, 2^62]
    if (er >= 127u) Y = 1ll << 62;
    else if (er < 126u) Y = 1ll << 61;
    else Y = (int64_t)((ur & 0x7FFFFFu) | 0x800000u) << 38;
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const uint64_t y2 = __umul64hi((uint64_t)Y, (uint64_t)Y);   // y^2 in Q60
        const uint64_t ay2 = __umul64hi(A, y2);                     // a y^2 in Q58
        const int64_t err = (int64_t)((1ull << 58) - ay2);          // 1 - a y^2 in Q58
        Y += __mul64hi(Y, err) << 5;                                // + y (1 - a y^2) / 2
    }
    uint64_t Q = (__umul64hi(A, (uint64_t)Y) >> 8) - 1;             // g = a y in Q60, to Q52
    int64_t R = (int64_t)((M << 52) - Q * Q);
    if (R < 0) {
        Q -= 1;
        R += (int64_t)(2 * Q + 1);
    }
#pragma unroll
    for (int it = 0; it < 3; it++) {
        const bool up = R > (int64_t)(2 * Q);
        R -= up ? (int64_t)(2 * Q + 1) : 0;
        Q += up ? 1u : 0u;
    }
    if (R < 0 || R > (int64_t)(2 * Q)) return sqrt_hw(x);   // outside the error bounds
    Q += R > (int64_t)Q ? 1u : 0u;
    const int be = ((int)e - 1075 - (int)odd) / 2 + 1049;          // biased exponent of the result
    return from_bits(((uint64_t)(be - 1) << 52) + Q);
}

}  // namespace sfp
}  // namespace armon

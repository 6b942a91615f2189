// quot64.cuh -- correctly rounded FP64 quotients and square roots without a
// branch per operation.
//
// a / b compiles to a sequence that ends in a branch to a slow path, so two
// divisions never overlap: each waits out the other's dependency chain, and
// every quotient of one density repeats the reciprocal.  Here a denominator's
// reciprocal is formed once (den) and each quotient costs a product and one
// residual correction (quo), all of it straight-line code that the compiler
// interleaves freely.  FP64 tile kernels, a branch per division against these:
// Sod 1024 cells 14.6 -> 7.6 us per step, 2-D KH 2048^2 with a passive scalar
// 1.51 -> 0.98 ms, 3-D 128^2 x 256 with a passive scalar 5.2 -> 3.2 ms, all
// with the same bits.
//
// Method: Newton's iteration on the hardware's reciprocal approximation, then
// the residual correction of Markstein (IBM J. Res. Dev. 34, 1990; Cornea,
// Harrison and Tang, "Scientific Computing on Itanium", 2002, ch. 4): with y
// the reciprocal of b and q0 = RN(a y), RN(q0 + y RN(a - b q0)) is the rounded
// quotient.  The square root is the same scheme on the reciprocal square root.
// Both need operands far from overflow and underflow: callers gather a group's
// operands in a Range and take the plain operators where one lies outside.
//
// What the quotient rests on.  The theorem wants the rounded reciprocal.  Two
// quadratic steps from a seed good to 2^-19 or better leave 2^-76, so about one
// y in 2^22 lies on the wrong side of a midpoint.  The quotient is still the
// rounded one unless |1 - b y| exceeds 2^-52 / b (b scaled to [1, 2); a quotient
// that is no midpoint is 2^-53 / b of a unit or more away from one): with y off by
// half a unit and 2^-76 that takes b > 2 (1 - 2^-23).  Those denominators share
// their high word, and with it the seed, which is one half exactly: for
// b = 2 - k 2^-52 the first step gives 1/2 + k 2^-54, rounded up, and the second
// the rounded reciprocal: 1/b lies k^2 2^-107 past a midpoint for odd k, and the step
// falls short of 1/b by less than 2^-107.  (Rounded to nearest, the first step left
// k = 1, a significand of all ones, at 1/2 and the second a unit short: densities
// next to 1 in a gas at rest.)  b > 0 throughout: rounding up is away from zero.
// tests/test_gpu_extreme_operands.py
// divides by all odd k to 2^14 the numerators whose quotients lie next to a
// midpoint, and takes every stage entry point through extreme operands;
// tests/test_gpu_quot64.py converts states over all exponents, bit for bit
// against the CPU's operators.
#pragma once

#include <cstdint>

namespace hcl::q64 {

// Denominators and pressures of a group must lie within 2^-300 and 2^200.
constexpr int kExp = 300;
constexpr int kTopExp = 200;
// Numerators (momenta, differences, the two quotients of a slope) may be as
// small as 2^-800: a quotient then stays above 2^-1000 and a residual, 2^-106
// of its numerator at the least, above 2^-906.  A kinetic energy whose own
// numerator (the squared momentum) is too small for a right residual, below
// 2^-916, is below 2^-616 itself and vanishes next to an internal energy of
// 2^-310 under either rounding.  Gas at rest ahead of a front needs the range:
// there velocities fall by orders of magnitude per cell, down to exact zeros.
constexpr int kNumExp = 800;
// A one-sided quotient is a difference over a width: from 2^-116 up, a quotient
// above 2^-800 had a difference above 2^-916.
constexpr int kWidthExp = 116;

// The high word of a double read as a float orders like the double's
// magnitude (sign, the upper eight exponent bits, then the rest); infinities
// and NaNs read as float NaNs.
__device__ __forceinline__ float hi_float(double a)
{
    return __int_as_float(__double2hiint(a));
}
__device__ __forceinline__ float lo_bound()
{
    return __int_as_float((1023 - kExp) << 20);
}
__device__ __forceinline__ float hi_bound()
{
    return __int_as_float((1023 + kTopExp) << 20);
}
__device__ __forceinline__ float num_bound()
{
    return __int_as_float((1023 - kNumExp) << 20);
}
__device__ __forceinline__ bool nonzero(double a)
{
    return ((__double2hiint(a) & 0x7fffffff) | __double2loint(a)) != 0;
}
// a numerator that quo() may take: zero, or of the size above
__device__ __forceinline__ bool num_ok(double a)
{
    const float f = fabsf(hi_float(a));
    return !nonzero(a) || (f >= num_bound() && f <= hi_bound());
}
__device__ __forceinline__ bool within(double a)
{
    const float f = fabsf(hi_float(a));
    return f >= lo_bound() && f <= hi_bound();
}
__device__ __forceinline__ bool within0(double a)
{
    return within(a) || a == 0.0;
}
// A denominator of either sign: rounding up is towards zero for a negative one,
// whose significand of all ones is therefore left to the plain operators.  (Without
// the low word's test for the positive ones the fast FP64 march came out 3 % slower.)
__device__ __forceinline__ bool den_ok(double b)
{
    return within(b) && __double2loint(b) != -1;
}
__device__ __forceinline__ bool width_ok(double b)
{
    const float f = hi_float(b);
    return f >= __int_as_float((1023 - kWidthExp) << 20) && f <= hi_bound();
}

// The operands of a group, gathered at half an instruction per bound and
// operand (three-input minimum and maximum, NaN-propagating); numerators, which
// may be zero, at two and a half.
struct Range {
    float mn, mx;
    float nz;      // smallest numerator besides zeros
    unsigned ones; // largest low word of the denominators that may be negative or whose reciprocal is derived

    __device__ __forceinline__ explicit Range(bool good = true) : mn(good ? 1.f : 0.f), mx(1.f), nz(1.f), ones(0u) {}
    __device__ __forceinline__ void add(double a)
    {
        const float f = fabsf(hi_float(a));
        asm("min.NaN.f32 %0, %0, %1;" : "+f"(mn) : "f"(f));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(mx) : "f"(f));
    }
    __device__ __forceinline__ void add(double a, double b)
    {
        const float f = fabsf(hi_float(a)), g = fabsf(hi_float(b));
        asm("min.NaN.f32 %0, %0, %1, %2;" : "+f"(mn) : "f"(f), "f"(g));
        top(a, b);
    }
    // positive ones
    __device__ __forceinline__ void pos(double a, double b)
    {
        const float f = hi_float(a), g = hi_float(b);
        asm("min.NaN.f32 %0, %0, %1, %2;" : "+f"(mn) : "f"(f), "f"(g));
        asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(mx) : "f"(f), "f"(g));
    }
    __device__ __forceinline__ void top(double a, double b)
    {
        const float f = fabsf(hi_float(a)), g = fabsf(hi_float(b));
        asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(mx) : "f"(f), "f"(g));
    }
    // numerators
    __device__ __forceinline__ void num(double a, double b)
    {
        top(a, b);
        low_num(a);
        low_num(b);
    }
    __device__ __forceinline__ void low_num(double a)
    {
        if (nonzero(a)) {
            asm("min.f32 %0, %0, %1;" : "+f"(nz) : "f"(fabsf(hi_float(a))));
        }
    }
    // the two quotients of a slope and the upper bound of its own denominator
    // (at least one), where the slope is not zero
    __device__ __forceinline__ void slope(bool use, double r, double l, double b)
    {
        const float f = fabsf(hi_float(r)), g = fabsf(hi_float(l)), h = fabsf(hi_float(b));
        top(r, l);
        if (use) {
            asm("min.f32 %0, %0, %1, %2;" : "+f"(nz) : "f"(f), "f"(g));
            asm("max.NaN.f32 %0, %0, %1;" : "+f"(mx) : "f"(h));
        }
    }
    // such a denominator where nothing else is of concern
    __device__ __forceinline__ void num_if(bool use, double b)
    {
        if (use) {
            asm("min.f32 %0, %0, %1;" : "+f"(nz) : "f"(fabsf(hi_float(b))));
            asm("max.NaN.f32 %0, %0, %1;" : "+f"(mx) : "f"(fabsf(hi_float(b))));
        }
    }
    // low words of such denominators, added elsewhere
    __device__ __forceinline__ void low(double b)
    {
        ones = max(ones, (unsigned)__double2loint(b));
    }
    __device__ __forceinline__ void den(double b)
    {
        add(b);
        low(b);
    }
    // what was found unfit elsewhere
    __device__ __forceinline__ void also(bool good)
    {
        mn = good ? mn : 0.f;
    }
    // all but the numerators' lower bound
    __device__ __forceinline__ bool dens_ok() const
    {
        return mn >= lo_bound() && mx <= hi_bound() && ones != 0xffffffffu;
    }
    __device__ __forceinline__ bool ok() const
    {
        return dens_ok() && nz >= num_bound();
    }
};

struct Den {
    double b; // the denominator
    double y; // its rounded reciprocal
};

__device__ __forceinline__ Den den_from(double b, double y0)
{
    return Den{b, __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0)};
}
__device__ __forceinline__ Den den(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __fma_ru(y, __fma_rn(-b, y, 1.0), y);
    return den_from(b, y);
}
// a / d.b; the residual is formed as b q0 - a so that a zero numerator keeps
// its sign (d.b > 0)
__device__ __forceinline__ double quo(double a, const Den& d)
{
    const double q = __dmul_rn(a, d.y);
    return __fma_rn(-__fma_rn(d.b, q, -a), d.y, q);
}

// the same for a numerator down to the smallest, scaled by a power of two; good
// turns false where the scaling back would round again
__device__ __forceinline__ double quo_tiny(double a, const Den& d, bool& good)
{
    const bool up = fabs(a) < 0x1p-700;
    const double q = quo(a * (up ? 0x1p300 : 1.0), d) * (up ? 0x1p-300 : 1.0);
    good = good && (!nonzero(a) || fabs(q) >= 0x1p-1021);
    return q;
}

__device__ __forceinline__ double root(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = __dmul_rn(x, y);
    double h = __dmul_rn(0.5, y);
    double r = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-h, g, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

} // namespace hcl::q64

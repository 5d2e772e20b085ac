// Sums that the reference forms in float64 and rounds to float32, computed off the
// float64 pipe (GB300: 2 lanes per clock and SM) with the same result.
#pragma once

#include <cuda_runtime.h>

namespace frg {

// float -> double on the integer pipe: the conversion instruction runs on the
// float64 pipe (GB300: 1/64 of the float32 rate), while a normal float's bits
// map to the double's by a re-biased exponent and a shifted fraction.  Exact;
// zeros likewise; subnormals, infinities and NaN take the conversion.
__device__ __forceinline__ double f2d(float f)
{
    const unsigned b = __float_as_uint(f);
    const unsigned e = (b >> 23) & 0xffu;
    if (e == 0u || e == 0xffu) {
        if ((b << 1) == 0u) return __hiloint2double((int)(b & 0x80000000u), 0);
        return (double)f;
    }
    const unsigned hi = (b & 0x80000000u) | ((e + 896u) << 20) | ((b >> 3) & 0xfffffu);
    return __hiloint2double((int)hi, (int)(b << 29));
}

// A float64 sum that ends as a float32, off the float64 pipe: the terms are added
// as an unevaluated pair of float32s (Knuth's two-sum; the pair's error is below
// kDfErr(n) times the sum of the terms' magnitudes for n terms), and value() gives
// the float32 nearest to it.  When the pair is so near the middle between two
// float32s that the float64 sum's own rounding could decide the other way, or
// anything is not finite or too small for the test, value() reports failure and
// the caller forms the float64 sum.  A term costs 10 instructions of one clock
// where a float64 addition holds a scheduler's pipe for 64.
struct DfSum {
    float hi = 0.0f, lo = 0.0f, mag = 0.0f;
    unsigned factors = 0;  // the bits of the products' factors: zero when every product is an exact +0
    __device__ __forceinline__ void add(float p)
    {
        const float s = __fadd_rn(hi, p);
        const float b = __fsub_rn(s, hi);
        lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(p, b)));
        hi = s;
        mag = __fadd_rn(mag, fabsf(p));
    }
    // p + e, the product of a and a weight: p its float32, e an error term far below p
    __device__ __forceinline__ void add_pair(float a, float p, float e)
    {
        add(p);
        lo = __fadd_rn(lo, e);
        factors |= __float_as_uint(a);
    }
    // the exact product a * w
    __device__ __forceinline__ void add_product(float a, float w)
    {
        const float p = __fmul_rn(a, w);
        add_pair(a, p, __fmaf_rn(a, w, -p));
    }
    // err: kDfErr(n)
    __device__ __forceinline__ bool value(float err, float* out) const
    {
        const float s = __fadd_rn(hi, lo);
        const float b = __fsub_rn(s, hi);
        const float r = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(lo, b));  // hi + lo = s + r
        *out = s;
        const unsigned u = __float_as_uint(s);
        const unsigned e = (u >> 23) & 0xffu;
        // half the spacing of float32 at s; below a power of two the spacing halves
        const float half = __uint_as_float((e - 24u) << 23);
        const bool usual = e > 60u && e < 0xffu && (u & 0x7fffffu) != 0u;
        // mag 0: products of factors other than +0 may have underflowed, and only the float64 sum holds them
        return (mag == 0.0f && factors == 0u) || (usual && __fmaf_rn(mag, err, fabsf(r)) < half);
    }
};

// For n terms (a product counts as two): every two-sum is exact, each addition to
// the low word rounds a value below n 2^-24 mag, so the pair is within n^2 2^-48
// mag; a quarter more covers the float64 sum's n 2^-53 mag and the rounding of
// mag.  (A product below 2^-100, whose error term may underflow, cannot reach the
// spacing of a sum that passes the exponent test.)
__host__ __device__ constexpr float kDfErr(int n) { return 1.25f * (float)n * (float)n * 3.5527137e-15f; }

}  // namespace frg

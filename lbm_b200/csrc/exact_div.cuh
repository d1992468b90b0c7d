// exact_div.cuh -- FP64 quotients from a reciprocal computed once per divisor.
//
// The FP64 kernels keep the reference's operation order, divisions included.
// The kinetic collision divides the 15 populations of a cell by the same
// tau_h, (h - E p) / tau_h, so the Poisson kernels compute the reciprocal once
// per cell, as an unevaluated sum of two doubles, and take every quotient from
// it with one multiplication and one FMA (N. Brisebarre and J.-M. Muller,
// "Correctly rounded multiplication by arbitrary precision constants", IEEE
// Trans. Computers 57(2), 2008, the same two operations for a constant known
// to twice the precision):
//   hi = RN(1/b)                          (an IEEE division)
//   lo = RN(RN(1 - b hi) hi)              the remainder 1 - b hi is exact, so
//                                         hi + lo = (1/b)(1 + d), |d| <= 2^-105
//   q  = RN(a hi + RN(a lo))
// The exact value rounded into q differs from a/b by at most 2^-104 |a/b|, so
// q is RN(a/b) unless a/b lies that close to a midpoint of two doubles, and
// never further from a/b than 0.5 ulp + 2^-51 ulp.  A random a/b lies there
// with a probability of 2^-50; lbm_selftest_division (selftest.cu) finds no
// difference from CUDA's IEEE division on 2^32 operand pairs.  Where a lo
// falls below the normal range (|a/b| < 2^-916) it adds at most half an ulp.
// Divisors must be normal and finite.  A numerator of -0 may give +0 (where lo is
// negative).  For infinite numerators lo has to have hi's sign, else a hi + a lo is
// inf - inf or inf * 0: recip_for.
//
// Two operations per quotient instead of the two range comparisons and five
// operations of a remainder-corrected division matter in the two-sweep pass,
// which is bound by FP64 issue and latency and not by memory: 0.64 -> 0.45 ms
// per sweep on 32 x 8 tiles at 256^3 (B200).
#pragma once

#include <cuda_runtime.h>

namespace lbm {

struct RecipPair {
    double hi, lo;   // 1/b = hi + lo to twice the precision
};

// lo of a reciprocal whose hi = RN(1/b) is known.
__device__ __forceinline__ double recip_lo(double b, double hi) { return __dmul_rn(__fma_rn(-b, hi, 1.0), hi); }

__device__ __forceinline__ RecipPair recip_pair(double b)
{
    RecipPair r;
    r.hi = __ddiv_rn(1.0, b);
    r.lo = recip_lo(b, r.hi);
    return r;
}

// The pair for a collision's numerators h - E p.  Where p is not finite (the sum
// of the cell's h, so wherever one of them is not) they are infinite or NaN, and
// hi in lo's place gives the IEEE division's quotient, an infinity of the right
// sign or NaN.  recip_for selects; recip_for_branch branches, so that the quotients
// do not wait for p's test: single sweeps at 24^3 2.410 us, 2.454 with the select
// (2.409 without either), but the two-sweep pass at 96^3 30.0 with the branch, 28.85
// with the select and without either.
__device__ __forceinline__ bool infinite_or_nan(double p) { return (__double2hiint(p) & 0x7ff00000) == 0x7ff00000; }

__device__ __forceinline__ RecipPair recip_for(const RecipPair& r, double p)
{
    return {r.hi, infinite_or_nan(p) ? r.hi : r.lo};
}

__device__ __forceinline__ RecipPair recip_for_branch(RecipPair r, double p)
{
    if (infinite_or_nan(p)) {
        r.lo = r.hi;
        asm volatile("" : "+d"(r.lo));   // (keeps the compiler from making it a select)
    }
    return r;
}

__device__ __forceinline__ double div_rn(double a, const RecipPair& r) { return __fma_rn(a, r.hi, __dmul_rn(a, r.lo)); }

}  // namespace lbm

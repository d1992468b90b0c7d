// Host test of lbm_b200/csrc/exact_div.cuh, its device functions compiled for
// the CPU with the intrinsics they call: quotients against the IEEE division
// and, at a/b next to midpoints of two doubles, against 113-bit arithmetic.
// Exit code 0 on success.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#include <random>

static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __ddiv_rn(double a, double b) { return a / b; }
static inline long long __double_as_longlong(double a)
{
    long long b;
    std::memcpy(&b, &a, 8);
    return b;
}
static inline int __double2hiint(double a) { return static_cast<int>(__double_as_longlong(a) >> 32); }

#include <cuda_runtime.h>

// (the asm statement that keeps a branch a branch names a PTX register)
#define asm
#define volatile(...)
#include "../../lbm_b200/csrc/exact_div.cuh"
#undef asm
#undef volatile

namespace {

bool same(double x, double y)
{
    return (std::isnan(x) && std::isnan(y)) || __double_as_longlong(x) == __double_as_longlong(y);
}
double quotient(double a, double b) { return lbm::div_rn(a, lbm::recip_pair(b)); }

}  // namespace

int main()
{
    std::mt19937_64 rng(20261205);
    std::uniform_real_distribution<double> unit(1.0, 2.0);
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    auto random = [&](int emin, int emax) {
        const double m = std::ldexp(unit(rng), emin + static_cast<int>(rng() % static_cast<unsigned>(emax - emin + 1)));
        return rng() & 1 ? -m : m;
    };
    // random operands, the relaxation times in [0.5, 2) most of all
    for (int i = 0; i < 4000000; ++i) {
        const double a = random(-320, 320), b = i % 3 ? std::ldexp(unit(rng), -1 + static_cast<int>(rng() & 1)) : random(-200, 200);
        if (!same(quotient(a, b), a / b)) return 1;
    }
    // divisors with an exact reciprocal (lo is zero), one above and one below it;
    // zero numerators; infinite ones, as where p is not finite
    for (int i = 0; i < 20000; ++i) {
        const double p2 = std::ldexp(rng() & 1 ? 1.0 : -1.0, static_cast<int>(rng() % 401) - 200);
        const double divisors[] = {random(-200, 200), std::ldexp(unit(rng), -1), p2, std::nextafter(p2, inf), std::nextafter(p2, -inf)};
        for (double b : divisors) {
            const double a = random(-300, 300);
            if (!same(quotient(a, b), a / b) || quotient(0.0, b) != 0.0 || quotient(-0.0, b) != 0.0) return 2;
            for (double h : {a, 0.0, inf, -inf, nan})
                for (double p : {inf, -inf, nan}) {
                    const double num = h - p / 9.0;
                    if (!same(lbm::div_rn(num, lbm::recip_for(lbm::recip_pair(b), p)), num / b)) return 3;
                    if (!same(lbm::div_rn(num, lbm::recip_for_branch(lbm::recip_pair(b), p)), num / b)) return 7;
                }
            const lbm::RecipPair r = lbm::recip_pair(b);
            for (const lbm::RecipPair& s : {lbm::recip_for(r, a), lbm::recip_for_branch(r, a)})
                if (!same(s.hi, r.hi) || !same(s.lo, r.lo)) return 6;
        }
    }
    // a/b within a few units of 2^-106 of a midpoint: with B, M odd and
    // B M = A 2^54 + c for a small c, A / B is M / 2^54 but for c / (B 2^54).  The
    // quotient is one of the two doubles beside it and no further off than half
    // an ulp and 2^-51 ulp.
    for (int i = 0; i < 400000; ++i) {
        const uint64_t B = (rng() >> 11) | (1ULL << 52) | 1ULL;
        uint64_t inv = B;                                   // B^-1 modulo 2^64 (Newton)
        for (int k = 0; k < 6; ++k) inv *= 2 - B * inv;
        const int64_t c = 2 * static_cast<int64_t>(rng() % 8) + 1;
        const uint64_t M = (inv * static_cast<uint64_t>(rng() & 1 ? c : -c)) & ((1ULL << 54) - 1);
        if (M < (1ULL << 53)) continue;                     // 54 bits: a midpoint
        const unsigned __int128 prod = static_cast<unsigned __int128>(B) * M;
        const uint64_t A = static_cast<uint64_t>((prod + (1ULL << 53)) >> 54);
        if (A < (1ULL << 52) || A >= (1ULL << 53)) continue;
        const double a = static_cast<double>(A), b = static_cast<double>(B), q = quotient(a, b);
        const __float128 exact = static_cast<__float128>(a) / b;
        const double ulp = std::ldexp(1.0, std::ilogb(a / b) - 52);
        __float128 off = (static_cast<__float128>(q) - exact) / ulp;
        if (off < 0) off = -off;
        if (off > 0.5 + std::ldexp(1.0, -51)) return 4;
    }
    // below the normal range of a lo: within an ulp (subnormal quotients too)
    for (int i = 0; i < 100000; ++i) {
        const double a = random(-1021, -900), b = random(-1, 0), ref = a / b;
        if (std::fabs(quotient(a, b) - ref) > std::nextafter(std::fabs(ref), inf) - std::fabs(ref)) return 5;
    }
    std::puts("exact_div ok");
    return 0;
}

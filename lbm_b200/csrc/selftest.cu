// selftest.cu -- lbm_selftest_division: the FP64 kernels' division from
// a reciprocal pair (exact_div.cuh) against CUDA's IEEE division on
// pseudo-random operands of the kinds the kernels use, infinite numerators
// among them.  lbm_selftest_transposed_pull: the transposed pull of all
// populations at once (tpull_all) against that of one at a time (tpull).
#include <cuda_runtime.h>

#include <vector>

#include "../../include/lbm_b200.h"
#include "exact_div.cuh"
#include "lbm_device.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long x)
{
    // splitmix64 finaliser (S. Vigna), used as a counter-based generator
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

// A normal double with a random significand, an exponent in [emin, emax] and,
// if `sign`, a random sign.
__device__ __forceinline__ double random_double(unsigned long long r, int emin, int emax, bool sign)
{
    const unsigned long long mant = r & ((1ULL << 52) - 1);
    const int e = emin + static_cast<int>((r >> 52) % static_cast<unsigned long long>(emax - emin + 1));
    const unsigned long long bits = (sign && (r >> 63) ? (1ULL << 63) : 0ULL) |
                                    (static_cast<unsigned long long>(e + 1023) << 52) | mant;
    return __longlong_as_double(static_cast<long long>(bits));
}

__global__ void division_selftest_kernel(unsigned long long n, unsigned long long seed,
                                         unsigned long long* __restrict__ mismatches)
{
    unsigned long long bad = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long r1 = mix64(seed ^ (2 * i)), r2 = mix64(seed ^ (2 * i + 1));
        // (every 256th numerator infinite, as where a cell's p is)
        const double p = i % 256 ? 0.0 : copysign(HUGE_VAL, random_double(r1, 0, 0, true));
        const double a = random_double(r1, -320, 320, true) + p;
        double b;
        switch (r2 & 7) {
        case 0: b = 10.0; break;
        case 1: b = 5.0; break;
        case 2: b = 6.0; break;
        case 3: b = random_double(r2, -1, 0, false); break;        // relaxation times in [0.5, 2)
        case 4: b = random_double(r2, -10, 10, false); break;      // densities
        default: b = random_double(r2, -200, 200, true); break;   // any normal divisor
        }
        const double q = lbm::div_rn(a, lbm::recip_for(lbm::recip_pair(b), p));
        const double qb = lbm::div_rn(a, lbm::recip_for_branch(lbm::recip_pair(b), p));
        const double ref = __ddiv_rn(a, b);
        if (__double_as_longlong(q) != __double_as_longlong(ref) || __double_as_longlong(qb) != __double_as_longlong(ref))
            ++bad;
    }
    if (bad) atomicAdd(mismatches, bad);
}

template <class I>
__global__ void transposed_pull_kernel(lbm::Geom g, const double* __restrict__ y, unsigned long long* __restrict__ mismatches)
{
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= g.n) return;
    const int x = static_cast<int>(c % g.lx), yy = static_cast<int>(c / g.lx % g.ly), z = static_cast<int>(c / g.lx / g.ly);
    const I n = static_cast<I>(g.n);
    const lbm::Wrap w(g, x, yy, z);
    double m[lbm::Q];
    lbm::tpull_all(m, y, n, g, w, x, yy, z);
    int bad = 0;
    lbm::static_for<0, lbm::Q>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        bad += __double_as_longlong(m[q]) != __double_as_longlong(lbm::tpull<q>(y, n, g, w, x, yy, z));
    });
    if (bad) atomicAdd(mismatches, static_cast<unsigned long long>(bad));
}

}  // namespace

extern "C" lbm_status lbm_selftest_transposed_pull(int lx, int ly, int lz, int periodic_x, uint64_t* mismatches)
{
    if (!mismatches || lx < 2 || ly < 1 || lz < 1 || static_cast<long long>(lx) * ly * lz > (1 << 24)) return LBM_ERR_BAD_ARG;
    lbm::Geom g{};
    g.lx = lx;
    g.ly = ly;
    g.lz = lz;
    g.periodic_x = periodic_x ? 1 : 0;
    g.n = static_cast<long long>(lx) * ly * lz;
    const size_t count = lbm::Q * static_cast<size_t>(g.n);
    std::vector<double> host(count);
    for (size_t i = 0; i < count; ++i) host[i] = static_cast<double>(i + 1) / 7.0;
    double* y = nullptr;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&y, count * sizeof(double)) != cudaSuccess || cudaMalloc(&d, sizeof(*d)) != cudaSuccess) {
        cudaFree(y);
        cudaGetLastError();
        return LBM_ERR_OOM;
    }
    cudaMemcpy(y, host.data(), count * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemset(d, 0, sizeof(*d));
    const unsigned blocks = static_cast<unsigned>((g.n + 255) / 256);
    transposed_pull_kernel<int><<<blocks, 256>>>(g, y, d);
    transposed_pull_kernel<long long><<<blocks, 256>>>(g, y, d);
    unsigned long long h = 0;
    const bool ok = cudaGetLastError() == cudaSuccess && cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(y);
    cudaFree(d);
    if (!ok) return LBM_ERR_CUDA;
    *mismatches = h;
    return LBM_OK;
}

extern "C" lbm_status lbm_selftest_division(uint64_t samples, uint64_t seed, uint64_t* mismatches)
{
    if (!mismatches) return LBM_ERR_BAD_ARG;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, sizeof(unsigned long long)) != cudaSuccess) return LBM_ERR_OOM;
    cudaMemset(d, 0, sizeof(unsigned long long));
    division_selftest_kernel<<<148 * 8, 256>>>(samples, seed, d);
    unsigned long long h = 0;
    const bool ok = cudaGetLastError() == cudaSuccess &&
                    cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(d);
    if (!ok) return LBM_ERR_CUDA;
    *mismatches = h;
    return LBM_OK;
}

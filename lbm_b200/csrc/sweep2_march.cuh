// sweep2_march.cuh -- two FP64 applications of a stream-collide operator in one
// pass over memory (temporal blocking): the FP64 box's two-sweep pass and the
// Krylov form's pairs of applications.
//
// A CTA owns a 30 x 6 xy tile and marches a run of `zlen` planes in z; each of
// its 256 threads owns one cell of the tile plus its one-cell halo (32 x 8, one
// warp per row) for the whole march.  Per plane it completes sweep k at its
// cell of plane z+1 into a shared-memory plane ring, issues the pulls of plane
// z+2 (in flight while the CTA works from the ring), and after a barrier
// computes sweep k+1 of plane z at its own cell from the ring (lbm_device.cuh); a
// second barrier frees the slots that the next plane overwrites.  A cell's
// coefficients are kept beside the ring for sweep k+1.  Coordinates wrap, so the
// stream and the slip overwrite are those of two single launches for any box.
// Cells outside the box (partial tiles) store nothing.  fp64_pass_fits is required (the launchers check).
//
// What bounds it: FP64 latency and the two barriers at 16 warps per SM; 126
// registers (15 populations in flight and 15 at work) allow no more, and fewer
// registers spill (0.54 ms per sweep at 96 registers, 0.62 at 80).  Measured on
// B200 at 256^3, ms per sweep: 0.444 (4.8 TB/s of the 128 B/cell it moves)
// against 0.657 for single sweeps; other shapes: 32 x 8 tiles with 11 warps in
// one CTA 0.45, 30 x 14 in one CTA 0.47, 16 x 12 0.47; neighbouring warps
// joined by named barriers in place of the CTA barriers 0.44; separate warps
// for the two sweeps 0.47; the rows requested into L2 a plane ahead 0.48.
#pragma once

#include <cuda_runtime.h>

#include "lbm_device.cuh"
#include "sweep_rules.hpp"

namespace lbm {

constexpr int F2_RX = F2_TX + 2, F2_RY = F2_TY + 2;      // region: tile and halo
constexpr int F2_RC = F2_RX * F2_RY;
constexpr int F2_PLANES = ring_planes();
// Shared memory with `coefs` coefficients per cell (73,728 B with 3).
constexpr int f2_smem(int coefs) { return (F2_PLANES + 2 * coefs) * F2_RC * static_cast<int>(sizeof(double)); }

inline dim3 f2_grid(const Geom& g, int zlen)
{
    return dim3((g.lx + F2_TX - 1) / F2_TX, (g.ly + F2_TY - 1) / F2_TY, (g.lz + zlen - 1) / zlen);
}

namespace {

// Ops: fields(c) loads a cell's fields (requested with the pulls), cell(fields)
// makes its kCoefs coefficients, collide<q>(h, p, coefs) the new population; p
// is the sum of the pulled populations in q order.
template <class Ops>
__device__ __forceinline__ void sweep2_march(const Geom& g, int zlen, const double* __restrict__ hin,
                                             double* __restrict__ hout, const Ops& ops, double* ring)
{
    constexpr int K = Ops::kCoefs;
    double* coef = ring + F2_PLANES * F2_RC;      // [2][K][F2_RC]
    const int t = threadIdx.x;
    const int lane = t % F2_RX, row = t / F2_RX;
    const unsigned n = static_cast<unsigned>(g.n);
    const unsigned plane = static_cast<unsigned>(g.lx) * g.ly;
    const int z0 = blockIdx.z * zlen;
    const int z1 = min(z0 + zlen, g.lz);
    const int x = blockIdx.x * F2_TX - 1 + lane, y = blockIdx.y * F2_TY - 1 + row;
    const int xw = (x + g.lx) % g.lx, yw = (y + g.ly) % g.ly;
    // in-plane parts of the pull offsets, indexed by 1 - c
    const unsigned xs[3] = {static_cast<unsigned>(xw == 0 ? g.lx - 1 : xw - 1), static_cast<unsigned>(xw),
                            static_cast<unsigned>(xw == g.lx - 1 ? 0 : xw + 1)};
    const unsigned ys[3] = {static_cast<unsigned>(yw == 0 ? g.ly - 1 : yw - 1) * g.lx,
                            static_cast<unsigned>(yw) * g.lx,
                            static_cast<unsigned>(yw == g.ly - 1 ? 0 : yw + 1) * g.lx};
    auto sum = [](const double (&h)[Q]) {
        double acc = 0.0;
        static_for<0, Q>([&](auto qc) { acc = acc + h[decltype(qc)::value]; });
        return acc;
    };

    double a[Q];
    typename Ops::Fields fld{};
    auto prefetch = [&](int zz) {
        const int zw = zz < 0 ? zz + g.lz : (zz >= g.lz ? zz - g.lz : zz);
        const unsigned zs[3] = {(zw == 0 ? g.lz - 1 : zw - 1) * plane, zw * plane, (zw == g.lz - 1 ? 0 : zw + 1) * plane};
        static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            a[q] = __ldg(hin + (q * n + zs[1 - cz(q)]) + (ys[1 - cy(q)] + xs[1 - cx(q)]));
        });
        fld = ops.fields(zs[1] + ys[1] + xs[1]);
    };
    auto finish = [&](int i) {
        bounce_regs(a, g, xw);
        const double pv = sum(a);
        double k[K];
        Ops::cell(fld, k);
        double* cf = coef + (i & 1) * K * F2_RC + t;
#pragma unroll
        for (int j = 0; j < K; ++j) cf[j * F2_RC] = k[j];
        static_for<0, Q>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            ring[ring_plane<q>(i) * F2_RC + t] = Ops::template collide<q>(a[q], pv, k);
        });
    };

    prefetch(z0 - 1);
    finish(0);
    prefetch(z0);
    finish(1);
    prefetch(z0 + 1);
    const bool inner = lane >= 1 && lane <= F2_TX && row >= 1 && row <= F2_TY && x < g.lx && y < g.ly;
    for (int z = z0; z < z1; ++z) {
        const int i = z - z0 + 1;
        finish(i + 1);
        if (z + 1 < z1) prefetch(z + 2);
        __syncthreads();
        if (inner) {
            double hv[Q];
            static_for<0, Q>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                hv[q] = ring[ring_plane<q>(i - cz(q)) * F2_RC + t - cy(q) * F2_RX - cx(q)];
            });
            const double* cf = coef + (i & 1) * K * F2_RC + t;
            double k[K];
#pragma unroll
            for (int j = 0; j < K; ++j) k[j] = cf[j * F2_RC];
            bounce_regs(hv, g, x);
            const unsigned c = z * plane + ys[1] + xs[1];
            const double pv = sum(hv);
            static_for<0, Q>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                hout[q * n + c] = Ops::template collide<q>(hv[q], pv, k);
            });
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace lbm

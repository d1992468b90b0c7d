// batch_mixed.cu -- batched mixed-precision boxes (include/lbm_b200.h,
// lbm_batch_*): many independent droplet boxes of different sizes and physics
// on one GPU.
//
// Layout: every instance's populations, macro fields and pressures sit in
// pooled buffers at its own offsets (q-major SoA inside each instance, as in
// a single box).  A work list of (instance, xy tile, z run) items covers all
// instances; every phase of a step is ONE launch of a persistent grid
// (ctas_per_sm x SMs CTAs striding over the items), whatever the number of
// instances.  The per-cell arithmetic is the single mixed box's
// (mixed_cells.cuh), so an instance of a batch steps as the same box alone.
//
// Poisson loop: each instance carries its own device state (DevState: source
// mean, gauge, relative change, ...) and control word (BCtl: active flag,
// parity of its current h buffer, sweep cap).  A segment (check_interval
// sweeps, check kernels A and B, the per-instance finalisations) is one
// captured CUDA graph for the whole batch; items of instances that have left
// the loop are skipped (the two-sweep passes' list is rebuilt without them
// before each segment), and each instance's h parity advances only while it is
// active.  The segments repeat on the device (a conditional WHILE graph node
// and b_loop_decide) until no instance is active, at most 64 per launch; the
// host reads the control words once per launch and relaunches while any
// instance is still active.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../include/lbm_b200.h"
#include "capture.hpp"
#include "finalize.cuh"
#include "mixed_cells.cuh"
#include "phys_host.hpp"

namespace lbm {
namespace {

struct BInst {
    Geom g;
    MixPhys M;
    MixMoments mom;
    long long pop;      // element offset of the instance in the pooled population buffers
    long long fld;      // element offset in the pooled macro-field buffers
    int item0, nitems;  // its work items (contiguous)
};

struct BItem {
    int inst;
    int x0, y0, z0, z1;
};

struct BCtl {
    int active;                 // 1 while the instance is in its Poisson loop
    int parity;                 // h buffer holding its current post-collision state
    unsigned long long cap;     // sweep cap (0: none) or the replayed count
    int replay;                 // 1: stop exactly at cap
    int fail_on_limit;          // 1: a cap without convergence is LBM_ERR_POISSON_BUDGET
};

struct BPool {
    float *f[2], *g[2], *h[2];
    double* f0;         // rest populations in FP64 (pooled like the macro fields)
    float *phi, *rho, *u, *v, *w, *div, *s, *omega;
    double *p, *p_prev, *p_chk;
};

// This thread's cell of item w (tile_x x tile_y tile of 256 threads).
__device__ __forceinline__ void item_cell(const BItem& w, int tile_x, int& x, int& y)
{
    x = w.x0 + static_cast<int>(threadIdx.x) % tile_x;
    y = w.y0 + static_cast<int>(threadIdx.x) / tile_x;
}

// Block partial sums of item it (column t at part[t * n_items + it]); the
// trailing barrier lets the CTA reuse the reduction scratch for its next item.
template <int T>
__device__ __forceinline__ void item_sum(double (&red)[T], double* part, int n_items, int it)
{
    block_sum_store<T>(red, part, n_items, it);
    __syncthreads();
}

template <bool kFirst>
__global__ void __launch_bounds__(256)
b_collide(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
          const float* __restrict__ fin, float* __restrict__ fout, const float* __restrict__ gin,
          float* __restrict__ gout, BPool B, double* __restrict__ part)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        int x, y;
        item_cell(w, tile_x, x, y);
        double red[3] = {0.0, 0.0, 0.0};
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_collide<kFirst>(I.g, I.M, fin + I.pop, fout + I.pop, B.f0 + I.fld, gin + I.pop, gout + I.pop,
                                     B.phi + I.fld,
                                     B.rho + I.fld, B.u + I.fld, B.v + I.fld, B.w + I.fld, B.div + I.fld, x, y, z,
                                     red);
        item_sum<3>(red, part, n_items, it);
    }
}

__global__ void __launch_bounds__(256)
b_moments(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
          const float* __restrict__ f, const float* __restrict__ gp, BPool B, double* __restrict__ part)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        int x, y;
        item_cell(w, tile_x, x, y);
        double red[1] = {0.0};
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_moments(I.g, I.mom, f + I.pop, B.f0 + I.fld, gp + I.pop, B.phi + I.fld, B.rho + I.fld, B.u + I.fld,
                             B.v + I.fld, B.w + I.fld, x, y, z, red);
        item_sum<1>(red, part, n_items, it);
    }
}

__global__ void __launch_bounds__(256)
b_prep(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
       const DevState* __restrict__ ds, BPool B, double* __restrict__ part)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        const double mean = ds[w.inst].div_mean;
        int x, y;
        item_cell(w, tile_x, x, y);
        double red[3] = {0.0, 0.0, 0.0};
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_prep(I.g, mean, B.div + I.fld, B.rho + I.fld, B.p + I.fld, B.s + I.fld, B.omega + I.fld, x, y,
                          z, red);
        item_sum<3>(red, part, n_items, it);
    }
}

// h0 and its first collision, into h[0] (each solve starts at parity 0):
// h0 = E_q p (update_hh, CPU/Inamuro.cpp:825-840), or on the first step after
// a load the loaded h, zero (the reference's arrays after initializeArrays),
// staged in h[1].
__global__ void __launch_bounds__(256)
b_init(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x, int h_loaded,
       BPool B)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        int x, y;
        item_cell(w, tile_x, x, y);
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_init(I.g, h_loaded != 0, B.h[1] + I.pop, B.h[0] + I.pop, B.p + I.fld, B.omega + I.fld,
                          B.s + I.fld, x, y, z);
    }
}

// Plain sweep j of the segment for every active instance: state in
// h[(parity + j) & 1].
__global__ void __launch_bounds__(256)
b_sweep(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
        const BCtl* __restrict__ ctl, int j, BPool B)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BCtl cw = ctl[w.inst];
        if (!cw.active) continue;
        const BInst I = inst[w.inst];
        const bool odd = ((cw.parity + j) & 1) != 0;
        const float* hin = (odd ? B.h[1] : B.h[0]) + I.pop;
        float* hout = (odd ? B.h[0] : B.h[1]) + I.pop;
        int x, y;
        item_cell(w, tile_x, x, y);
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_sweep32(I.g, hin, hout, B.omega + I.fld, B.s + I.fld, x, y, z);
    }
}

// Tiles of the two-sweep passes: 32 x 8 recomputes fewer halo cells, 16 x 8 wastes
// fewer cells past the end of a row.  A batch takes 16 x 8 where 32 x 8 covers more
// than 1.17 times the cells (pick_tile2).  us per sweep of ten boxes, all in their
// loops, 32 x 8 and 16 x 8: 64^3 42.0 and 46.6, 32^3 (64 boxes) 33.3 and 34.7, two of
// 96^3 26.7 and 29.8 (1.0 times the cells); 98^3 (four) 72.9 and 73.1, 112x64x48 48.6
// and 49.0 (1.14); 80^3 (five) 49.7 and 44.2, 66x50x70 (six) 33.1 and 31.7 (1.2); 48^3
// 24.6 and 19.6, 33^3 16.5 and 13.0, 36x40x64 27.3 and 23.0 (1.33); 16x48x96 23.1 and
// 13.6 (2).  16 x 16, 32 x 16, 30 x 8, 30 x 14, 16 x 32 and 14 x 14 were no better than
// these on boxes of 48 to 96 cells a side.
struct Tile2 {
    int tx, ty, ctas;   // cells, resident CTAs per SM
};
constexpr Tile2 kTile2[2] = {{32, 8, 2}, {16, 8, 4}};   // 352 threads, 46,240 B; 192 threads, 24,480 B
constexpr int kPlanRuns = 64;      // longest run (sweep2_zrun's limit)
constexpr int kPlanShortest = 4;   // shortest, unless sweep2_zrun is below it

__host__ __device__ __forceinline__ int tiles2(const Geom& g, int tx, int ty)
{
    return ((g.lx + tx - 1) / tx) * ((g.ly + ty - 1) / ty);
}

// Work list of the two-sweep passes of a segment, rebuilt before it: the items
// of the instances still in their loops, without gaps, so that the CTAs of the
// passes have the same share whichever instances have left.  An instance's
// column of tiles is cut into runs of equal length, at most zmax planes: the
// length for which the passes' waves (items over `slots` resident CTAs) times
// the planes a CTA works through (its run and two halo planes) is least.
// One CTA per instance; each finds the length and its own offset (a few us per
// segment).  With a fixed list whose items of instances that have left are
// skipped: 38.5 us per sweep with five of the ten boxes left and 23.4 with two.
__global__ void __launch_bounds__(256)
b_plan2(const BInst* __restrict__ inst, const BCtl* __restrict__ ctl, int n, int tx, int ty, int zmax, int slots,
        BItem* __restrict__ items, int* __restrict__ n_items)
{
    __shared__ int total[kPlanRuns + 1];
    __shared__ int best, first;
    const int me = blockIdx.x;
    for (int z = threadIdx.x; z <= kPlanRuns; z += blockDim.x) total[z] = 0;
    if (threadIdx.x == 0) first = 0;
    __syncthreads();
    // thread: one length, every fourth instance
    const int z = threadIdx.x % kPlanRuns + 1;
    int mine = 0;
    for (int i = threadIdx.x / kPlanRuns; i < n; i += 256 / kPlanRuns)
        if (ctl[i].active) mine += tiles2(inst[i].g, tx, ty) * ((inst[i].g.lz + z - 1) / z);
    atomicAdd(&total[z], mine);
    __syncthreads();
    if (threadIdx.x == 0) {
        long long least = 0;
        best = zmax;
        for (int k = zmax; k >= 1 && (k >= kPlanShortest || k == zmax); --k) {
            const long long cost = static_cast<long long>((total[k] + slots - 1) / slots) * (k + 2);
            if (k == zmax || cost < least) {
                best = k;
                least = cost;
            }
        }
    }
    __syncthreads();
    int before = 0;
    for (int i = threadIdx.x; i < me; i += blockDim.x)
        if (ctl[i].active) before += tiles2(inst[i].g, tx, ty) * ((inst[i].g.lz + best - 1) / best);
    atomicAdd(&first, before);
    __syncthreads();
    if (me == 0 && threadIdx.x == 0) *n_items = total[best];
    if (!ctl[me].active) return;
    const Geom g = inst[me].g;
    const int nx = (g.lx + tx - 1) / tx, per = tiles2(g, tx, ty);
    // (len <= best, so that (nz - 1) len < lz: no run is empty)
    const int nz = (g.lz + best - 1) / best, len = (g.lz + nz - 1) / nz;
    for (int k = threadIdx.x; k < per * nz; k += blockDim.x) {
        const int r = k % per, z0 = k / per * len;
        items[first + k] = BItem{me, r % nx * tx, r / nx * ty, z0, min(z0 + len, g.lz)};
    }
}

// Two plain sweeps (flip index j: state in h[(parity + j) & 1], result in the
// other buffer) for every item of the plan, with temporal blocking (sweep2_run).
template <int kTile>
__global__ void __launch_bounds__(sweep2_threads(kTile2[kTile].tx, kTile2[kTile].ty), kTile2[kTile].ctas)
b_sweep2(const BItem* __restrict__ items, const int* __restrict__ n_items, const BInst* __restrict__ inst,
         const BCtl* __restrict__ ctl, int j, BPool B)
{
    extern __shared__ float ring[];
    const int count = *n_items;
    for (int it = blockIdx.x; it < count; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        const bool odd = ((ctl[w.inst].parity + j) & 1) != 0;
        const float* hin = (odd ? B.h[1] : B.h[0]) + I.pop;
        float* hout = (odd ? B.h[0] : B.h[1]) + I.pop;
        sweep2_run<kTile2[kTile].tx, kTile2[kTile].ty>(I.g, w.x0, w.y0, w.z0, w.z1, hin, hout, B.omega + I.fld, B.s + I.fld, ring);
        __syncthreads();   // the ring is reused by the CTA's next item
    }
}

__global__ void __launch_bounds__(256)
b_check_a(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
          const BCtl* __restrict__ ctl, int j, BPool B, double* __restrict__ part)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BCtl cw = ctl[w.inst];
        if (!cw.active) continue;
        const BInst I = inst[w.inst];
        const bool odd = ((cw.parity + j) & 1) != 0;
        const float* hin = (odd ? B.h[1] : B.h[0]) + I.pop;
        float* hout = (odd ? B.h[0] : B.h[1]) + I.pop;
        int x, y;
        item_cell(w, tile_x, x, y);
        double red[1] = {0.0};
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z) mixc_check_a(I.g, hin, hout, B.p_chk + I.fld, x, y, z, red);
        item_sum<1>(red, part, n_items, it);
    }
}

__global__ void __launch_bounds__(256)
b_check_b(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x,
          const BCtl* __restrict__ ctl, const DevState* __restrict__ ds, int j, BPool B, double* __restrict__ part)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BCtl cw = ctl[w.inst];
        if (!cw.active) continue;
        const BInst I = inst[w.inst];
        const double shift = ds[w.inst].sigma;
        const double tgt = ds[w.inst].target;
        const bool odd = ((cw.parity + j) & 1) != 0;
        const float* hin = (odd ? B.h[1] : B.h[0]) + I.pop;
        float* hout = (odd ? B.h[0] : B.h[1]) + I.pop;
        int x, y;
        item_cell(w, tile_x, x, y);
        double red[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_check_b<false>(I.g, hin, hout, nullptr, B.p_chk + I.fld, B.p_prev + I.fld, B.p + I.fld,
                                    B.omega + I.fld, B.s + I.fld, shift, tgt, x, y, z, red);
        item_sum<5>(red, part, n_items, it);
    }
}

__global__ void __launch_bounds__(256)
b_correct(const BItem* __restrict__ items, int n_items, const BInst* __restrict__ inst, int tile_x, BPool B)
{
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const BItem w = items[it];
        const BInst I = inst[w.inst];
        int x, y;
        item_cell(w, tile_x, x, y);
        if (x < I.g.lx && y < I.g.ly)
            for (int z = w.z0; z < w.z1; ++z)
                mixc_correct(I.g, B.u + I.fld, B.v + I.fld, B.w + I.fld, B.p + I.fld, B.rho + I.fld, x, y, z);
    }
}

// One finalisation of kind `kind` per instance (one CTA each).  FIN_SIGMA and
// FIN_CHECK skip instances outside their Poisson loop (their items wrote no
// partials).  FIN_PREP opens the loop (active, parity 0); FIN_CHECK advances
// the parity by the segment's n_flips buffer swaps and closes the loop on
// convergence, on the replayed count or at the cap.
__global__ void __launch_bounds__(256)
b_finalize(int kind, DevState* __restrict__ ds, BCtl* __restrict__ ctl, const BInst* __restrict__ inst,
           const double* __restrict__ part, long long stride, int n_flips)
{
    const int i = blockIdx.x;
    if ((kind == FIN_SIGMA || kind == FIN_CHECK) && !ctl[i].active) return;
    const BInst I = inst[i];
    finalize_body(kind, ds + i, part + I.item0, stride, I.nitems, nullptr, 0, 0);
    if (threadIdx.x != 0) return;
    if (kind == FIN_PREP) {
        ctl[i].active = 1;
        ctl[i].parity = 0;
    } else if (kind == FIN_CHECK) {
        BCtl& c = ctl[i];
        DevState& d = ds[i];
        c.parity = (c.parity + n_flips) & 1;
        bool done;
        if (c.replay) {
            done = d.iterations >= c.cap;
        } else {
            done = d.converged != 0;
            if (!done && c.cap && d.iterations >= c.cap) {
                done = true;
                if (c.fail_on_limit && d.error == 0) d.error = LBM_ERR_POISSON_BUDGET;
            }
        }
        if (d.error) done = true;
        c.active = done ? 0 : 1;
    }
}

__global__ void b_to_float(const double* __restrict__ src, float* __restrict__ dst, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (float)src[i];
}

__global__ void b_to_double(const float* __restrict__ src, double* __restrict__ dst, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

__global__ void b_fill(float* __restrict__ dst, long long n, float v)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = v;
}

// f0 = phi - phi_G from the loaded phi (or the uniform fill when none is given).
__global__ void b_rest_from_phi(const double* __restrict__ phi, double fill, double* __restrict__ f0, double fei_G,
                                long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        f0[i] = (phi ? phi[i] : fill) - fei_G;
}

thread_local std::string g_batch_create_error;

const char* site_message(int site)
{
    switch (site) {
    case SITE_SOURCE: return "Poisson source contains NaN/Inf";
    case SITE_PROJECTED: return "projected Poisson source contains NaN/Inf";
    case SITE_GAUGE_TARGET: return "pressure mean is NaN/Inf";
    case SITE_GAUGE_SHIFT: return "pressure gauge shift is NaN/Inf";
    case SITE_RESIDUAL: return "Poisson pressure/residual contains NaN/Inf";
    default: return "non-finite value";
    }
}

constexpr int kLoopKey = 1 << 20;           // graph-map key offset of the device-side loop
constexpr unsigned kBatchLoopSegments = 64;   // segments per launch of the device-side loop

// After a segment: continue while any instance is still in its Poisson loop,
// for at most kBatchLoopSegments segments per launch.
__global__ void __launch_bounds__(256)
b_loop_decide(const BCtl* __restrict__ ctl, int n, unsigned* __restrict__ segs, cudaGraphConditionalHandle w)
{
    int any = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) any |= ctl[i].active;
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        const unsigned s = ++*segs;
        cudaGraphSetConditional(w, (any && s < kBatchLoopSegments) ? 1u : 0u);
    }
}

}  // namespace
}  // namespace lbm

using namespace lbm;

struct lbm_batch {
    int device = 0;
    int n = 0;
    int sm_count = 148;
    cudaStream_t stream = nullptr;
    std::vector<lbm_params> prm;
    std::vector<BInst> inst_h;
    long long total_cells = 0;
    long long max_cells = 0;
    long long pop_elems = 0;         // elements of one pooled population buffer
    long long item_capacity = 0;     // partial-sum slots allocated (largest work list of any tuning)
    int n_items = 0;
    int tile2 = 0;                   // tile of the two-sweep passes (kTile2)
    int* n_items2_d = nullptr;       // two-sweep work list of the running segment (b_plan2)
    BInst* inst_d = nullptr;
    BItem* items_d = nullptr;
    BItem* items2_d = nullptr;
    DevState* ds = nullptr;
    DevState* ds_host = nullptr;     // pinned, n entries
    BCtl* ctl = nullptr;
    BCtl* ctl_host = nullptr;        // pinned, n entries
    BPool pool{};
    double *part_src = nullptr, *part_mass = nullptr, *part_prep = nullptr, *part_a = nullptr, *part_b = nullptr;
    double* scratch = nullptr;       // FP64 staging of one instance's field
    lbm_poisson_cfg pcfg{100, 1.0e-3, 0, 0, 0};
    lbm_batch_tuning tune{32, 8, 4, 4, 0, 0, 0.0};
    int fcur = 0;
    bool first_step = true;
    std::map<int, cudaGraphExec_t> graphs;    // key: plain sweeps per segment (+ kLoopKey: the loop)
    unsigned* loop_segs = nullptr;            // device-side loop: segments run by a launch, pinned copy
    unsigned* loop_segs_host = nullptr;
    bool loop_ok = true;                      // false once the loop graph failed to build
    cudaEvent_t ev[6]{};
    lbm_timing acc{};
    std::string err;
};

namespace {

lbm_status bfail(lbm_batch* b, lbm_status s, const std::string& msg)
{
    if (b) b->err = msg;
    return s;
}

#define BCUDA(b, call)                                                                        \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            return bfail((b), e_ == cudaErrorMemoryAllocation ? LBM_ERR_OOM : LBM_ERR_CUDA,   \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                 \
    } while (0)

bool valid_tuning(const lbm_batch_tuning& t)
{
    const bool tile = (t.tile_x == 32 && t.tile_y == 8) || (t.tile_x == 16 && t.tile_y == 16) ||
                      (t.tile_x == 8 && t.tile_y == 32);
    return tile && t.zrun >= 1 && t.zrun <= 64 && t.ctas_per_sm >= 1 && t.ctas_per_sm <= 16 &&
           t.sweep2_zrun >= 0 && t.sweep2_zrun <= 64;
}

long long count_items(const std::vector<lbm_params>& prm, int tx, int ty, int zrun)
{
    long long c = 0;
    for (const auto& p : prm)
        c += static_cast<long long>((p.lx + tx - 1) / tx) * ((p.ly + ty - 1) / ty) * ((p.lz + zrun - 1) / zrun);
    return c;
}

// Tile of the two-sweep passes for these boxes (kTile2).
int pick_tile2(const std::vector<lbm_params>& prm)
{
    double covered[2];
    for (int t = 0; t < 2; ++t)
        covered[t] = static_cast<double>(count_items(prm, kTile2[t].tx, kTile2[t].ty, 1)) * kTile2[t].tx * kTile2[t].ty;
    return covered[0] > 1.17 * covered[1] ? 1 : 0;
}

// Rebuilds the work list for the batch's tuning (instance-major items).
lbm_status build_items(lbm_batch* b)
{
    const lbm_batch_tuning& t = b->tune;
    std::vector<BItem> items;
    for (int i = 0; i < b->n; ++i) {
        BInst& I = b->inst_h[i];
        I.item0 = static_cast<int>(items.size());
        for (int z0 = 0; z0 < I.g.lz; z0 += t.zrun)
            for (int y0 = 0; y0 < I.g.ly; y0 += t.tile_y)
                for (int x0 = 0; x0 < I.g.lx; x0 += t.tile_x)
                    items.push_back(BItem{i, x0, y0, z0, std::min(z0 + t.zrun, I.g.lz)});
        I.nitems = static_cast<int>(items.size()) - I.item0;
    }
    if (static_cast<long long>(items.size()) > b->item_capacity)
        return bfail(b, LBM_ERR_BAD_ARG, "work list larger than the partial-sum buffers");
    b->n_items = static_cast<int>(items.size());
    if (b->items_d) cudaFree(b->items_d);
    b->items_d = nullptr;
    BCUDA(b, cudaMalloc(&b->items_d, items.size() * sizeof(BItem)));
    BCUDA(b, cudaMemcpy(b->items_d, items.data(), items.size() * sizeof(BItem), cudaMemcpyHostToDevice));
    BCUDA(b, cudaMemcpy(b->inst_d, b->inst_h.data(), b->n * sizeof(BInst), cudaMemcpyHostToDevice));
    for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
    b->graphs.clear();
    return LBM_OK;
}

int grid_of(const lbm_batch* b)
{
    return std::max(1, std::min(b->n_items, b->tune.ctas_per_sm * b->sm_count));
}

void free_batch(lbm_batch* b)
{
    for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
    b->graphs.clear();
    float** fl[] = {&b->pool.f[0], &b->pool.f[1], &b->pool.g[0], &b->pool.g[1], &b->pool.h[0], &b->pool.h[1],
                    &b->pool.phi, &b->pool.rho, &b->pool.u, &b->pool.v, &b->pool.w, &b->pool.div, &b->pool.s,
                    &b->pool.omega};
    for (float** p : fl) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    double** db[] = {&b->pool.p, &b->pool.p_prev, &b->pool.p_chk, &b->pool.f0, &b->part_src, &b->part_mass, &b->part_prep,
                     &b->part_a, &b->part_b, &b->scratch};
    for (double** p : db) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
    if (b->inst_d) cudaFree(b->inst_d);
    if (b->items_d) cudaFree(b->items_d);
    if (b->items2_d) cudaFree(b->items2_d);
    if (b->n_items2_d) cudaFree(b->n_items2_d);
    b->items2_d = nullptr;
    b->n_items2_d = nullptr;
    if (b->ds) cudaFree(b->ds);
    if (b->ctl) cudaFree(b->ctl);
    if (b->ds_host) cudaFreeHost(b->ds_host);
    if (b->ctl_host) cudaFreeHost(b->ctl_host);
    if (b->loop_segs) cudaFree(b->loop_segs);
    if (b->loop_segs_host) cudaFreeHost(b->loop_segs_host);
    b->loop_segs = nullptr;
    b->loop_segs_host = nullptr;
    b->inst_d = nullptr;
    b->items_d = nullptr;
    b->ds = nullptr;
    b->ctl = nullptr;
    b->ds_host = nullptr;
    b->ctl_host = nullptr;
    for (auto& e : b->ev)
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    b->stream = nullptr;
}

lbm_status load_instance(lbm_batch* b, int i, const double* const src[6])
{
    cudaStream_t st = b->stream;
    const BInst& I = b->inst_h[i];
    const long long n = I.g.n;
    const lbm_params& p = b->prm[i];
    float* dst[5] = {b->pool.phi + I.fld, b->pool.rho + I.fld, b->pool.u + I.fld, b->pool.v + I.fld,
                     b->pool.w + I.fld};
    const float bg[5] = {(float)p.fei_min, (float)p.rho_G, 0.f, 0.f, 0.f};
    for (int f = 0; f < 5; ++f) {
        if (src[f]) {
            BCUDA(b, cudaMemcpyAsync(b->scratch, src[f], n * sizeof(double), cudaMemcpyHostToDevice, st));
            b_to_float<<<592, 256, 0, st>>>(b->scratch, dst[f], n);
        } else {
            b_fill<<<592, 256, 0, st>>>(dst[f], n, bg[f]);
        }
        // the rest population holds phi - phi_G until the first collision
        if (f == 0) b_rest_from_phi<<<592, 256, 0, st>>>(src[0] ? b->scratch : nullptr, p.fei_min,
                                                         b->pool.f0 + I.fld, I.mom.fei_G, n);
    }
    if (src[5])
        BCUDA(b, cudaMemcpyAsync(b->pool.p + I.fld, src[5], n * sizeof(double), cudaMemcpyHostToDevice, st));
    else
        BCUDA(b, cudaMemsetAsync(b->pool.p + I.fld, 0, n * sizeof(double), st));
    BCUDA(b, cudaMemsetAsync(b->pool.p_prev + I.fld, 0, n * sizeof(double), st));
    BCUDA(b, cudaGetLastError());
    BCUDA(b, cudaStreamSynchronize(st));
    return LBM_OK;
}

// The two-sweep passes' work list for the segment to come, and one pass.
int grid2_of(const lbm_batch* b) { return kTile2[b->tile2].ctas * b->sm_count; }

void enqueue_plan2(lbm_batch* b, cudaStream_t st)
{
    const Tile2& t = kTile2[b->tile2];
    b_plan2<<<b->n, 256, 0, st>>>(b->inst_d, b->ctl, b->n, t.tx, t.ty, b->tune.sweep2_zrun, grid2_of(b), b->items2_d,
                                  b->n_items2_d);
}

void enqueue_sweep2(lbm_batch* b, int j, cudaStream_t st)
{
    const Tile2& t = kTile2[b->tile2];
    auto kern = b->tile2 == 0 ? b_sweep2<0> : b_sweep2<1>;
    kern<<<grid2_of(b), sweep2_threads(t.tx, t.ty), sweep2_smem(t.tx, t.ty), st>>>(b->items2_d, b->n_items2_d, b->inst_d,
                                                                                  b->ctl, j, b->pool);
}

// One segment's kernels on st (a capturing stream): n_normal plain sweeps
// (in pairs after b_plan2 when two-sweep passes are on), check A, FIN_SIGMA, check B, FIN_CHECK.
void enqueue_segment(lbm_batch* b, int n_normal, cudaStream_t st)
{
    const int grid = grid_of(b);
    const int tx = b->tune.tile_x;
    // j counts buffer swaps: a two-sweep launch swaps once, a single sweep once
    int j = 0;
    int singles = n_normal;
    if (b->tune.sweep2_zrun > 0 && n_normal > 1) {
        enqueue_plan2(b, st);
        for (int k = 0; k + 1 < n_normal; k += 2) enqueue_sweep2(b, j++, st);
        singles = n_normal & 1;
    }
    for (int k = 0; k < singles; ++k)
        b_sweep<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->ctl, j++, b->pool);
    b_check_a<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->ctl, j++, b->pool, b->part_a);
    b_finalize<<<b->n, 256, 0, st>>>(FIN_SIGMA, b->ds, b->ctl, b->inst_d, b->part_a, b->n_items, 0);
    b_check_b<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->ctl, b->ds, j++, b->pool, b->part_b);
    b_finalize<<<b->n, 256, 0, st>>>(FIN_CHECK, b->ds, b->ctl, b->inst_d, b->part_b, b->n_items, j);
}

// One segment graph: the segment's kernels and the copy of the control words
// to the host.
lbm_status get_segment(lbm_batch* b, int n_normal, cudaGraphExec_t* out)
{
    auto it = b->graphs.find(n_normal);
    if (it != b->graphs.end()) {
        *out = it->second;
        return LBM_OK;
    }
    cudaStream_t st = b->stream;
    cudaGraph_t graph = nullptr;
    const cudaError_t e = capture_graph(st, &graph, [&] {
        enqueue_segment(b, n_normal, st);
        return cudaMemcpyAsync(b->ctl_host, b->ctl, b->n * sizeof(BCtl), cudaMemcpyDeviceToHost, st);
    });
    if (e != cudaSuccess) return bfail(b, LBM_ERR_CUDA, std::string("segment capture: ") + cudaGetErrorString(e));
    cudaGraphExec_t ex = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&ex, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return bfail(b, LBM_ERR_CUDA, std::string("segment instantiate: ") + cudaGetErrorString(ie));
    b->graphs[n_normal] = ex;
    *out = ex;
    return LBM_OK;
}

void fill_batch_stats(const DevState& d, lbm_step_stats* s)
{
    std::memset(s, 0, sizeof(*s));
    const double nan = std::nan("");
    s->iterations = d.iterations;
    s->relative_error = d.rel;
    s->pressure_l1_delta = d.l1_delta;
    s->pressure_l1_norm = d.l1_norm;
    s->fixed_point_h_l1 = nan;
    s->fixed_point_h_scale = nan;
    s->fixed_point_h_relative = nan;
    s->fixed_point_p_l1 = nan;
    s->fixed_point_p_scale = nan;
    s->fixed_point_p_relative = nan;
    s->fixed_point_relative = nan;
    s->source_mean = -d.div_mean / 3.0;
    s->source_abs_mean = d.div_abs_sum / (3.0 * d.n_cells);
    s->projected_source_mean = -d.proj_sum / (3.0 * d.n_cells);
    s->pressure_gauge_target = d.target;
    s->pressure_gauge_max_shift = d.max_shift;
    s->mass = d.mass;
    s->pressure_converged = d.pressure_converged;
    s->converged = d.converged;
}

// One step of every instance.  replay: per-instance sweep counts, or null.
// The device-side loop of segments: a graph whose conditional WHILE node runs
// the segment's kernels and b_loop_decide until no instance is active (or
// kBatchLoopSegments ran), then copies the control words and the segment
// count to the host.  False (and nothing reported) when it cannot be built:
// the host then launches one segment graph at a time.
bool get_loop(lbm_batch* b, int n_normal, cudaGraphExec_t* out)
{
    auto it = b->graphs.find(kLoopKey + n_normal);
    if (it != b->graphs.end()) {
        *out = it->second;
        return true;
    }
    if (!b->loop_segs) {
        if (cudaMalloc(&b->loop_segs, sizeof(unsigned)) != cudaSuccess) {
            b->loop_segs = nullptr;
            cudaGetLastError();   // (the host loop takes over: no error of its captures)
            return false;
        }
        if (cudaMallocHost(&b->loop_segs_host, sizeof(unsigned)) != cudaSuccess) {
            cudaFree(b->loop_segs);
            b->loop_segs = nullptr;
            b->loop_segs_host = nullptr;
            cudaGetLastError();
            return false;
        }
    }
    cudaStream_t st = b->stream;
    cudaGraph_t top = nullptr;
    if (cudaGraphCreate(&top, 0) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaGraphExec_t ex = nullptr;
    cudaError_t e = cudaSuccess;
    cudaGraphConditionalHandle hw = 0;
    cudaGraphNode_t wnode = nullptr, c1 = nullptr, c2 = nullptr;
    cudaGraphNodeParams wp{};
    e = cudaGraphConditionalHandleCreate(&hw, top, 1, cudaGraphCondAssignDefault);
    if (e == cudaSuccess) {
        wp.type = cudaGraphNodeTypeConditional;
        wp.conditional.handle = hw;
        wp.conditional.type = cudaGraphCondTypeWhile;
        wp.conditional.size = 1;
        e = cudaGraphAddNode(&wnode, top, nullptr, 0, &wp);
    }
    if (e == cudaSuccess) e = cudaStreamBeginCaptureToGraph(st, wp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                            cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        enqueue_segment(b, n_normal, st);
        b_loop_decide<<<1, 256, 0, st>>>(b->ctl, b->n, b->loop_segs, hw);
        cudaGraph_t captured = nullptr;
        const cudaError_t ec = cudaStreamEndCapture(st, &captured);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = ec;
    }
    if (e == cudaSuccess)
        e = cudaGraphAddMemcpyNode1D(&c1, top, &wnode, 1, b->ctl_host, b->ctl, b->n * sizeof(BCtl),
                                     cudaMemcpyDeviceToHost);
    if (e == cudaSuccess)
        e = cudaGraphAddMemcpyNode1D(&c2, top, &c1, 1, b->loop_segs_host, b->loop_segs, sizeof(unsigned),
                                     cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&ex, top, 0);
    cudaGraphDestroy(top);
    if (e != cudaSuccess) {
        cudaStreamCaptureStatus cs;
        if (cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(st, &g);
            if (g) cudaGraphDestroy(g);
        }
        cudaGetLastError();
        return false;
    }
    b->graphs[kLoopKey + n_normal] = ex;
    *out = ex;
    return true;
}

lbm_status batch_step_once(lbm_batch* b, const uint64_t* replay, lbm_step_stats* stats)
{
    cudaStream_t st = b->stream;
    const int ci = b->pcfg.check_interval;
    const int grid = grid_of(b);
    const int tx = b->tune.tile_x;
    for (int i = 0; i < b->n; ++i) {
        DevState& d = b->ds_host[i];
        std::memset(&d, 0, sizeof(DevState));
        d.check_interval = ci;
        d.tolerance = b->pcfg.tolerance;
        d.dual = 0;
        d.n_cells = static_cast<double>(b->inst_h[i].g.n);
        BCtl& c = b->ctl_host[i];
        c.active = 0;
        c.parity = 0;
        c.replay = replay ? 1 : 0;
        c.cap = replay ? replay[i] : b->pcfg.max_sweeps;
        c.fail_on_limit = b->pcfg.fail_on_limit;
    }
    BCUDA(b, cudaMemcpyAsync(b->ds, b->ds_host, b->n * sizeof(DevState), cudaMemcpyHostToDevice, st));
    BCUDA(b, cudaMemcpyAsync(b->ctl, b->ctl_host, b->n * sizeof(BCtl), cudaMemcpyHostToDevice, st));
    BCUDA(b, cudaEventRecord(b->ev[0], st));
    const int fin = b->fcur, fout = 1 - b->fcur;
    const bool first = b->first_step;
    if (first)
        b_collide<true><<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->pool.f[fin], b->pool.f[fout],
                                              b->pool.g[fin], b->pool.g[fout], b->pool, b->part_src);
    else
        b_collide<false><<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->pool.f[fin], b->pool.f[fout],
                                               b->pool.g[fin], b->pool.g[fout], b->pool, b->part_src);
    BCUDA(b, cudaEventRecord(b->ev[1], st));
    b_moments<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->pool.f[fout], b->pool.g[fout], b->pool,
                                    b->part_mass);
    BCUDA(b, cudaEventRecord(b->ev[2], st));
    b_finalize<<<b->n, 256, 0, st>>>(FIN_SOURCE, b->ds, b->ctl, b->inst_d, b->part_src, b->n_items, 0);
    b_finalize<<<b->n, 256, 0, st>>>(FIN_MASS, b->ds, b->ctl, b->inst_d, b->part_mass, b->n_items, 0);
    b_prep<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->ds, b->pool, b->part_prep);
    b_finalize<<<b->n, 256, 0, st>>>(FIN_PREP, b->ds, b->ctl, b->inst_d, b->part_prep, b->n_items, 0);
    if (first) BCUDA(b, cudaMemsetAsync(b->pool.h[1], 0, b->pop_elems * sizeof(float), st));
    b_init<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, first ? 1 : 0, b->pool);
    BCUDA(b, cudaGetLastError());
    BCUDA(b, cudaEventRecord(b->ev[3], st));
    b->fcur = fout;
    b->first_step = false;

    cudaGraphExec_t seg = nullptr;
    const lbm_status gs = get_segment(b, ci - 1, &seg);
    if (gs != LBM_OK) return gs;
    uint64_t segments = 0, decides = 0;
    const char* lenv = std::getenv("LBM_POISSON_LOOP");
    cudaGraphExec_t loop = nullptr;
    const bool use_loop = b->loop_ok && !(lenv && lenv[0] == '0') && (b->loop_ok = get_loop(b, ci - 1, &loop));
    for (;;) {
        if (use_loop) {
            *b->loop_segs_host = 0;
            BCUDA(b, cudaMemcpyAsync(b->loop_segs, b->loop_segs_host, sizeof(unsigned), cudaMemcpyHostToDevice, st));
            BCUDA(b, cudaGraphLaunch(loop, st));
            BCUDA(b, cudaStreamSynchronize(st));
            const unsigned ran = *b->loop_segs_host;
            if (ran < 1) return bfail(b, LBM_ERR_CUDA, "device Poisson loop ran no segment");
            segments += ran;
            decides += ran;
        } else {
            BCUDA(b, cudaGraphLaunch(seg, st));
            BCUDA(b, cudaStreamSynchronize(st));
            ++segments;
        }
        bool any = false;
        for (int i = 0; i < b->n; ++i) any = any || b->ctl_host[i].active;
        if (!any) break;
        if (segments > (1ull << 40)) return bfail(b, LBM_ERR_OVERFLOW, "Poisson segment counter overflow");
    }
    BCUDA(b, cudaEventRecord(b->ev[4], st));
    b_correct<<<grid, 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, tx, b->pool);
    BCUDA(b, cudaGetLastError());
    BCUDA(b, cudaEventRecord(b->ev[5], st));
    BCUDA(b, cudaMemcpyAsync(b->ds_host, b->ds, b->n * sizeof(DevState), cudaMemcpyDeviceToHost, st));
    BCUDA(b, cudaStreamSynchronize(st));
    float t[5];
    for (int i = 0; i < 5; ++i) cudaEventElapsedTime(&t[i], b->ev[i], b->ev[i + 1]);
    b->acc.collide_ms += t[0];
    b->acc.moments_ms += t[1];
    b->acc.prep_ms += t[2];
    b->acc.poisson_ms += t[3];
    b->acc.correct_ms += t[4];
    b->acc.steps += 1;
    // per segment: ci - 1 plain sweeps (in pairs after a plan when two-sweep
    // passes are on)
    // + check A + check B (together one sweep) + two finalisations; per step:
    // 7 prologue launches and the correction
    b->acc.sweep_kernels += segments * static_cast<uint64_t>(ci + 1);
    const bool fused = b->tune.sweep2_zrun > 0 && ci > 2;
    const uint64_t plain = fused ? static_cast<uint64_t>(1 + (ci - 1) / 2 + (ci - 1) % 2) : ci - 1;
    b->acc.kernel_launches += 8 + segments * (plain + 4) + decides;
    if (fused) b->acc.fused_sweeps += segments * static_cast<uint64_t>((ci - 1) / 2 * 2);
    lbm_status status = LBM_OK;
    for (int i = 0; i < b->n; ++i) {
        const DevState& d = b->ds_host[i];
        b->acc.sweeps += d.iterations;
        if (stats) fill_batch_stats(d, stats + i);
        if (d.error && status == LBM_OK) {
            status = static_cast<lbm_status>(d.error);
            b->err = "instance " + std::to_string(i) + ": " +
                     (d.error == LBM_ERR_POISSON_BUDGET ? std::string("Poisson sweep limit reached without convergence")
                                                        : std::string(site_message(d.error_site)));
        }
    }
    return status;
}

}  // namespace

extern "C" {

lbm_status lbm_batch_create(const lbm_params* params, int n_instances, int device, lbm_batch** out)
{
    if (!params || !out || n_instances < 1) return LBM_ERR_BAD_ARG;
    *out = nullptr;
    for (int i = 0; i < n_instances; ++i) {
        const lbm_params& p = params[i];
        if (p.lx < 2 || p.ly < 1 || p.lz < 1 || !(p.rho_L != p.rho_G) || !(p.tauf > 0.0) || !(p.taug > 0.0)) {
            g_batch_create_error = "instance " + std::to_string(i) + ": invalid box or physics";
            return LBM_ERR_BAD_ARG;
        }
        if (15LL * p.lx * p.ly * p.lz >= 0x7fffffffLL) {
            g_batch_create_error = "instance " + std::to_string(i) + ": box too large for a batch";
            return LBM_ERR_BAD_ARG;
        }
    }
    int ndev = 0;
    const cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev <= 0 || device < 0 || device >= ndev) {
        cudaGetLastError();
        g_batch_create_error = std::string("no usable CUDA device: ") + cudaGetErrorString(ce);
        return LBM_ERR_NO_DEVICE;
    }
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess || prop.major != 10) {
        g_batch_create_error = "device is not sm_100";
        return LBM_ERR_NO_DEVICE;
    }
    if (cudaSetDevice(device) != cudaSuccess) {
        g_batch_create_error = "cudaSetDevice failed";
        return LBM_ERR_NO_DEVICE;
    }
    lbm_batch* b = new lbm_batch();
    b->device = device;
    b->n = n_instances;
    b->sm_count = prop.multiProcessorCount;
    b->prm.assign(params, params + n_instances);
    b->inst_h.resize(n_instances);
    long long pop = 0, fld = 0;
    for (int i = 0; i < n_instances; ++i) {
        const lbm_params& p = params[i];
        BInst& I = b->inst_h[i];
        std::memset(&I, 0, sizeof(I));
        I.g.lx = p.lx;
        I.g.ly = p.ly;
        I.g.lz = p.lz;
        I.g.periodic_x = p.periodic_x ? 1 : 0;
        I.g.n = static_cast<long long>(p.lx) * p.ly * p.lz;
        const Phys P = make_phys(p);
        I.M = mix_phys(P);
        I.mom = MixMoments{P.fei_G, P.fei_L, P.rho_G, P.rho_L, P.fei_avg, P.dfei, P.half_drho};
        // Offsets rounded to 64 elements keep every instance's arrays aligned.
        I.pop = pop;
        I.fld = fld;
        pop += (15 * I.g.n + 63) / 64 * 64;
        fld += (I.g.n + 63) / 64 * 64;
        b->max_cells = std::max(b->max_cells, I.g.n);
        b->total_cells += I.g.n;
    }
    b->pop_elems = pop;
    auto bail = [&](lbm_status s) {
        g_batch_create_error = b->err;
        free_batch(b);
        delete b;
        return s;
    };
    const int tiles[3][2] = {{32, 8}, {16, 16}, {8, 32}};
    for (auto& t : tiles) b->item_capacity = std::max(b->item_capacity, count_items(b->prm, t[0], t[1], 1));
    auto okf = [&](float** p, long long count) { return cudaMalloc(p, count * sizeof(float)) == cudaSuccess; };
    auto okd = [&](double** p, long long count) { return cudaMalloc(p, count * sizeof(double)) == cudaSuccess; };
    bool ok = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) == cudaSuccess;
    for (int k = 0; k < 2 && ok; ++k)
        ok = okf(&b->pool.f[k], pop) && okf(&b->pool.g[k], pop) && okf(&b->pool.h[k], pop);
    ok = ok && okf(&b->pool.phi, fld) && okf(&b->pool.rho, fld) && okf(&b->pool.u, fld) && okf(&b->pool.v, fld) &&
         okf(&b->pool.w, fld) && okf(&b->pool.div, fld) && okf(&b->pool.s, fld) && okf(&b->pool.omega, fld);
    ok = ok && okd(&b->pool.p, fld) && okd(&b->pool.p_prev, fld) && okd(&b->pool.p_chk, fld) && okd(&b->pool.f0, fld) &&
         okd(&b->scratch, b->max_cells);
    const long long cap = b->item_capacity;
    ok = ok && okd(&b->part_src, 3 * cap) && okd(&b->part_mass, cap) && okd(&b->part_prep, 3 * cap) &&
         okd(&b->part_a, cap) && okd(&b->part_b, 5 * cap);
    ok = ok && cudaMalloc(&b->items2_d, count_items(b->prm, kTile2[1].tx, kTile2[1].ty, 1) * sizeof(BItem)) == cudaSuccess &&
         cudaMalloc(&b->n_items2_d, sizeof(int)) == cudaSuccess;
    ok = ok && cudaMalloc(&b->inst_d, n_instances * sizeof(BInst)) == cudaSuccess &&
         cudaMalloc(&b->ds, n_instances * sizeof(DevState)) == cudaSuccess &&
         cudaMalloc(&b->ctl, n_instances * sizeof(BCtl)) == cudaSuccess &&
         cudaMallocHost(&b->ds_host, n_instances * sizeof(DevState)) == cudaSuccess &&
         cudaMallocHost(&b->ctl_host, n_instances * sizeof(BCtl)) == cudaSuccess;
    for (auto& e : b->ev) ok = ok && cudaEventCreate(&e) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        b->err = "device allocation failed";
        return bail(LBM_ERR_OOM);
    }
    cudaMemset(b->pool.s, 0, fld * sizeof(float));
    cudaMemset(b->pool.omega, 0, fld * sizeof(float));
    b->tile2 = pick_tile2(b->prm);
    if (const char* e = std::getenv("LBM_BATCH_TUNING")) {
        lbm_batch_tuning t{};
        const int got = std::sscanf(e, "%d,%d,%d,%d,%d", &t.tile_x, &t.tile_y, &t.zrun, &t.ctas_per_sm,
                                    &t.sweep2_zrun);
        if (got >= 4 && valid_tuning(t)) b->tune = t;
    }
    lbm_status s = build_items(b);
    if (s != LBM_OK) return bail(s);
    const double* none[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    for (int i = 0; i < n_instances && s == LBM_OK; ++i) s = load_instance(b, i, none);
    if (s != LBM_OK) return bail(s);
    *out = b;
    return LBM_OK;
}

void lbm_batch_destroy(lbm_batch* b)
{
    if (!b) return;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    free_batch(b);
    delete b;
}

int lbm_batch_size(const lbm_batch* b) { return b ? b->n : 0; }

// A load restarts every instance of the batch from its current macro fields
// (equilibrium populations, h0 = 0), as constructing the reference's class
// from a CPU object does.
lbm_status lbm_batch_load_fields(lbm_batch* b, int inst, const double* phi, const double* rho, const double* u,
                                 const double* v, const double* w, const double* p)
{
    if (!b || inst < 0 || inst >= b->n) return LBM_ERR_BAD_ARG;
    cudaSetDevice(b->device);
    const double* src[6] = {phi, rho, u, v, w, p};
    const lbm_status s = load_instance(b, inst, src);
    if (s == LBM_OK) b->first_step = true;
    return s;
}

lbm_status lbm_batch_set_poisson(lbm_batch* b, const lbm_poisson_cfg* cfg)
{
    if (!b || !cfg) return LBM_ERR_BAD_ARG;
    if (cfg->check_interval < 2 || !(cfg->tolerance > 0.0) || cfg->dual_residual != 0)
        return bfail(b, LBM_ERR_BAD_ARG, "batched boxes: check_interval >= 2, tolerance > 0, no dual residual");
    if (cfg->max_sweeps % static_cast<uint64_t>(cfg->check_interval) != 0)
        return bfail(b, LBM_ERR_BAD_ARG, "max_sweeps must be a multiple of check_interval");
    b->pcfg = *cfg;
    return LBM_OK;
}

lbm_status lbm_batch_step(lbm_batch* b, int n_steps, lbm_step_stats* stats)
{
    if (!b || n_steps < 0) return LBM_ERR_BAD_ARG;
    cudaSetDevice(b->device);
    for (int s = 0; s < n_steps; ++s) {
        const lbm_status st = batch_step_once(b, nullptr, stats ? stats + static_cast<size_t>(s) * b->n : nullptr);
        if (st != LBM_OK) return st;
    }
    return LBM_OK;
}

lbm_status lbm_batch_step_replay(lbm_batch* b, int n_steps, const uint64_t* sweeps, lbm_step_stats* stats)
{
    if (!b || n_steps < 0 || !sweeps) return LBM_ERR_BAD_ARG;
    const uint64_t ci = static_cast<uint64_t>(b->pcfg.check_interval);
    for (long long k = 0; k < static_cast<long long>(n_steps) * b->n; ++k)
        if (sweeps[k] == 0 || sweeps[k] % ci != 0)
            return bfail(b, LBM_ERR_BAD_ARG, "replayed sweep counts must be positive multiples of check_interval");
    cudaSetDevice(b->device);
    for (int s = 0; s < n_steps; ++s) {
        const lbm_status st = batch_step_once(b, sweeps + static_cast<size_t>(s) * b->n,
                                              stats ? stats + static_cast<size_t>(s) * b->n : nullptr);
        if (st != LBM_OK) return st;
    }
    return LBM_OK;
}

lbm_status lbm_batch_download(lbm_batch* b, int inst, lbm_field which, double* host)
{
    if (!b || !host || inst < 0 || inst >= b->n || which < LBM_FIELD_PHI || which > LBM_FIELD_P)
        return LBM_ERR_BAD_ARG;
    cudaSetDevice(b->device);
    cudaStream_t st = b->stream;
    const BInst& I = b->inst_h[inst];
    const long long n = I.g.n;
    if (which == LBM_FIELD_P) {
        BCUDA(b, cudaMemcpyAsync(host, b->pool.p + I.fld, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    } else {
        float* src[5] = {b->pool.phi, b->pool.rho, b->pool.u, b->pool.v, b->pool.w};
        b_to_double<<<592, 256, 0, st>>>(src[which] + I.fld, b->scratch, n);
        BCUDA(b, cudaGetLastError());
        BCUDA(b, cudaMemcpyAsync(host, b->scratch, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    }
    BCUDA(b, cudaStreamSynchronize(st));
    return LBM_OK;
}

lbm_status lbm_batch_set_tuning(lbm_batch* b, const lbm_batch_tuning* t)
{
    if (!b || !t || !valid_tuning(*t)) return LBM_ERR_BAD_ARG;
    cudaSetDevice(b->device);
    b->tune = *t;
    return build_items(b);
}

lbm_status lbm_batch_get_tuning(const lbm_batch* b, lbm_batch_tuning* out)
{
    if (!b || !out) return LBM_ERR_BAD_ARG;
    *out = b->tune;
    return LBM_OK;
}

lbm_status lbm_batch_tune(lbm_batch* b, lbm_batch_tuning* chosen)
{
    if (!b) return LBM_ERR_BAD_ARG;
    cudaSetDevice(b->device);
    cudaStream_t st = b->stream;
    // Every instance active at parity 0: the batched sweep then does the
    // work of a real segment.  h, s and omega are rebuilt at the next step.
    for (int i = 0; i < b->n; ++i) b->ctl_host[i] = BCtl{1, 0, 0, 0, 0};
    BCUDA(b, cudaMemcpyAsync(b->ctl, b->ctl_host, b->n * sizeof(BCtl), cudaMemcpyHostToDevice, st));
    const int tiles[3][2] = {{32, 8}, {16, 16}, {8, 32}};
    const int zruns[4] = {1, 2, 4, 8};
    const int ctas[3] = {2, 4, 8};
    lbm_batch_tuning best = b->tune;
    best.sweep_ms = 1e30;
    const int reps = 6;
    auto singles = [&](const lbm_batch_tuning& t, int first, int count) {
        for (int r = first; r < first + count; ++r)
            b_sweep<<<grid_of(b), 256, 0, st>>>(b->items_d, b->n_items, b->inst_d, t.tile_x, b->ctl, r, b->pool);
    };
    for (auto& tl : tiles)
        for (int zr : zruns)
            for (int cp : ctas) {
                const lbm_batch_tuning t{tl[0], tl[1], zr, cp, 0, 0, 0.0};
                b->tune = t;
                lbm_status s = build_items(b);
                if (s != LBM_OK) return s;
                singles(t, 0, 2);
                BCUDA(b, cudaEventRecord(b->ev[0], st));
                singles(t, 0, reps);
                BCUDA(b, cudaEventRecord(b->ev[1], st));
                BCUDA(b, cudaGetLastError());
                BCUDA(b, cudaEventSynchronize(b->ev[1]));
                float ms = 0.f;
                cudaEventElapsedTime(&ms, b->ev[0], b->ev[1]);
                // (a clear win only: the checks' FP64 sums follow the list, and of two
                // forms as fast as each other one run would take this, one that)
                if (ms / reps < 0.995 * best.sweep_ms) {
                    best = t;
                    best.sweep_ms = ms / reps;
                }
            }
    // Single sweeps against passes: each in a graph, as the segments run them
    // (launched one by one the sweeps of small boxes wait for the host, single
    // sweeps the longest).  *ms: time per sweep of `sweeps` sweeps.
    auto time_graph = [&](int sweeps, auto&& launch, double* ms) -> lbm_status {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t ex = nullptr;
        cudaError_t e = capture_graph(st, &graph, [&] {
            launch();
            return cudaSuccess;
        });
        BCUDA(b, e);
        e = cudaGraphInstantiate(&ex, graph, 0);
        cudaGraphDestroy(graph);
        BCUDA(b, e);
        e = cudaGraphLaunch(ex, st);
        if (e == cudaSuccess) e = cudaEventRecord(b->ev[0], st);
        if (e == cudaSuccess) e = cudaGraphLaunch(ex, st);
        if (e == cudaSuccess) e = cudaEventRecord(b->ev[1], st);
        if (e == cudaSuccess) e = cudaEventSynchronize(b->ev[1]);
        float t = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&t, b->ev[0], b->ev[1]);
        cudaGraphExecDestroy(ex);
        BCUDA(b, e);
        *ms = t / sweeps;
        return LBM_OK;
    };
    b->tune = best;
    lbm_status ts = build_items(b);
    if (ts == LBM_OK) ts = time_graph(reps, [&] { singles(best, 0, reps); }, &best.sweep_ms);
    if (ts != LBM_OK) return ts;
    // two sweeps per launch on z runs of 8, 16, 32 (per-sweep time = launch / 2).  With
    // every box in its loop, as here, passes may be 4 % slower: once boxes have left,
    // their list is rebuilt without them (ten of 33^3 12.95 us against 12.55, 8.26
    // against 9.3 when they leave at different checks).
    double least = 1.04 * best.sweep_ms;
    const int zr2[3] = {8, 16, 32};
    for (int zr : zr2) {
        lbm_batch_tuning t = best;
        t.sweep2_zrun = zr;
        t.sweep_ms = 0.0;
        b->tune = t;
        lbm_status s = build_items(b);
        if (s != LBM_OK) return s;
        enqueue_plan2(b, st);
        double ms = 0.0;
        s = time_graph(reps, [&] {
            for (int r = 0; r < reps / 2; ++r) enqueue_sweep2(b, r, st);
        }, &ms);
        if (s != LBM_OK) return s;
        if (ms < least) {
            best = t;
            best.sweep_ms = least = ms;
        }
    }
    b->tune = best;
    const lbm_status s = build_items(b);
    if (s != LBM_OK) return s;
    if (chosen) *chosen = best;
    return LBM_OK;
}

lbm_status lbm_batch_get_timing(const lbm_batch* b, lbm_timing* out)
{
    if (!b || !out) return LBM_ERR_BAD_ARG;
    *out = b->acc;
    return LBM_OK;
}

lbm_status lbm_batch_reset_timing(lbm_batch* b)
{
    if (!b) return LBM_ERR_BAD_ARG;
    b->acc = lbm_timing{};
    return LBM_OK;
}

const char* lbm_batch_last_error(const lbm_batch* b)
{
    if (!b) return g_batch_create_error.c_str();
    return b->err.c_str();
}

}  // extern "C"

// sweep_rules.hpp -- which boxes run their Poisson sweeps two per pass, on what
// tiles and z runs.  Arithmetic on extents and the SM count alone, free of CUDA
// types, so the host tests can go over boxes of any size
// (tests/cpp/sweep_rules_test.cpp).
#pragma once

namespace lbm {

// Tiles of the passes and their resident CTAs per SM (sweep2_march.cuh,
// kernels_mixed.cu).
constexpr int F2_TX = 30, F2_TY = 6, F2_CTAS = 2;
constexpr int S2_TX = 32, S2_TY = 8, S2_CTAS = 2;
constexpr int S2_TALL = 16, S2_TALL_CTAS = 1;

// Tile rows are a pass's grid y, which the device limits.  (Tile columns are
// its grid x; z runs are at most the box's planes, 65535.)
constexpr int kMaxGridY = 65535;
inline bool pass_rows_fit(int ly, int tile_y) { return (ly - 1) / tile_y < kMaxGridY; }

// The passes index the 15 n populations with 32 bits.
inline bool pass_offsets_fit(long long n) { return 15 * n < 0x7fffffffLL; }

// z run length of a two-sweep pass: the grid's waves (tiles x runs over the
// resident CTAs) times the planes a CTA works through (its run and two halo
// planes) is least.  *cost: that product.
inline int two_sweep_zlen(long long tiles, int lz, long long slots, long long* cost)
{
    int best = 0;
    long long least = 0;
    for (int nz = 1; nz <= lz; ++nz) {
        const int zlen = (lz + nz - 1) / nz;
        if (zlen > 40 && nz < lz) continue;
        if (zlen < 4 && best) break;
        const long long c = (tiles * ((lz + zlen - 1) / zlen) + slots - 1) / slots * (zlen + 2);
        if (!best || c < least) {
            best = zlen;
            least = c;
        }
    }
    if (cost) *cost = least;
    return best;
}

inline long long pass_tiles(int lx, int ly, int tx, int ty)
{
    return static_cast<long long>((lx - 1) / tx + 1) * ((ly - 1) / ty + 1);
}

// Whether a pass can run on the box at all, whichever way its z runs are chosen.
inline bool fp64_pass_fits(int ly, long long n) { return pass_rows_fit(ly, F2_TY) && pass_offsets_fit(n); }
inline bool mixed_pass_fits(int ly, long long n) { return pass_rows_fit(ly, S2_TY) && pass_offsets_fit(n); }

// FP64: z run length of the passes where they are faster than single sweeps, 0
// elsewhere, from both sides' times on B200 (us per sweep): a pass takes 1.12
// per wave and plane of its CTAs (128^3: 60 at 54, 256^3: 444 at 374, 96^3: 29
// at 26, 64^3: 10.6 at 10).  A single sweep takes 2 + 21 per 10^6 cells while
// both h buffers stay in L2 (64^3: 7.5, 48^3: 4.2, 32^3: 2.6; 240 B per cell),
// 33.5 per 10^6 cells from 3 to 4.5 * 10^5 cells, where part of them does
// (80x64x64: 10.5, 72^3: 13.1, 90x66x60: 12.4; the pass 10.7, 12.1, 10.9), and 39
// from DRAM (128^3: 84, 90 x 75 x 131: 39).
inline int fp64_pass_zlen(int lx, int ly, int lz, int sms)
{
    const long long n = static_cast<long long>(lx) * ly * lz;
    if (!fp64_pass_fits(ly, n)) return 0;
    long long cost = 0;
    const int zlen = two_sweep_zlen(pass_tiles(lx, ly, F2_TX, F2_TY), lz, F2_CTAS * sms, &cost);
    const double mcells = 1e-6 * static_cast<double>(n);
    const double single = mcells <= 0.3    ? 2.0 + 21.0 * mcells
                          : mcells <= 0.45 ? 33.5 * mcells
                                           : 39.0 * mcells;
    return 1.12 * static_cast<double>(cost) < single ? zlen : 0;
}

// Mixed: z run length of the passes (partial tiles store nothing outside the
// box) and whether they take the tall tile; zlen 0 where single sweeps are
// faster.  Both sides' times on B200
// (us per sweep): a pass takes 0.93 per wave and plane of its CTAs on 32 x 8
// tiles (two per SM; 128^3: 29.8 at 34, 256^3: 226 at 238, 141 x 99 x 141: 31.9
// at 36) and 0.91 on 32 x 16 (one per SM; 29.1, 223, 34.2 at 38).  A single
// sweep takes 1.75 + 13 per 10^6 cells while both h buffers stay in L2 (120 B per
// cell; 80^3: 8.4, 64^3: 4.6, 32^3: 2.1), beyond 5.4 * 10^5 cells 20.5 per 10^6
// cells less a remainder that stays there (84^3: 11.0, 88^3: 13.0, where the pass
// takes 11.8), and 20.5 from DRAM (128^3: 45, 96^3: 18.4, 141 x 99 x 75: 27).
//
// The refinement form's correction sweeps read a source r of 15 values per cell
// beside the 15 populations and take the tall tile: refine_zlen by a rule of
// their own.  A pass takes 1.1 per wave and plane and 8 per 10^6 cells (128^3: 56.2
// at 34, 136^3: 74.8 at 50, 136 x 98 x 177: 75.0 at 50, 88^3: 20.0 at 13); a single
// sweep from DRAM, per 10^6 cells, 31 where rows are of whole 16 bytes (62.0, 76.6,
// 71.2, 20.9), else 33 (91 x 98 x 73: 20.8, the pass 19.8), and 34 on tiles 16 cells
// wide (45 x 183 x 190: 56.2, the pass 50.9).  With both sides measured on 144 boxes
// of 5.4 * 10^5 to 1.7 * 10^7 cells this takes a form at most 3.6 % slower than the
// other; the plain sweeps' rule took one up to 14 % slower (5 % where it chose
// passes: 136 x 98 x 177).  Smaller boxes' single sweeps run from L2 (80^3: 14.2).
struct MixedPass {
    int zlen = 0;
    bool tall = false;
    int refine_zlen = 0;
};
inline MixedPass mixed_pass(int lx, int ly, int lz, int sms)
{
    MixedPass m;
    const long long n = static_cast<long long>(lx) * ly * lz;
    if (!mixed_pass_fits(ly, n)) return m;
    long long low_cost = 0, tall_cost = 0;
    const int low = two_sweep_zlen(pass_tiles(lx, ly, S2_TX, S2_TY), lz, static_cast<long long>(S2_CTAS) * sms, &low_cost);
    const int high = two_sweep_zlen(pass_tiles(lx, ly, S2_TX, S2_TALL), lz, static_cast<long long>(S2_TALL_CTAS) * sms,
                                    &tall_cost);
    m.tall = tall_cost <= low_cost;
    const double mcells = 1e-6 * static_cast<double>(n);
    const double single = mcells <= 0.54   ? 1.75 + 13.0 * mcells
                          : mcells <= 0.75 ? 20.5 * mcells - 1.2
                                           : 20.5 * mcells;
    const double pass = m.tall ? 0.91 * static_cast<double>(tall_cost) : 0.93 * static_cast<double>(low_cost);
    if (pass < single) m.zlen = m.tall ? high : low;
    const bool narrow = lx % 32 != 0 && lx <= 48;
    const double correction = (narrow ? 34.0 : lx % 4 == 0 ? 31.0 : 33.0) * mcells;
    if (mcells > 0.54 && 1.1 * static_cast<double>(tall_cost) + 8.0 * mcells < correction) m.refine_zlen = high;
    return m;
}

}  // namespace lbm

// Rules by which sums are split that bound scratch memory.  Plain C++, so that
// the host can check them.
#pragma once
#include <algorithm>
#include <cstddef>

namespace mv {

// Cuts of the branch part's runs of particles (fold_sum_kernel, kAmpShell).
// A block's run is a few h-bins, known on the device only and of very uneven
// length over the blocks (sorted by |k|); cut, the longest runs no longer hold
// the launch.  Every cut has partial sums and running sums of the whole
// lattice (bytes_a_cut), so a lattice takes as many cuts as fit 256 MB, at
// least one.  Large ones have thousands of blocks and lose by cuts: Wendland
// sets, ms of the branch part with 1, 2, 4 and 8 cuts
//   128^3, 262,144 particles  2.14  1.19  0.74  0.58   (0.03 GB a cut: 8)
//   160^3,  50,000            0.31  0.24  0.22  0.24   (0.05 GB: 4)
//   192^3, 100,000            0.60  0.52  0.53  0.57   (0.09 GB: 2)
//   256^3, 200,000            1.37  1.51  1.63  2.01   (0.2 GB: 1)
//   384^3,  60,000            1.87  2.17  2.97  4.31   (0.7 GB: 1)
constexpr double kMostBranchScratch = 256e6;

inline long long branch_cuts(long long most, size_t bytes_a_cut) {
    const long long fit = (long long)(kMostBranchScratch / (double)std::max<size_t>(1, bytes_a_cut));
    return std::max(1LL, std::min({8LL, most, fit}));
}

// Particles a split of a direct slice (mv_slice_sum.cu), in units of 64; more
// than a tile (4 units) in whole tiles.  The least of the blocks' work an SM
// (which 60% of its resident blocks keep busy), half a block's time for the last
// wave, a block's start (half a unit) and the splits' partial sums to write and
// reduce (0.005 units a block of them, 5 us a unit).
// A set of few tiles is so cut to fill the chip: 4096 particles on 64 x 64 took
// 43 us in 16 blocks of a tile, 5 in 64; 100,003 on 256 x 128 took 1.21 ms in
// one wave of 833 blocks of 8 tiles, whose SMs held 5 or 6.
// All splits together take 256 MB of scratch at most: every one has partial sums
// of the whole slice, and running sums where it has more than a tile.  Without
// radii, with a limit on the partial sums alone and so: 300,000 particles at a
// cutoff of 128 950 us (308 MB) and 895 (231), 1,000,003 at 256 10.9 ms (686 MB)
// and 11.6 (243), at 512 42.5 (642 MB) and 44.3 (214).
constexpr double kMostSliceScratch = 256e6;

inline int slice_chunk(int n, int tile, long long blocks, size_t partial_bytes, size_t sums_bytes, int resident,
                       int sm_count) {
    constexpr int kUnit = 64;
    const int tile_units = tile / kUnit;
    const double sms = sm_count;
    const long long units = std::max<long long>(1, ((long long)n + kUnit - 1) / kUnit);
    const long long most = (units + tile_units - 1) / tile_units * tile_units;  // one split
    long long chosen = most;
    double best_cost = 1e300;
    for (long long per = 1; per <= most;
         per += per < tile_units ? 1 : std::max<long long>(tile_units, per / 4 / tile_units * tile_units)) {
        const long long splits = (units + per - 1) / per;
        const double bytes = (double)splits * (double)(partial_bytes + (per > tile_units ? sums_bytes : 0));
        if (splits > 65535 || (splits > 1 && bytes > kMostSliceScratch)) continue;
        const double an_sm = (double)blocks * (double)splits / sms;
        const double cost = std::max(an_sm, 0.6 * resident) * ((double)per + 0.5) +
                            0.5 * (double)per * std::min<double>(resident, an_sm) + 0.005 * (double)(blocks * splits);
        if (cost < best_cost) {
            best_cost = cost;
            chosen = per;
        }
    }
    return (int)(chosen * kUnit);
}

}  // namespace mv

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

}  // namespace mv

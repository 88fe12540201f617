"""The splits that bound scratch memory (csrc/mv_split_rules.h): their own code,
compiled for the host."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "libmeshlessvis_b200" / "csrc"

CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include "mv_split_rules.h"

int main(int argc, char** argv) {
    for (int i = 1; i + 1 < argc; i += 2)
        std::printf("%lld\n", mv::branch_cuts(std::atoll(argv[i]), (size_t)std::atoll(argv[i + 1])));
    return 0;
}
"""


def _branch_bytes(g):
    """Partial sums (8 bytes an element) and running sums (64 a representative, in blocks of 256) of g^3."""
    blocks = -(-((g // 2 + 1) ** 3) // 256)
    return 8 * g * g * (g // 2 + 1) + 64 * 256 * blocks


@pytest.fixture(scope="module")
def branch_cuts(tmp_path_factory):
    d = tmp_path_factory.mktemp("split_rules")
    (d / "check.cpp").write_text(CHECK)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(d / "check.cpp"), "-o", str(d / "check")], check=True)

    def run(most, size):
        return int(subprocess.run([str(d / "check"), str(most), str(size)], check=True, capture_output=True, text=True).stdout)

    return run


@pytest.mark.parametrize("g", [16, 64, 96, 128, 160, 192, 256, 384, 544])
def test_branch_scratch_is_bounded(branch_cuts, g):
    size = _branch_bytes(g)
    cuts = branch_cuts(1000, size)
    assert 1 <= cuts <= 8
    assert cuts == 1 or cuts * size <= 256e6
    assert cuts == 8 or (cuts + 1) * size > 256e6  # no fewer than fit
    assert branch_cuts(3, size) == min(3, cuts) and branch_cuts(1, size) == 1


SLICE = r"""
#include <cstdio>
#include <cstdlib>
#include "mv_split_rules.h"

int main() {  // cutoff, particles, table form: bytes of scratch and splits
    int c, n, table;
    while (std::scanf("%d %d %d", &c, &n, &table) == 3) {
        const int g = (c + 3) / 4, warps = (2 * g * (g + 1) + 31) / 32;
        const long long blocks = table ? (warps + 3) / 4 : (long long)((c + 63) / 64) * ((c + 63) / 64);
        const size_t partial = (size_t)(2 * c - 1) * c * 8, sums = (size_t)blocks * (table ? 16 * 128 : 32 * 256) * 16;
        const int chunk = mv::slice_chunk(n, 256, blocks, partial, sums, table ? 6 : 2, 148);
        const long long splits = (n + (long long)chunk - 1) / chunk;
        std::printf("%d %lld %.0f\n", chunk, splits, (double)splits * (double)(partial + (chunk > 256 ? sums : 0)));
    }
    return 0;
}
"""


def test_slice_scratch_is_bounded(tmp_path):
    """Partial and running sums of all splits fit 256 MB wherever there is more
    than one; a split of more than a tile holds whole tiles."""
    (tmp_path / "check.cpp").write_text(SLICE)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", str(tmp_path / "check.cpp"), "-o", str(tmp_path / "check")],
                   check=True)
    cases = [(c, n, t) for c in (1, 32, 64, 65, 128, 256, 512, 2000) for t in (0, 1)
             for n in (1, 64, 257, 4096, 100003, 300000, 1 << 20, 1 << 24)]
    out = subprocess.run([str(tmp_path / "check")], input="\n".join("%d %d %d" % c for c in cases), check=True,
                         capture_output=True, text=True).stdout.splitlines()
    assert len(out) == len(cases)
    for (c, n, _), line in zip(cases, out):
        chunk, splits, size = (int(v) for v in line.split())
        assert chunk > 0 and splits * chunk >= n and splits <= 65535
        assert chunk < 256 and chunk % 64 == 0 or chunk % 256 == 0
        assert splits == 1 or size <= 256e6, (c, n, line)

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

"""The rows' order of the folded table sums (csrc/mv_row_order.h) is a
permutation on every lattice and step, whatever the compiler contracts: its own
code, compiled for the host with contraction allowed, and a row's place counted
in one piece as well as in the four parts of the device's lanes."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "libmeshlessvis_b200" / "csrc"

CHECK = r"""
#include <cstdio>
#include <vector>
#include "mv_row_order.h"

__attribute__((noinline)) int place(const mv::RowOrder& o, int y, int z) { return mv::rows_before(o, y, z, 0, 1); }

int main() {
    const double steps[] = {1.0, 0.5, 0.1, 0.1f, 0.3, 0.3f, 0.7, 1.0 / 3, (double)(float)(1.0 / 3), 1e-3, 37.7};
    const int shapes[][3] = {{1, 2, 0}, {9, 8, 0}, {10, 8, 0}, {18, 2, 0}, {33, 33, 0}, {46, 36, 0}, {39, 30, 1}, {65, 65, 0}};
    int wrong = 0;
    for (double ky : steps)
        for (double kz : {ky, 0.75 * ky, -ky})
            for (const int* s : shapes) {
                const mv::RowOrder o{nullptr, s[0], s[1], s[2], ky, kz, 0};
                std::vector<int> seen((size_t)s[0] * s[1], 0);
                for (int y = 0; y < s[0]; ++y)
                    for (int z = 0; z < s[1]; ++z) {
                        const int p = place(o, y, z);
                        int parts = 0;
                        for (int l = 0; l < 4; ++l) parts += mv::rows_before(o, y, z, l, 4);
                        if (p != parts || p < 0 || p >= (int)seen.size() || seen[p]++) ++wrong;
                    }
            }
    std::printf("%d\n", wrong);
    return 0;
}
"""


FMA = ["-mfma", "-ffp-contract=fast"] if " fma " in Path("/proc/cpuinfo").read_text() else []


@pytest.mark.parametrize("flags", [["-O0"], ["-O3", *FMA]])
def test_places_are_a_permutation(tmp_path, flags):
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", *flags, f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout) == 0


def test_small_sums_and_radii_take_the_rows_as_they_lie(tmp_path):
    """An order that costs more than it saves is not made; particles and table
    cells a step of k, on both sides of the line, and without a known radius."""
    src = tmp_path / "check.cpp"
    src.write_text('#include <cstdio>\n#include "mv_row_order.h"\nint main() {\n'
                   + "".join(f'std::printf("%d ", mv::rows_worth_sorting({n}, {c}));\n'
                             for n, c in ((62, 5.8), (62, 23.0), (4000, 1.2), (500, 5.8), (250, 23.0), (20011, 5.8),
                                          (1, 300.0), (62, -1.0)))
                   + "}\n")
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0", "0", "1", "1", "1", "1"]

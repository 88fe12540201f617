"""Division by a shared divisor (csrc/mv_divide.h) has the bits of the division
itself: its own code, compiled for the host, over mantissas, exponents, signs,
zeros, infinities and NaNs, for the colour map's divisors and ranges of images
from 1e-29 to 1e29."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "libmeshlessvis_b200" / "csrc"

CHECK = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#include "mv_divide.h"

static float number(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static bool same(float a, float b) { return a == b || (a != a && b != b); }

int main() {
    const float colour[] = {0.25f, 0.475f, 0.694f - 0.475f, 0.745f - 0.694f, 1.f - 0.745f,
                            std::log(0.011f) - std::log(1e-3f)};
    uint32_t seed = 1;
    auto random = [&seed] { return seed = seed * 1664525u + 1013904223u, seed >> 9; };
    long long wrong = 0;
    auto check = [&wrong](float x, float c) {
        for (float s : {x, -x}) wrong += !same(mv::divide_by(s, c, 1.f / c), s / c);
    };
    const float inf = std::numeric_limits<float>::infinity();
    auto divisor = [&](float c) {
        for (int e = -149; e <= 127; ++e)
            for (int i = 0; i < 2000; ++i) check(std::ldexp(number(0x3f800000u | random()), e), c);
        for (float x : {0.f, inf, std::numeric_limits<float>::quiet_NaN(), 1e-45f, 1e-38f, 3e38f}) check(x, c);
    };
    for (float c : colour) divisor(c);
    for (int e = -96; e <= 96; e += 4) divisor(std::ldexp(number(0x3f800000u | random()), e));
    for (float c : colour)  // every mantissa
        for (uint32_t m = 0; m < 1u << 23; ++m) check(number(0x3f800000u | m), c);
    std::printf("%lld\n", wrong);
    return 0;
}
"""


FMA = ["-mfma"] if " fma " in Path("/proc/cpuinfo").read_text() else []


@pytest.mark.parametrize("flags", [["-O2", *FMA]])
def test_quotients_have_the_divisions_bits(tmp_path, flags):
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", *flags, "-ffp-contract=off", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout) == 0

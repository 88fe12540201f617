"""Division by a shared divisor (csrc/mv_divide.h) has the bits of the division
itself where the colour map uses it: its own code, compiled for the host, for
ranges of images from 1e-29 to 1e29 and the map's own divisors after them, over
mantissas, exponents, infinities and NaNs."""
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
    const float colour[] = {0.25f, 0.475f, 0.694f - 0.475f, 0.745f - 0.694f, 1.f - 0.745f};
    uint32_t seed = 1;
    auto random = [&seed] { return seed = seed * 1664525u + 1013904223u, seed >> 9; };
    long long wrong = 0;
    auto check = [&wrong](float x, float c) { wrong += !same(mv::divide_by(x, c, 1.f / c), x / c); };
    auto weight = [&wrong](float x, float c) { wrong += !same(mv::divide_finite(x, c, 1.f / c), x / c); };
    const float inf = std::numeric_limits<float>::infinity(), log_range = std::log(0.011f) - std::log(1e-3f);
    for (int e = -96; e <= 96; ++e) {
        const float range = std::ldexp(number(0x3f800000u | random()), e), least = mv::divide_by_least(range);
        for (float x : {0.f, least, 3e38f, inf, std::numeric_limits<float>::quiet_NaN()}) check(x, range);
        for (int f = -149; f <= 127; ++f)
            for (int i = 0; i < 1000; ++i) {
                const float x = std::ldexp(number(0x3f800000u | random()), f);
                if (x < least) continue;
                check(x, range);
                const float a = x / range;
                if (a > 1.f) continue;
                for (float c : colour) weight(a, c);
            }
    }
    for (float c : colour)  // every mantissa
        for (uint32_t m = 0; m < 1u << 23; ++m) weight(number(0x3f800000u | m), c);
    for (uint32_t m = 0; m < 1u << 23; ++m)
        for (float x : {number(0x3f800000u | m), std::ldexp(number(0x3f800000u | m), -22)}) check(x, log_range);
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

"""The exact walk's term (csrc/bh_soft64.cuh) with r^2 formed as the walk forms
it, one square by soft::square, for components of every magnitude: the value is
IEEE's bit for bit, or the term is refused (and the walk takes the IEEE
operations)."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include "bh_soft64.cuh"
using namespace bh::soft;
static uint64_t state = 88172645463325252ull;
static uint64_t rnd()
{
    state ^= state << 13; state ^= state >> 7; state ^= state << 17;
    return state * 0x2545F4914F6CDD1Dull;
}
static long bad = 0, taken = 0;
static void check(double dx, double dy, double dz, double gm)
{
    const volatile double xx = dx * dx, yy = dy * dy, zz = dz * dz;
    const volatile double s = xx + yy;
    const volatile double r2 = s + zz;
    const volatile double walk = s + square(bits_of(dz));
    double t[3];
    if (!term(dx, dy, dz, walk, gm, t[0], t[1], t[2])) return;
    ++taken;
    const volatile double inv = 1.0 / std::sqrt((double)r2);
    const volatile double i2 = inv * inv;
    const volatile double i3 = i2 * inv;
    const volatile double sc = gm * i3;
    const double d[3] = {dx, dy, dz};
    for (int k = 0; k < 3; ++k) {
        const volatile double w = sc * d[k];
        if (w == 0 ? t[k] != 0 : bits_of((double)w) != bits_of(t[k])) {
            if (++bad < 5) std::printf("%a %a %a: %a, not %a\n", dx, dy, dz, t[k], (double)w);
        }
    }
}
static double value(int field) { return from_bits((uint64_t)field << 52 | (rnd() & 0xFFFFFFFFFFFFFull)); }
int main()
{
    // every exponent of a component, subnormal and non-finite ones too,
    // beside two of any size
    for (int field = 0; field < 2048; ++field)
        for (int k = 0; k < 200; ++k) {
            const int near = k & 1 ? 1023 + (int)(rnd() % 16) : (int)(rnd() % 2048);
            const double big = value(field), a = value(near), b = value(1023 - (int)(rnd() % 4));
            const double gm = value(1023 - (int)(rnd() % 60));
            check(a, b, k & 2 ? -big : big, gm);
            check(a, k & 2 ? -big : big, b, gm);
            check(k & 2 ? -big : big, b, a, gm);
        }
    check(3.1, 2.7, 2e154, 1.0);
    check(1.23, 2.35, HUGE_VAL, 1.0);
    check(1.23, 2.35, -HUGE_VAL, 1.0);
    check(1.23, 2.35, NAN, 1.0);
    std::printf("%ld %ld\n", bad, taken);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_components_of_every_magnitude(tmp_path):
    src, exe = tmp_path / "range.cpp", tmp_path / "range"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'barnes-hut_gb300' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    bad, taken = map(int, r.stdout.split())
    assert bad == 0 and taken > 10_000

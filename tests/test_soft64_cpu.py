"""The integer FP64 operations of the exact walk (csrc/bh_soft64.cuh) against
the host's IEEE arithmetic: correctly rounded, so equal bit for bit, over
random and adversarial significands, with the FP32 estimate they start from
moved to both ends of its error bound."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
static float nudge();
#define BH_SOFT_RSQRT(f) (1.0f / std::sqrt(f) * nudge())
#include "bh_soft64.cuh"
using namespace bh::soft;
// the estimate's bound, 2^-22, to either side and halfway
static float nudge()
{
    static unsigned k = 0;
    const float by[5] = {0.f, 2.38e-7f, -2.38e-7f, 1.2e-7f, -1.2e-7f};
    return 1.0f + by[k++ % 5];
}
static uint64_t state = 88172645463325252ull;
static uint64_t rnd()
{
    state ^= state << 13; state ^= state >> 7; state ^= state << 17;
    return state * 0x2545F4914F6CDD1Dull;
}
// A double of exponent e: random, all ones, a few high or low bits, near the
// ends of the binade, or a power of two.
static double value(int e)
{
    uint64_t m = rnd();
    switch (rnd() >> 60) {
    case 0: m = 0; break;
    case 1: m = ~0ull; break;
    case 2: m &= ~((1ull << (rnd() % 52)) - 1); break;
    case 3: m = rnd() & 0xF; break;
    case 4: m |= (1ull << 52) - 1 - (rnd() & 0x1F); break;
    }
    return from_bits(((uint64_t)(e + 1023) << 52) | (m & 0xFFFFFFFFFFFFFull));
}
static uint64_t packed(const Sig& s) { return (s.a >> 11) + ((uint64_t)(uint32_t)(s.e + 1022) << 52); }
int main()
{
    long bad = 0, odd = 0, taken = 0;
    for (long i = 0; i < 4000000; ++i) {
        const double x = value((int)(rnd() % 390) - 195);
        bool o = false;
        const Sig r = rcp_sqrt(unpack(bits_of(x)), o);
        const double root = std::sqrt(x), want = 1.0 / root;
        if (o) { ++odd; if ((bits_of(want) & 0xFFFFFFFFFFFFFull) != 0) ++bad; }
        else if (packed(r) != bits_of(want)) ++bad;
        const Sig a = unpack(bits_of(value((int)(rnd() % 100) - 50))), b = unpack(bits_of(value((int)(rnd() % 100) - 50)));
        if (low_zero(a) || low_zero(b)) continue;
        const volatile double p = from_bits(packed(a)) * from_bits(packed(b));
        if (mul_bits(a.a, b.a, a.e + b.e) != bits_of((double)p)) ++bad;
        o = false;
        const Sig q = mul(a, b, o);
        if (!o && packed(q) != bits_of((double)p)) ++bad;
    }
    for (long i = 0; i < 4000000; ++i) {
        double d[3];
        for (double& v : d) {
            v = value((int)(rnd() % 40) - 30);
            if (rnd() & 1) v = -v;
            if ((rnd() & 31) == 0) v = (rnd() & 1) ? 0.0 : -0.0;
        }
        const volatile double xx = d[0] * d[0], yy = d[1] * d[1], zz = d[2] * d[2];
        const volatile double s = xx + yy;
        const volatile double r2 = s + zz;
        const double gm = value(-(int)(rnd() % 100));
        double t[3];
        if (!low_zero(unpack(bits_of(d[2]))) && bits_of(square(bits_of(d[2]))) != bits_of((double)zz)) ++bad;
        if (!term(d[0], d[1], d[2], r2, gm, t[0], t[1], t[2])) continue;
        ++taken;
        const volatile double inv = 1.0 / std::sqrt((double)r2);
        const volatile double i2 = inv * inv;
        const volatile double i3 = i2 * inv;
        const volatile double sc = gm * i3;
        for (int k = 0; k < 3; ++k) {
            const volatile double w = sc * d[k];
            if (w == 0 ? t[k] != 0 : bits_of((double)w) != bits_of(t[k])) ++bad;
        }
    }
    // The list form's factor: within an ulp of the value in long double.
    long in = 0;
    for (long i = 0; i < 4000000; ++i) {
        double d[3], got;
        const int e = (int)(rnd() % 160) - 80;
        for (double& v : d) {
            v = value(e - (int)(rnd() % 20));
            if (rnd() & 1) v = -v;
            if ((rnd() & 31) == 0) v = 0.0;
            if ((rnd() & 31) == 0) v = value(e - 60 - (int)(rnd() % 60));
        }
        const double gm = value((int)(rnd() % 200) - 150);
        if (!scale(d[0], d[1], d[2], gm, got)) continue;
        ++in;
        const long double r2 = (long double)d[0] * d[0] + (long double)d[1] * d[1] + (long double)d[2] * d[2];
        const long double want = gm / (r2 * sqrtl(r2));
        // 0.53 ulp, and what the long double itself is off by where it has no
        // more than 53 bits (Arm's has 113, x86's 64)
        if (!(fabsl((long double)got - want) <= 0.55L * 0x1p-52L * want)) ++bad;
    }
    if (in < 1000000) ++bad;
    // Out of range: refused, not wrong.
    double t[3];
    const double out[][5] = {{1, 1, 1, 0x1p-250, 1}, {1, 1, 1, 0x1p+250, 1}, {1, 1, 1, 0.0, 1}, {1, 1, 1, 3, 0.0},
                             {1, 1, 1, 3, -1.0}, {1, 1, 1, 3, 0x1p-310}, {0x1p-320, 1, 1, 3, 1},
                             {1, 1, 1, HUGE_VAL, 1}, {1, 1, 1, 3, HUGE_VAL}, {1, 1, 1, NAN, 1}, {1, 1, 1, -1.0, 1}};
    for (auto& o : out)
        if (term(o[0], o[1], o[2], o[3], o[4], t[0], t[1], t[2])) ++bad;
    const double far[][4] = {{0, 0, 0, 1}, {0x1p-120, 0, 0, 1}, {0x1p+120, 1, 1, 1}, {1, HUGE_VAL, 0, 1},
                             {1, 1, NAN, 1}, {1, 1, 1, 0.0}, {1, 1, 1, -1.0}, {1, 1, 1, 0x1p-320}};
    for (auto& o : far)
        if (scale(o[0], o[1], o[2], o[3], t[0])) ++bad;
    std::printf("%ld %ld %ld\n", bad, odd, taken);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_soft64_rounds_as_ieee(tmp_path):
    src, exe = tmp_path / "soft.cpp", tmp_path / "soft"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'barnes-hut_gb300' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    bad, _, taken = map(int, r.stdout.split())
    assert bad == 0 and taken > 1_000_000

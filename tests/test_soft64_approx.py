"""The integer-pipe quotient and root (trans_gb300/csrc/soft64.cuh) with approximations of 1/x and 1/sqrt(x) that are off
by up to 2^-22 relative, upwards, downwards and either way, in place of the host's rounded ones: correctly
rounded all the same, which is what the digits' bias is for.  (The device's are documented at 1 ulp and
2^-22.9.)"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <math.h>
#include <stdint.h>
// the float farthest from the exact value e within 2^-22 relative, above or below, or one between them
static int side;                                       // 1 up, -1 down, 0 either way
static uint64_t st;
static uint64_t rnd() { st += 0x9e3779b97f4a7c15ull; uint64_t z = st; z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
                        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull; return z ^ (z >> 31); }
static float off(double e) {
    const double w = side ? side : (double)(int64_t)rnd() / 9223372036854775808.0, t = e * (1.0 + w * 0x1p-22);
    float f = (float)t;
    if (w > 0 && (double)f > t) f = nextafterf(f, 0.0f);
    if (w < 0 && (double)f < t) f = nextafterf(f, 4.0f);
    return f;
}
#define SX_HOST_RCP(x) off(1.0 / (double)(x))
#define SX_HOST_RSQRT(x) off(1.0 / sqrt((double)(x)))
#include "soft64.cuh"
#include <stdio.h>
#include <stdlib.h>
using sx::bits_of; using sx::of_bits; using sx::FRAC;
int main(int, char** v) {
    side = atoi(v[1]);
    const int kind = atoi(v[2]); const long n = atol(v[3]); st = 77 + kind; long bad = 0;
    const uint64_t known[] = {0x400f01d0de54aa1full};
    for (long i = 0; i < n; ++i) {
        uint64_t a = (rnd() & FRAC) | ((1003 + rnd() % 40) << 52), b = (rnd() & FRAC) | ((1003 + rnd() % 40) << 52);
        if (kind == 1) { a &= ~0xffffffffull; b &= ~0xfffffffffull; }                    // short significands
        if (kind == 2) { a = (a & ~FRAC) | (FRAC - (rnd() & 0xffff)); b = (b & ~FRAC) | (rnd() & 0xffff); }
        if (kind == 3) { b = (b & ~FRAC) | (FRAC - (rnd() & 0xffff)); a = (a & ~FRAC) | (rnd() & 0xffff); }
        if (kind == 4) { a |= (1ull << (rnd() % 52)) - 1; b |= (1ull << (rnd() % 52)) - 1; }   // runs of ones
        if (kind == 5) {                                                                 // roots just beside short ones
            const double r = of_bits((a & ~0x3fffffffull) | 0x3ff0000000000000ull);
            a = bits_of(r * r) + rnd() % 5 - 2;
        }
        if (i < 1) a = known[i];
        const double x = of_bits(a), y = of_bits(b);
        if (bits_of(sx::div(x, y)) != bits_of(x / y)) ++bad;
        if (bits_of(sx::sqrt(x)) != bits_of(::sqrt(x))) ++bad;
    }
    printf("%ld\n", bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("soft64_approx")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "trans_gb300", "csrc"), str(d / "h.cpp"),
                    "-o", str(d / "h")], check=True)
    return str(d / "h")


@pytest.mark.parametrize("side", [1, -1, 0], ids=["up", "down", "either"])
@pytest.mark.parametrize("kind", range(6))
def test_correctly_rounded_with_approximations(harness, kind, side):
    out = subprocess.run([harness, str(side), str(kind), "4000000"], capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "0"

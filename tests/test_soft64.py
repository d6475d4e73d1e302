"""The integer-pipe double division, square root and comparisons of the FP64 path (trans_gb300/csrc/soft64.cuh)
against IEEE arithmetic, compiled for the host: the correctly rounded result bit for bit over
every kind of operand pair where the digit recurrence or the rounding could go wrong.  (The
device forms are held to the hardware's by trans_check_conversions, tests/test_gpu_cvt.py.)"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include "soft64.cuh"
#include <stdio.h>
#include <stdlib.h>
using sx::bits_of; using sx::of_bits; using sx::FRAC;
static uint64_t st;
static uint64_t rnd() { st += 0x9e3779b97f4a7c15ull; uint64_t z = st; z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
                        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull; return z ^ (z >> 31); }
static int same(double a, double b) { return bits_of(a) == bits_of(b) || (a != a && b != b); }
int main(int, char** v) {
    const int kind = atoi(v[1]); const long n = atol(v[2]); st = kind + 1; long bad = 0;
    const uint64_t sp[] = {0, 1, FRAC, FRAC + 1, 0x7feull << 52 | FRAC, 0x7ffull << 52, 0x7ffull << 52 | 1, 1023ull << 52,
                           1022ull << 52 | FRAC, 1024ull << 52, 2ull << 52, 0x7fdull << 52, 1075ull << 52 | 1};
    for (long i = 0; i < n; ++i) {
        uint64_t a = rnd(), b = rnd();
        const uint64_t near_a = (a & (FRAC | 1ull << 63)) | ((1003 + (a >> 52) % 40) << 52);
        const uint64_t near_b = (b & (FRAC | 1ull << 63)) | ((1003 + (b >> 52) % 40) << 52);
        if (kind) { a = near_a; b = near_b; }
        if (kind == 2) { a &= ~0xffffffffull; b &= ~0xfffffffffull; }                   // short significands
        if (kind == 3) b = (b & ~FRAC) | ((a + rnd() % 5 - 2) & FRAC);                  // nearly equal ones
        if (kind == 4) { a = (a & ~FRAC) | (FRAC - (rnd() & 3)); b = (b & ~FRAC) | (rnd() & 3); }
        if (kind == 5) { b = (b & ~FRAC) | (FRAC - (rnd() & 3)); a = (a & ~FRAC) | (rnd() & 3); }
        if (kind == 6) {                                                                 // exact quotients and roots
            const double q = (double)(rnd() >> 38), d = (double)(1 + (rnd() >> 38)), r = (double)(rnd() >> 38);
            a = bits_of(q * d); b = bits_of(d);
            if (!same(sx::sqrt(r * r), r)) ++bad;
        }
        if (kind == 7) { a = sp[i % 13] | (rnd() << 63); b = sp[(i / 13) % 13] | (rnd() << 63); }   // limits, 0, inf, NaN
        if (kind == 8) { a = (a & ~(0x7ffull << 52)) | ((rnd() % 2047) << 52); b = (b & ~(0x7ffull << 52)) | (((a >> 52 & 2047) + 2047 - 1021 - rnd() % 8) % 2047 << 52); }
        const double x = of_bits(a), y = of_bits(b), z = fabs(x);
        if (!same(sx::div(x, y), x / y)) ++bad;
        if (!same(sx::sqrt(z), ::sqrt(z))) ++bad;
        const double w[3] = {y, x, -x};                                                  // comparisons
        for (double u : w)
            if (sx::less(x, u) != (x < u) || sx::less(u, x) != (u < x) || sx::less_equal(x, u) != (x <= u) ||
                sx::less_equal(u, x) != (u <= x) || sx::equal(x, u) != (x == u)) ++bad;
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
    d = tmp_path_factory.mktemp("soft64")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "trans_gb300", "csrc"), str(d / "h.cpp"),
                    "-o", str(d / "h")], check=True)
    return str(d / "h")


@pytest.mark.parametrize("kind", range(9))
def test_correctly_rounded(harness, kind):
    out = subprocess.run([harness, str(kind), "2000000"], capture_output=True, text=True, check=True)
    assert out.stdout.strip() == "0"

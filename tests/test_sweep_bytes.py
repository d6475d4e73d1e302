"""Which order the LU-SGS sweep arrays take (trans_gb300/csrc/sweep_bytes.h), compiled for the host: the bytes of
both orders from the blocks' sizes, and the rule between them at budgets and free memory around
their edges."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# argv: mixed ni nj nk free_percent_of_march left (-1: no budget) -> march planes chosen
HARNESS = r"""
#include "sweep_bytes.h"
#include <stdio.h>
#include <stdlib.h>
using namespace tg;
int main(int, char** v) {
    const int mixed = atoi(v[1]), ni = atoi(v[2]), nj = atoi(v[3]), nk = atoi(v[4]);
    const MarchBytes m = mixed ? march_block_bytes(ni, nj, nk, 8, 4, 20, 8, 4, 64, 44, 0, 2) : march_block_bytes(ni, nj, nk, 8, 4, 82, 8, 8, 112, 44, 8, 2);
    const size_t p = (size_t)ni * nj * nk * (mixed ? plane_cell_bytes(20, 3, 8, 4, 0) : plane_cell_bytes(160, 2, 8, 8, 0));
    const long long left = atoll(v[6]) < 0 ? -1 : atoll(v[6]);
    printf("%zu %zu %d\n", m.bytes, p, (int)march_fits(m.bytes, p, (size_t)(m.bytes / 100.0 * atof(v[5])), left));
    return 0;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("sweep_bytes")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-I", os.path.join(ROOT, "trans_gb300", "csrc"), str(d / "h.cpp"), "-o", str(d / "h")], check=True)

    def run(mixed, dims, free=1000.0, left=-1):
        out = subprocess.run([str(d / "h"), str(int(mixed)), *map(str, dims), str(free), str(left)], capture_output=True, text=True, check=True)
        m, p, chosen = map(int, out.stdout.split())
        return m, p, bool(chosen)
    return run


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("dims", [(3, 3, 3), (24, 16, 5), (96, 9, 5), (40, 8, 4), (41, 17, 9)])
def test_bytes(rule, mixed, dims):
    ni, nj, nk = dims
    tiles, steps = -(-nj // 8) * -(-nk // 4), ni + 10
    m, p, _ = rule(mixed, dims)
    if mixed:
        assert m == tiles * (steps * (32 * 28 * 4 + 12 * 64) + 44)
        assert p == ni * nj * nk * ((20 + 24) * 4 + 48)
    else:
        assert m == tiles * (steps * (32 * 90 * 8 + 12 * 112) + 44 + 8 * ((steps + 1) // 2))
        assert p == ni * nj * nk * ((160 + 16) * 8 + 48)


def test_the_smaller_order_near_the_memory_limit(rule):
    """A large FP64 block marches whatever is free (the other order needs 1.7 times as much); a block of few
    lines takes the hyperplane order when marching would take more than half of the free memory."""
    m, p, chosen = rule(0, (120, 64, 64), free=105)
    assert m < p / 1.6 and chosen
    m, p, chosen = rule(0, (400, 3, 3), free=199)
    assert m > p and not chosen
    assert rule(0, (400, 3, 3), free=201)[2]


@pytest.mark.parametrize("mixed", [0, 1])
def test_budget(rule, mixed):
    """What the marching arrays take beyond the charge has to fit the budget that is left."""
    for dims in [(24, 16, 5), (96, 9, 5), (3, 3, 3)]:
        m, p, chosen = rule(mixed, dims)
        assert m > p and chosen
        assert not rule(mixed, dims, left=0)[2]
        assert not rule(mixed, dims, left=m - p - 1)[2]
        assert rule(mixed, dims, left=m - p)[2]
    assert rule(mixed, (120, 64, 64), left=0)[2]

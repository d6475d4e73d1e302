"""Wall distance of points in any order (trans_wall_distance): a warp a point, points grouped by place, or
as they come, by their number and the surfaces' size.  The bits of the reference's sequential minimum over
every panel, at numbers around the edges of the three forms and for points that a grid groups badly; and
points in no order take no longer than points along lines."""
import ctypes as C
import time

import numpy as np
import pytest

from test_gpu_wall_chunks import DP, _brute, _panels, _surface

pytestmark = pytest.mark.gpu


def _args(pts, surfaces, out):
    nodes = np.ascontiguousarray(np.concatenate([S[..., m].ravel(order="F") for S in surfaces for m in range(3)]))
    dims = np.array([x for S in surfaces for x in S.shape[:2]], dtype=np.int32)
    keep = (pts, nodes, dims, out)
    return keep, (len(pts), pts.ctypes.data_as(DP), len(surfaces), dims.ctypes.data_as(C.POINTER(C.c_int)),
                  nodes.ctypes.data_as(DP), 1.0e-20, out.ctypes.data_as(DP))


def _points(kind, n, rng):
    if kind == "scattered":
        return rng.standard_normal((n, 3)) * 2.0
    if kind == "same":
        return np.tile([[0.4, 0.3, 0.2]], (n, 1))
    if kind == "plane":                                # no extent in one direction, clusters in another
        p = rng.standard_normal((n, 3)) * [1.0, 1.0e-6, 0.0]
        return p + [0.5, 0.5, 0.1]
    p = rng.uniform(-1.0, 1.0, (n, 3))                 # a few far points, most of them in one cell of a coarse grid
    p[:: max(1, n // 7)] *= 1.0e4
    return p


# 1, 8 and 16 chunks of panels: the largest numbers with a warp a point, one more, grouped
@pytest.mark.parametrize("kind", ["scattered", "same", "plane", "outliers"])
@pytest.mark.parametrize("n,dims", [(1, [(17, 33)]), (33, [(33, 33)]), (4096, [(9, 9)]), (4097, [(9, 9)]), (16385, [(17, 33)]),
                                    (32768, [(33, 33)]), (32769, [(33, 33)]), (37501, [(33, 33)]), (75001, [(9, 33), (2, 2), (33, 9)])])
def test_any_order(gpu_lib, n, dims, kind):
    rng = np.random.default_rng(11)
    surfaces = [_surface(ni, nj, rng, flat=q == 0) for q, (ni, nj) in enumerate(dims)]
    pts = np.ascontiguousarray(_points(kind, n, rng))
    pts[-1] = _panels(surfaces[0])[:, -1]              # a panel's centre
    out = np.zeros(n)
    keep, a = _args(pts, surfaces, out)
    assert gpu_lib.trans_wall_distance(*a) == 0
    assert np.array_equal(out, _brute(pts, surfaces, 1.0e-20))


def test_no_order_costs_no_more(gpu_lib):
    """200,000 points of a block over 25,600 panels, along its lines and shuffled: grouped, both are the same
    work but for the gathers (1.25: the spread of calls of a few milliseconds)."""
    rng = np.random.default_rng(5)
    surfaces = [_surface(161, 161, rng, flat=False)]
    g = np.stack(np.meshgrid(np.linspace(-1, 1.2, 100), np.linspace(0.1, 1.3, 50), np.linspace(0, 1.5, 40), indexing="ij"), axis=-1)
    lines = np.ascontiguousarray(g.transpose(2, 1, 0, 3).reshape(-1, 3))
    best = []
    for pts in (lines, np.ascontiguousarray(lines[rng.permutation(len(lines))])):
        keep, a = _args(pts, surfaces, np.zeros(len(pts)))
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            assert gpu_lib.trans_wall_distance(*a) == 0
            t.append(time.perf_counter() - t0)
        best.append(min(t))
    assert best[1] < 1.25 * best[0], best

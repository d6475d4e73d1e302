"""Wall distance with chunks of panels passed over (trans_wall_distance): the bits of the reference's
sequential minimum over every panel, at surface sizes around the chunks' 8 x 8, for points close
together and far apart, on a panel, equally far from many, and with a surface without panels."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DP = C.POINTER(C.c_double)


def _surface(ni, nj, rng, flat):
    u, v = np.meshgrid(np.linspace(0.0, 1.0, ni), np.linspace(0.0, 1.0, nj), indexing="ij")
    if flat:
        return np.stack([u, v, np.zeros_like(u)], axis=-1)
    return np.stack([np.cos(3.0 * u) + 0.01 * rng.standard_normal(u.shape), np.sin(3.0 * u), v + 0.3 * u], axis=-1)


def _panels(S):
    X = S.transpose(2, 0, 1)
    return ((X[:, :-1, :-1] + X[:, 1:, :-1] + X[:, :-1, 1:] + X[:, 1:, 1:]) / 4.0).reshape(3, -1)


def _brute(pts, surfaces, tiny):
    d = np.full(len(pts), 1.0e20)
    for S in surfaces:
        q, a = _panels(S), np.full(len(pts), 1.0e20)
        for k in range(q.shape[1]):
            dx, dy, dz = (pts[:, m] - q[m, k] for m in range(3))
            a = np.minimum(a, dx * dx + dy * dy + dz * dz)
        d = np.maximum(d, tiny)
        d = np.where(a < d, a, d)
    return np.sqrt(d)


@pytest.mark.parametrize("points", ["line", "scattered", "far"])
@pytest.mark.parametrize("dims", [[(2, 2)], [(9, 9)], [(10, 18), (8, 2)], [(1, 5), (33, 9)], [(41, 26), (17, 17), (2, 40)]])
def test_every_panel_counts(gpu_lib, dims, points):
    rng = np.random.default_rng(7)
    surfaces = [_surface(ni, nj, rng, flat=q == 0) for q, (ni, nj) in enumerate(dims)]
    n = 601                                            # a last warp that is partly empty
    if points == "line":
        pts = np.linspace([-0.2, 0.1, 0.01], [1.3, 0.8, 0.4], n)
    else:
        pts = rng.standard_normal((n, 3)) * (2.0 if points == "scattered" else 1.0e3)
    pts[5] = [0.5, 0.5, 10.0]                          # over the middle of the flat surface
    if _panels(surfaces[-1]).size:
        pts[7] = _panels(surfaces[-1])[:, 0]           # a panel's centre
    pts = np.ascontiguousarray(pts)
    nodes = np.ascontiguousarray(np.concatenate([S[..., m].ravel(order="F") for S in surfaces for m in range(3)]))
    d = np.array([x for ij in dims for x in ij], dtype=np.int32)
    out = np.zeros(n)
    assert gpu_lib.trans_wall_distance(n, pts.ctypes.data_as(DP), len(dims), d.ctypes.data_as(C.POINTER(C.c_int)),
                                       nodes.ctypes.data_as(DP), 1.0e-20, out.ctypes.data_as(DP)) == 0
    assert np.array_equal(out, _brute(pts, surfaces, 1.0e-20))

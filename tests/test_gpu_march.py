"""LU-SGS sweeps as marching warps (TRANS_SWEEP=march, 8 x 4 lines per tile), both precisions: every
DeltaQ has the bits of the hyperplane launches' (the same terms, summed in the same order), at
block sizes around the tile's edges, over several blocks, with the components the Runge-Kutta
path sweeps, and on repeated sweeps; a wait that runs out is reported."""
import ctypes as C

import pytest

from helpers import bit_equal_fraction, interior, small_cascade, small_channel

pytestmark = pytest.mark.gpu


def _states(make, mode, monkeypatch, iters, precision, **sw):
    from trans_gb300 import abi
    from trans_gb300.solver import Solver
    monkeypatch.setenv("TRANS_SWEEP", mode)
    c, conns, geo, st = make(Kind_Spatial=3, Kind_Roe=3, **sw)
    c.params.precision = precision
    s = Solver(c, conns, geo, st)
    for ki in range(1, iters + 1):
        s.iterate(ki)
    out = [s.get_field(ib, f) for ib in range(len(c.blocks)) for f in ("V", "D")]
    s.close()
    return c, out


# cells in j and k: one short of, at and past the tile's 8 x 4, several tiles, the smallest block;
# in i: shorter and longer than the shared-memory pipeline
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("ni,nj,nk", [(4, 4, 4), (12, 8, 4), (9, 9, 5), (25, 10, 6), (8, 17, 9), (41, 26, 14), (4, 33, 7)])
def test_march_equals_planes(gpu_lib, monkeypatch, ni, nj, nk, precision):
    def make(**sw):
        return small_channel(ni=ni, nj=nj, nk=nk, **sw)
    c, a = _states(make, "planes", monkeypatch, 3, precision)
    _, b = _states(make, "march", monkeypatch, 3, precision)
    m = interior(c.blocks[0].dims)
    for x, y in zip(a, b):
        assert bit_equal_fraction(x, y, m) == 1.0


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("rk", [0, 1])
def test_march_blocks_and_components(gpu_lib, monkeypatch, rk, precision):
    sw = dict(IF_RK=1, CFL_Sub_start=1.0, CFL_Sub_end=1.0) if rk else {}
    c, a = _states(small_cascade, "planes", monkeypatch, 5, precision, **sw)
    _, b = _states(small_cascade, "march", monkeypatch, 5, precision, **sw)
    for q, (x, y) in enumerate(zip(a, b)):
        assert bit_equal_fraction(x, y, interior(c.blocks[q // 2].dims)) == 1.0


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_march_wait_runs_out(gpu_lib, monkeypatch, precision):
    """No polls allowed: a tile whose neighbour has not arrived gives up and the host reports it;
    a context with the default limit then iterates."""
    from trans_gb300 import abi
    from trans_gb300.solver import Solver
    monkeypatch.setenv("TRANS_SWEEP", "march")
    monkeypatch.setenv("TRANS_SWEEP_SPIN", "0")
    c, conns, geo, st = small_channel(ni=41, nj=26, nk=14, Kind_Spatial=3, Kind_Roe=3)
    c.params.precision = precision
    s = Solver(c, conns, geo, st)
    for name in ("SPECRAD", "BC_STATE", "GRADIENT", "BC_GRAD", "RESIDUAL", "LUSGS"):
        s.run_stage(name, 1)
    assert s.lib.trans_run_stage(s.ctx, abi.STAGE_ID["UPDATE"], 1, 1) == abi.TRANS_E_TIMEOUT
    assert s.lib.trans_update_static_scratch(s.ctx, 1, C.cast(None, C.POINTER(abi.TransNorms))) == abi.TRANS_E_TIMEOUT
    s.close()
    monkeypatch.delenv("TRANS_SWEEP_SPIN")
    s = Solver(c, conns, geo, st)
    for ki in (1, 2):
        assert all(n["nan_flag"] == 0 and n["DRSa"] > 0 for n in s.iterate(ki))
    s.close()

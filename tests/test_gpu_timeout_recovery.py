"""A context whose sweep waits ran out goes on: the report of one time-out does not reach the graph
replays that follow in the same context, and their results are those of a context that never had
one.  (The waits are bounded; no kernel here faults or spins without a limit.)"""
import pytest

from helpers import bit_equal_fraction, interior, small_channel

pytestmark = pytest.mark.gpu
STATE = ("V", "PP", "T", "RMIU", "WT0", "WT1")


def _make(precision):
    c, conns, geo, st = small_channel(ni=41, nj=26, nk=14, Kind_Spatial=3, Kind_Roe=3)      # 16 tiles of 8 x 4 lines
    c.params.precision = precision
    return c, conns, geo, st


def _upload(s, c, st):
    for q, b in enumerate(c.blocks):
        for f in STATE:
            s.set_field(q, f, st[b.id][f])


@pytest.mark.parametrize("report", ["update", "static_scratch", "none"])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_context_goes_on_after_a_timeout(gpu_lib, monkeypatch, precision, report):
    from trans_gb300 import abi
    from trans_gb300.solver import Solver
    monkeypatch.delenv("TRANS_SWEEP", raising=False)
    args = _make(precision)
    c, conns, geo, st = args
    s = Solver(*args)
    for ki in range(1, 11):
        s.iterate(ki)
    want = s.get_field(0, "V")
    s.close()

    monkeypatch.setenv("TRANS_SWEEP_SPIN", "0")
    s = Solver(*args)
    assert b"march" in s.lib.trans_tuning(s.ctx)
    for name in ("SPECRAD", "BC_STATE", "GRADIENT", "BC_GRAD", "RESIDUAL", "LUSGS"):
        s.run_stage(name, 1)
    if report == "update":
        assert s.lib.trans_run_stage(s.ctx, abi.STAGE_ID["UPDATE"], 1, 1) == abi.TRANS_E_TIMEOUT
    if report == "static_scratch":
        assert s.lib.trans_update_static_scratch(s.ctx, 1, None) == abi.TRANS_E_TIMEOUT
    monkeypatch.delenv("TRANS_SWEEP_SPIN")          # read again when the iterations are captured
    _upload(s, c, st)
    s.iterate(1)
    ms = abi.C.c_double()
    assert s.lib.trans_time_iterations(s.ctx, 2, 9, ms, None) == 0, s.lib.trans_last_error(s.ctx)
    got = s.get_field(0, "V")
    assert bit_equal_fraction(got, want, interior(c.blocks[0].dims)) == 1.0

    # a replay that times out reports it once
    s.close()
    monkeypatch.setenv("TRANS_SWEEP_SPIN", "0")
    s = Solver(*args)
    nb = len(c.blocks)
    norms = (abi.TransNorms * nb)()
    assert s.lib.trans_iterate(s.ctx, 1, norms) == abi.TRANS_E_TIMEOUT       # launched directly
    assert s.lib.trans_iterate(s.ctx, 1, norms) == abi.TRANS_E_TIMEOUT       # replayed
    s.close()

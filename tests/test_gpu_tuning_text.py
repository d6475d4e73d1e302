"""trans_tuning names the schedule, and measurements only where the tuner made some; and the checks of the
integer-pipe conversions, quotients and roots report no count on a correct build."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sw,measured", [(dict(), False), (dict(IF_Precondition=1, XM=0.3), True)], ids=["march", "tuned"])
def test_measured_only_where_tuned(gpu_lib, monkeypatch, sw, measured):
    from helpers import small_channel
    from trans_gb300.solver import Solver
    monkeypatch.delenv("TRANS_SWEEP", raising=False)
    s = Solver(*small_channel(ni=9, nj=9, nk=5, Kind_Spatial=2, Kind_Roe=1, **sw))
    s.iterate(1)
    text = s.lib.trans_tuning(s.ctx).decode()
    s.close()
    assert ("measured" in text) == measured
    assert measured or text == "sweep=march"


def test_no_counts_on_a_correct_build(gpu_lib):
    from trans_gb300 import abi
    bad = (C.c_longlong * 2)()
    assert gpu_lib.trans_check_conversions(0, 1, bad) == abi.TRANS_E_ARG       # leaves a message
    assert gpu_lib.trans_check_conversions(1 << 20, 3, bad) == 0
    assert list(bad) == [0, 0] and b"mismatches of" not in gpu_lib.trans_last_error(None)

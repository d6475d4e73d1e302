"""Preconditioned FP64 sweeps: the lanes of the density and the energy form PrecondDW together.  With
eight lanes a position (planes) and with a warp per component (planes/wpc) a sweep then issues the
same FP64 instructions a position on its longest path, so the two launches take the same time to a
few per cent; one after the other, the lane-major launch took 1.7 times as long."""
import re

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,nk", [(25, 17, 6), (97, 49, 9)])
def test_lane_major_sweeps_keep_their_lanes_together(gpu_lib, monkeypatch, ni, nj, nk):
    from helpers import small_channel
    from trans_gb300.solver import Solver
    monkeypatch.delenv("TRANS_SWEEP", raising=False)
    c, conns, geo, st = small_channel(ni=ni, nj=nj, nk=nk, Kind_Spatial=2, Kind_Roe=1, IF_Precondition=1, XM=0.3)
    s = Solver(c, conns, geo, st)
    s.iterate(1)                                       # times the schedules
    ms = {}
    for name, t in re.findall(r"(\S+):([0-9.]+)ms", s.lib.trans_tuning(s.ctx).decode()):
        ms[name] = float(t)
    s.close()
    lane = min(v for k, v in ms.items() if re.match(r"planes(-\w+)?(/pf\d)?$", k))
    comp = min(v for k, v in ms.items() if re.match(r"planes(-\w+)?/wpc(/pf\d)?$", k))
    assert lane < 1.3 * comp, (lane, comp)

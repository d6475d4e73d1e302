"""The terms that faces of the FP64 path share (k_face_terms) against the kernels that form them face
by face, which a context takes when its budget leaves no room for the terms: the same bits (the same
operations on the same operands) for every reconstruction and flux scheme, over several blocks and on
the smallest one, in whole iterations, and stage by stage with the state changed in between."""
import numpy as np
import pytest

from helpers import bit_equal_fraction, interior, small_cascade, small_channel

pytestmark = pytest.mark.gpu


def _thin(**sw):
    return small_channel(ni=5, nj=4, nk=4, **sw)


def _batch(make, room, **sw):
    from trans_gb300.solver import Batch
    c, conns, geo, st = make(**sw)
    probe = Batch()
    need = probe.case_bytes(c, conns)
    probe.close()
    bt = Batch(budget_bytes=0 if room else need)
    return c, bt, bt.add(c, conns, geo, st)


@pytest.mark.parametrize("make", [small_cascade, small_channel, _thin])
@pytest.mark.parametrize("spatial,roe", [(1, 1), (2, 3), (3, 1), (3, 3), (4, 2)])
def test_terms_equal_face_by_face(gpu_lib, make, spatial, roe):
    out = []
    for room in (True, False):
        c, bt, cid = _batch(make, room, Kind_Spatial=spatial, Kind_Roe=roe)
        bt.iterate(3)
        out.append([bt.get_field(cid, ib, f) for ib in range(len(c.blocks)) for f in ("V", "D", "RMIU")])
        bt.close()
    for q, (x, y) in enumerate(zip(*out)):
        assert bit_equal_fraction(x, y, interior(c.blocks[q // 3].dims)) == 1.0


@pytest.mark.parametrize("spatial", [2, 3])
def test_state_changed_between_stages(gpu_lib, spatial):
    from trans_gb300 import abi
    out = []
    for room in (True, False):
        c, bt, cid = _batch(small_cascade, room, Kind_Spatial=spatial, Kind_Roe=3)
        bt.iterate(1)
        for stage in ("SPECRAD", "BC_STATE", "GRADIENT", "BC_GRAD"):
            assert gpu_lib.trans_run_stage(bt.ctx, abi.STAGE_ID[stage], 2, 1) == 0
        for ib in range(len(c.blocks)):
            for f in ("T", "PP"):
                a = bt.get_field(cid, ib, f)
                bt.set_field(cid, ib, f, a * (1.0 + 1.0e-3 * np.cos(np.arange(a.size)).reshape(a.shape)))
        assert gpu_lib.trans_run_stage(bt.ctx, abi.STAGE_ID["RESIDUAL"], 2, 1) == 0
        out.append([bt.get_field(cid, ib, "D") for ib in range(len(c.blocks))])
        bt.close()
    for ib, (x, y) in enumerate(zip(*out)):
        assert bit_equal_fraction(x, y, interior(c.blocks[ib].dims)) == 1.0

"""Whole iterations against the same iterations stage by stage, where each stage forms again what an
iteration takes from the stage before (the terms that faces share): the same bits with and without
turbulence, in a rotating frame, over several blocks, in both precisions."""
import pytest

from helpers import bit_equal_fraction, interior, small_cascade, small_channel

pytestmark = pytest.mark.gpu


def _annulus(**sw):
    from trans_gb300 import case as CS
    from trans_gb300 import cases
    c = cases.annular_sector(ni=14, nj=10, nk=6, rpm=2000.0, casing_kindsub=1, **sw)
    conns, geo = CS.compute_geometry(c)
    return c, conns, geo, CS.initial_state(c, geo, Q_dst=c.meta["Q_dst"])


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("make,sw", [(small_cascade, {}), (_annulus, {}), (small_channel, dict(IF_Turb_org=0)),
                                     (_annulus, dict(IF_RK=1, CFL_Sub_start=1.0, CFL_Sub_end=1.0))],
                         ids=["cascade", "rotating", "laminar", "runge_kutta"])
def test_iteration_equals_stages(gpu_lib, precision, make, sw):
    from trans_gb300 import abi
    from trans_gb300.solver import Solver
    out = []
    for whole in (True, False):
        c, conns, geo, st = make(Kind_Spatial=3, Kind_Roe=1, **sw)
        c.params.precision = precision
        s = Solver(c, conns, geo, st)
        for ki in (1, 2):
            if whole:
                s.iterate(ki)
                continue
            nsub = 3 if sw.get("IF_RK") else 1
            for it in range(1, nsub + 1):
                for stage in abi.STAGES[:-1]:
                    assert s.lib.trans_run_stage(s.ctx, abi.STAGE_ID[stage], ki, it) == 0, stage
            assert s.lib.trans_run_stage(s.ctx, abi.STAGE_ID["UPDATE_U"], ki, nsub) == 0
        out.append([s.get_field(ib, f) for ib in range(len(c.blocks)) for f in ("V", "D", "RMIU")])
        s.close()
    for q, (x, y) in enumerate(zip(*out)):
        assert bit_equal_fraction(x, y, interior(c.blocks[q // 3].dims)) == 1.0

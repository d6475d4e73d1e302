"""A batch context's device budget with the marching sweeps and the face fluxes' shared terms: what they hold
beyond the cases' charges is within the budget and in trans_batch_bytes_in_use; where it does not fit, the
sweeps keep the hyperplane order (with its tuner) and the fluxes form the terms themselves, with the same
bits; and it gives way to the next case."""
import numpy as np
import pytest

from helpers import bit_equal_fraction, interior, small_cascade, small_channel

pytestmark = pytest.mark.gpu


def _run(case, precision, budget, iters):
    from trans_gb300.solver import Batch
    bt = Batch(precision, budget_bytes=budget)
    cid = bt.add(*case)
    assert cid is not None
    bt.iterate(iters)
    out = (bt.get_field(cid, 0, "V"), bt.bytes_in_use(), bt.lib.trans_tuning(bt.ctx).decode(), bt.case_bytes(case[0], case[1]))
    bt.close()
    return out


# 24 x 16 x 5 and 40 x 9 x 5 cells: tiles of 8 x 4 lines that the lines fill to 62% and 35%
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("dims", [(25, 17, 6), (41, 10, 6)])
def test_budget_without_room(gpu_lib, monkeypatch, precision, dims):
    monkeypatch.delenv("TRANS_SWEEP", raising=False)
    case = small_channel(*dims, Kind_Spatial=3, Kind_Roe=3)
    case[0].params.precision = precision
    v, used, tuning, need = _run(case, precision, 0, 12)
    assert tuning.startswith("sweep=march") and used > need
    w, used, tuning, _ = _run(case, precision, need, 12)
    assert used == need and not tuning.startswith("sweep=march")
    assert bit_equal_fraction(v, w, interior(case[0].blocks[0].dims)) == 1.0


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_bytes_in_use_cover_what_is_held(gpu_lib, monkeypatch, precision):
    """8,000 x 3 x 3 cells, whose marching arrays are 1.9 (FP64) and 2.2 times what is charged for them: the device
    memory that the context took, less the transfer buffer and the tables of one entry a cell or tile
    (64 MB), is no more than it says."""
    import torch
    from trans_gb300.solver import Batch
    monkeypatch.delenv("TRANS_SWEEP", raising=False)
    case = small_channel(8001, 4, 4, Kind_Spatial=2, Kind_Roe=1)
    case[0].params.precision = precision
    warm = Batch(precision)                            # the library's own allocations
    warm.add(*small_channel(5, 5, 5, Kind_Spatial=2, Kind_Roe=1, precision=precision))
    warm.iterate(2)
    warm.close()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    bt = Batch(precision)
    assert bt.add(*case) is not None
    need = bt.bytes_in_use()
    bt.iterate(2)
    held = free0 - torch.cuda.mem_get_info()[0]
    used = bt.bytes_in_use()
    assert bt.lib.trans_tuning(bt.ctx).startswith(b"sweep=march") and used > need
    stage = 18 * 8 * 8005 * 8 * 8
    assert held <= used + stage + (64 << 20), (held, used, need)
    assert bt.lib.trans_device_bytes(bt.ctx) <= held
    bt.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_next_case_takes_the_room(gpu_lib, monkeypatch, precision):
    """The budget of two cases: the first alone holds more than its charge, the second is still admitted, and
    both go on with the bits of unlimited contexts."""
    from trans_gb300.solver import Batch
    monkeypatch.delenv("TRANS_SWEEP", raising=False)

    def make(which):
        case = small_cascade(Kind_Spatial=3, Kind_Roe=3) if which else small_channel(Kind_Spatial=3, Kind_Roe=3)
        case[0].params.precision = precision
        return case
    probe = Batch(precision)
    need = [probe.case_bytes(*make(w)[:2]) for w in (0, 1)]
    probe.close()
    fields = {}
    for budget in (0, sum(need)):
        bt = Batch(precision, budget_bytes=budget)
        a = bt.add(*make(0))
        bt.iterate(3)
        assert bt.bytes_in_use() > need[0] and (not budget or bt.bytes_in_use() <= budget)
        b = bt.add(*make(1))
        assert b is not None and (not budget or bt.bytes_in_use() <= budget)
        bt.iterate(9)
        assert not budget or bt.bytes_in_use() <= budget
        fields[budget] = [bt.get_field(a, 0, "V")] + [bt.get_field(b, q, "V") for q in range(len(make(1)[0].blocks))]
        bt.remove(b)
        assert bt.bytes_in_use() == need[0]
        bt.iterate(2)
        assert np.isfinite(bt.norms(a)[2][0]["DRSa"])
        bt.close()
    dims = [make(0)[0].blocks[0].dims] + [b.dims for b in make(1)[0].blocks]
    for x, y, d in zip(fields[0], fields[sum(need)], dims):
        assert bit_equal_fraction(x, y, interior(d)) == 1.0

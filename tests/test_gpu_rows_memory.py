"""What channels over packed rows keep on the device: refused and failed calls leave nothing behind."""
import numpy as np
import pytest

from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the suite's bound between FP64 evaluations
OOM, ARG = 2, 8


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("runs", [1, 7])
def test_a_refused_schedule_builds_no_tensor(gpu_lib, runs):
    """Below 8 runs no run-minor contraction: refused before the moments (864 bytes a tuple) are built."""
    mats, states = W.ensemble_runs(runs, seed=4, Ns=(32,))
    f = np.concatenate(states)
    e = E.BatchEngine(mats)
    try:
        ref, free = e.rhs(f), _free()
        for width in (4, 8, 16, 32):
            with pytest.raises(E.TortoiseError) as ex:
                e.set_schedule(0, 1, runs=width)
            assert ex.value.rc == ARG
        assert _free() == free and e.schedule(0).get("inside_only")
        assert rel_l2(e.rhs(f), ref) < TOL
    finally:
        e.close()


def test_a_tensor_without_room_is_reported_once(gpu_lib):
    """No room for the moments: TB_ERR_OOM, the rows stay, and the next call does not report it again."""
    import torch
    mats, states = W.ensemble_runs(1, seed=4, Ns=(40,))
    e = E.BatchEngine(mats)
    hog = None
    try:
        ref = e.rhs(states[0])
        torch.cuda.empty_cache()
        hog = torch.empty(_free() - (64 << 20), dtype=torch.uint8, device="cuda")
        with pytest.raises(E.TortoiseError) as ex:
            e.set_schedule(0, 1, pair=0)
        assert ex.value.rc == OOM
        assert e.schedule(0).get("inside_only") and rel_l2(e.rhs(states[0]), ref) < TOL
        del hog
        torch.cuda.empty_cache()
        e.set_schedule(0, 1, pair=0)
        assert not e.schedule(0).get("inside_only") and rel_l2(e.rhs(states[0]), ref) < TOL
    finally:
        hog = None
        torch.cuda.empty_cache()
        e.close()


def _used(mat, cap):
    """Device memory of a handle, and the bytes of rows that its channels would fill without any padding."""
    import torch
    before = _free()
    e = E.Engine(mat, tensor_budget_bytes=cap)
    try:
        f = W.initial_status(mat, kT=0.15, seed=7).vec
        rows = [max(e.points_inside(c)[0], 0) * 172 for c in range(len(mat.channels))]
        assert all(e.schedule(c).get("inside_only") for c, n in enumerate(rows) if n)   # every channel has its list
        return before - _free(), rows, e.rhs(f)
    finally:
        e.close()
        torch.cuda.empty_cache()


def test_rows_of_all_channels_stay_within_the_budget(gpu_lib):
    mat = W.build_material(7, ("P", "D"), (), ee=True, eph=False)   # four-leg channels only
    _used(mat, 0)   # what the first handle of a process allocates once
    small, rows, ref = _used(mat, 1)
    full, _, got = _used(mat, 0)
    assert len([n for n in rows if n]) > 1 and full - small > 0.9 * sum(rows) > 64 << 20
    assert rel_l2(got, ref) < TOL
    cap = int(1.1 * max(rows)) + (4 << 20)
    assert cap < 0.7 * sum(rows)
    part, _, got = _used(mat, cap)
    assert 0 < part - small <= cap + (4 << 20)   # and the row sets and further accumulators, in units of 2 MB
    assert rel_l2(got, ref) < TOL


def test_changing_factors_again_and_again_keeps_nothing(gpu_lib):
    """Each change of a channel's factors rebuilds the row sets; what they held before is given back."""
    mats, states = W.ensemble_runs(1, seed=4, Ns=(16,))
    e = E.BatchEngine(mats)
    try:
        def change(k):
            e.set_channel_amplitude(0, lambda b: np.full(len(b), 1.0 + 0.01 * k))
        for k in range(3):
            change(k)
        free = _free()
        for k in range(200):
            change(k)
        assert free - _free() <= 2 << 20   # one unit of the allocator; kept sets would take 10 MB
    finally:
        e.close()

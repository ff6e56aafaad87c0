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

"""The bounded wait for staged rows at limits where some lanes, warps or rows run out and others do not: a call either
reports TB_ERR_TIMEOUT or gives its normal result, and ends.  (Limit 0, where all lanes fail together: test_gpu_rows.py,
test_gpu_timeout.py.)"""
import os
import re

import numpy as np
import pytest

from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

TIMEOUT = 6
ROWS = os.path.join(os.path.dirname(__file__), "..", "tortoise_b200", "csrc", "tb_rows.cu")


def test_a_wait_that_may_end_a_loop_is_decided_for_the_whole_warp():
    """Every wait whose outcome is branched on goes through a warp vote; the others only bound what is in flight."""
    src = open(ROWS).read()
    waits = re.findall(r"if \(([^\n]*)mbar_wait\(", src)
    assert len(waits) == 2 and all("__all_sync(0xffffffffu, " in w for w in waits)


@pytest.mark.gpu
@pytest.mark.parametrize("runs", [1, 3, 8])
def test_small_wait_limits_end_with_a_status_or_the_result(gpu_lib, runs):
    mats, states = W.ensemble_runs(runs, seed=9, Ns=(12,))
    f = np.concatenate(states)
    be = E.BatchEngine(mats)
    try:
        ref = be.rhs(f), be.scattering_rates(f), be.rhs_vjp(f, f)[0]
        for polls in (1, 2, 3, 5, 8, 13, 21, 34, 55, 1 << 22):
            be.set_copy_wait_limit(polls)
            for call, want in zip((be.rhs, be.scattering_rates, lambda x: be.rhs_vjp(x, x)[0]), ref):
                try:
                    got = call(f)
                except E.TortoiseError as ex:
                    assert ex.rc == TIMEOUT and polls < 1 << 22
                else:
                    assert rel_l2(got, want) < 1e-13
    finally:
        be.close()

"""The deterministic mode over packed rows (AUTO channels), where creation, the number of runs or a non-finite value
could change what a call returns."""
import numpy as np
import pytest

from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the suite's bound between FP64 layouts


def _runs(n, Ns=(4,)):
    mats, states = W.ensemble_runs(n, seed=3, Ns=Ns)
    return mats, np.concatenate(states)


@pytest.mark.parametrize("runs", [1, 3])
@pytest.mark.parametrize("call", ["rhs", "scattering_rates", "vjp"])
def test_autotuned_handle_starts_from_empty_sums(gpu_lib, runs, call):
    """The first call of a handle whose creation timed the rows equals an untuned handle's."""
    mats, f = _runs(runs)
    got = []
    for tune in (False, True):
        e = E.BatchEngine(mats, deterministic=True, autotune=tune)
        try:
            got.append(e.rhs_vjp(f, f)[0] if call == "vjp" else getattr(e, call)(f))
        finally:
            e.close()
    assert rel_l2(got[1], got[0]) < TOL

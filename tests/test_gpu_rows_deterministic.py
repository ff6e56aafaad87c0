"""The deterministic mode over packed rows (AUTO channels), where creation, the number of runs or a non-finite value
could change what a call returns."""
import numpy as np
import pytest

import oracle
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


@pytest.mark.parametrize("runs", [2, 15, 16, 40])
def test_a_run_has_the_same_bits_alone_and_in_a_batch(gpu_lib, runs):
    """AUTO's arithmetic depends neither on the number of runs nor on what autotune timed."""
    mats, f = _runs(runs, Ns=(4, 5))
    th = np.random.default_rng(5).standard_normal(f.size)

    def calls(e, f, th):
        d = e.dp45(f, 0.0, 0.1, 0.05)
        return e.rhs(f), e.scattering_rates(f), e.rhs_vjp(f, th)[0], d["y"]

    be = E.BatchEngine(mats, deterministic=True)
    tuned = E.BatchEngine(mats, deterministic=True, autotune=True)
    try:
        got = calls(be, f, th)
        for a, b in zip(got, calls(tuned, f, th)):
            assert np.array_equal(a, b)
        for r in (0, 1, runs - 1):
            s = be.slices[r]
            for tune in (False, True):
                one = E.Engine(mats[r], deterministic=True, autotune=tune)
                try:
                    for a, b in zip(got, calls(one, f[s], th[s])):
                        assert np.array_equal(a[s], b)
                finally:
                    one.close()
            assert rel_l2(got[0][s], oracle.Oracle(mats[r]).rhs(f[s])) < TOL
    finally:
        be.close()
        tuned.close()


@pytest.mark.parametrize("where", ["state", "co-state"])
def test_vjp_non_finite_values_reach_tuples_without_a_point_inside(gpu_lib, where):
    """A non-finite coefficient of an element that is in no tuple with a point inside: the moments' contraction
    multiplies its tuples' zero moments by it, and a poisoned exact sum reads NaN everywhere."""
    mat = W.build_material(5, ("P", "D"), (0.2,), ee=False, eph=True, n_mc=1)
    f = W.initial_status(mat, seed=2).vec
    th = np.random.default_rng(3).standard_normal(f.size)
    rows, tensor = E.Engine(mat, deterministic=True), E.Engine(mat, layout=E.LAYOUT_T64, deterministic=True)
    try:
        assert any(rows.schedule(c).get("inside_only") for c in range(len(mat.channels)))
        some = 0
        for k in range(1, f.size, 3):
            a, b = f.copy(), th.copy()
            (a if where == "state" else b)[k] = np.nan
            got, ref = rows.rhs_vjp(a, b), tensor.rhs_vjp(a, b)
            for x, y in zip(got, ref):
                assert np.array_equal(np.isnan(x), np.isnan(y)), k
            some += np.isnan(ref[0]).all()
        assert some
        assert np.isfinite(rows.rhs_vjp(f, th)[0]).all()   # the poison is gone
    finally:
        rows.close()
        tensor.close()

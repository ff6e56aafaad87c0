"""Non-finite states and co-states over four-leg rows against the list kernel (a handle whose budget leaves no room for
rows): four-leg channels visit the tuples with a point inside only, so these alone carry a non-finite value, to every
leg of the operator and the transpose but the derivative with respect to the leg's own coefficient."""
import numpy as np
import pytest

from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W
from tortoise_b200.model import IN, OUT

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the suite's bound between FP64 evaluations


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("names", [["el:P"] * 4, ["el:P", "pn:0", "el:P", "pn:0"]])
def test_four_legs_spread_non_finite_values_like_the_list(gpu_lib, names, value):
    mat = W.build_material(5, ("P", "D"), (0.2,), ee=False, eph=False, mesh_nsplit=(5, 4))
    for c in mat.addScatteringChannelsWildcards(names, [IN, IN, OUT, OUT], 0):
        c.amplitude = 1.0
    f = W.initial_status(mat, kT=0.15, seed=5).vec
    th = np.random.default_rng(3).standard_normal(f.size)
    rows, lists = E.Engine(mat), E.Engine(mat, tensor_budget_bytes=1)
    try:
        touched = 0
        for k in (0, 5, f.size // 2, f.size - 1):
            g, b = f.copy(), th.copy()
            g[k] = b[k] = value
            for call in (lambda e: e.rhs(g), lambda e: e.scattering_rates(g), lambda e: e.rhs_vjp(f, b)[0],
                         lambda e: e.rhs_vjp(g, th)[0], lambda e: e.rhs_vjp(f, b)[1]):
                got, ref = call(rows), call(lists)
                ok = np.isfinite(ref)
                assert np.array_equal(np.isfinite(got), ok), k
                assert not ok.any() or rel_l2(got[ok], ref[ok]) < TOL
                touched += not ok.all()
        assert touched
    finally:
        rows.close()
        lists.close()

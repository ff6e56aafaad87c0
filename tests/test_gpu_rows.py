"""The packed-row evaluation of the collision operator (tb_rows.cu) against the oracle: the shapes where its dispatch, padding and sharing change.

Tolerance: 1e-12 relative L2, the bound of every FP64 layout of this suite (the
summation noise of a few thousand FP64 terms per coefficient is about 1e-14)."""
import numpy as np
import pytest

import oracle
from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W
from tortoise_b200.model import FERMION, IN, OUT

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _material(names, dirs, nsplit=(6, 5), umklapp=0, n_mc=50, bands=("P", "D"), crossing=False, amp=1.0):
    mat = W.build_material(max(nsplit), bands, (0.2,), ee=False, eph=False, field=(0.1, 0.0), rtol=1e-6, atol=1e-9,
                           n_mc=n_mc, mesh_nsplit=nsplit)
    if crossing:   # a tilted plane that crosses the parabola: two-leg channels with tuples
        b = mat.addBand("el:X", -1.0, FERMION, mat.bands[0].mesh, lambda kx, ky: 0.6 * kx + 0.3 * ky + 0.2)
        b.relativeErrorTolerance, b.absoluteErrorTolerance = 1e-6, 1e-9
    for c in mat.addScatteringChannelsWildcards(names, dirs, umklapp):
        c.amplitude = amp
    return mat


SHAPES = {
    "in_in_out": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT]),
    "in_out_out": dict(names=["el:*", "el:*", "pn:*"], dirs=[IN, OUT, OUT]),
    "out_in_out": dict(names=["pn:*", "el:*", "el:*"], dirs=[OUT, IN, OUT]),
    "two_legs": dict(names=["el:*", "el:*"], dirs=[IN, OUT], crossing=True, nsplit=(9, 7)),
    "umklapp": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], umklapp=1, nsplit=(5, 3)),
    "one_row_meshes": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], nsplit=(7, 1)),
    "one_point": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], n_mc=1),
    "64_points": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], n_mc=64, nsplit=(8, 8)),
    "65_points": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], n_mc=65),   # beyond the mask: the tensor
    "four_legs": dict(names=["el:P"] * 4, dirs=[IN, IN, OUT, OUT], nsplit=(5, 4)),   # one accumulator a block
    "four_legs_bosons": dict(names=["el:P", "pn:0", "el:P", "pn:0"], dirs=[IN, IN, OUT, OUT], nsplit=(3, 3)),
    "four_legs_64_points": dict(names=["el:P"] * 4, dirs=[IN, IN, OUT, OUT], nsplit=(3, 2), n_mc=64),
    "many_rows": dict(names=["el:*", "pn:*", "el:*"], dirs=[IN, IN, OUT], nsplit=(20, 17)),
}


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_rhs_and_rates_match_the_oracle(gpu_lib, shape, deterministic):
    mat = _material(**SHAPES[shape])
    f = W.initial_status(mat, kT=0.15, seed=5).vec
    o = oracle.Oracle(mat)
    e = E.Engine(mat, deterministic=deterministic)
    live = [c for c in range(len(mat.channels)) if o.num_tuples(c)]
    try:
        assert live
        for c in live:   # without any point inside there are no rows
            rows = shape != "65_points" and o.points_inside(c)[1] > 0
            assert bool(e.schedule(c).get("inside_only")) == rows
        assert rel_l2(e.rhs(f), o.rhs(f)) < TOL
        assert rel_l2(e.scattering_rates(f), o.scattering_rates(f)) < TOL
        for c in live:
            if np.linalg.norm(o.channel_propagate(c, f)) > 0:
                assert rel_l2(e.channel_propagate(c, f), o.channel_propagate(c, f)) < TOL
            for leg in range(mat.channels[c].nlegs):
                r = o.scattering_rates(f, c, leg)
                if np.linalg.norm(r) > 0:
                    assert rel_l2(e.scattering_rates(f, c, leg), r) < TOL
        th = np.random.default_rng(3).standard_normal(f.size)
        v = np.random.default_rng(4).standard_normal(f.size)
        g, _ = e.rhs_vjp(f, th)
        jv = (o.rhs(f + 1e-5 * v) - o.rhs(f - 1e-5 * v)) / 2e-5
        assert abs(th @ jv - g @ v) <= 1e-8 * (abs(th @ jv) + 1e-6 * np.linalg.norm(th) * np.linalg.norm(jv))
    finally:
        e.close()


@pytest.mark.parametrize("shape,runs", [("in_in_out", 2), ("in_in_out", 7), ("in_in_out", 8), ("in_out_out", 9),
                                        ("in_in_out", 16), ("two_legs", 17), ("in_in_out", 33),
                                        ("four_legs_64_points", 5), ("four_legs_64_points", 9)])
def test_shared_rows_of_a_batch(gpu_lib, shape, runs):
    """One run after another below 8 runs, run-minor in groups of 8, 16 and 32 from there; beside them a run on
    another mesh."""
    kw = SHAPES[shape]
    mats = [_material(amp=0.5 + 0.01 * r, **kw) for r in range(runs)] + [_material(**dict(kw, nsplit=(4, 5)))]
    states = [W.initial_status(m, kT=0.05 + 0.005 * r, seed=r).vec for r, m in enumerate(mats)]
    be = E.BatchEngine(mats)
    try:
        off = min(1, len(mats[0].channels) - 1)
        be.set_amplitude(off, 0.0)   # a channel of the first run switched off
        mats[0].channels[off].amplitude = 0.0
        refs = [oracle.Oracle(m) for m in mats]
        f = np.concatenate(states)
        for call in ("rhs", "scattering_rates", "rhs"):   # twice: what one evaluation leaves behind
            for o, x, g in zip(refs, states, be.split(getattr(be, call)(f))):
                assert rel_l2(g, getattr(o, call)(x)) < TOL
        k = be.slices[runs - 1].start + 5   # a non-finite coefficient stays in its own run
        f[k] = np.nan
        bad = np.isfinite(be.rhs(f))
        f[k] = 0.25
        assert bad[:be.slices[runs - 1].start].all() and bad[be.slices[runs].start:].all() and not bad.all()
        assert np.isfinite(be.rhs(f)).all()
        if runs == 16:   # every run's integration, while others have ended
            tf = np.linspace(0.05, 0.2, runs + 1)
            got = be.dp45(np.concatenate(states), 0.0, tf, 0.05)
            for m, x, g, t in zip(mats, states, got["runs"], tf):
                one = E.Engine(m)
                r = one.dp45(x, 0.0, t, 0.05)
                one.close()
                assert g["attempts"] == r["attempts"] and (len(r["dense"]) == 0 or rel_l2(g["dense"], r["dense"]) < 1e-11)
    finally:
        be.close()


@pytest.mark.parametrize("runs", [7, 9, 47, 48, 65])
def test_three_and_four_legs_of_a_batch_choose_by_themselves(gpu_lib, runs):
    """Three legs go run-minor from 8 runs, four legs (small channels) from 48: none, one and both kinds."""
    def make(r):
        m = _material(amp=0.5 + 0.01 * r, **dict(SHAPES["in_in_out"], nsplit=(3, 2)))
        for c in m.addScatteringChannelsWildcards(["el:P"] * 4, [IN, IN, OUT, OUT], 0):
            c.amplitude = 0.3 + 0.01 * r
        return m
    mats = [make(r) for r in range(runs)]
    states = [W.initial_status(m, kT=0.05 + 0.005 * r, seed=r).vec for r, m in enumerate(mats)]
    be = E.BatchEngine(mats)
    try:
        f = np.concatenate(states)
        for call in ("rhs", "scattering_rates", "rhs"):
            for m, x, g in zip(mats, states, be.split(getattr(be, call)(f))):
                assert rel_l2(g, getattr(oracle.Oracle(m), call)(x)) < TOL
    finally:
        be.close()


def test_amplitude_factors_and_pinned_schedules(gpu_lib):
    """functAmplitude through the rows; then a contraction schedule, whose tensor is built on request, and back."""
    mat = _material(**SHAPES["in_in_out"])
    fn = lambda b: 1.0 + 0.3 * b[:, 0, 0] - 0.2 * b[:, 1, 1]  # noqa: E731
    for c in mat.channels:
        c.functAmplitude = fn
    f = W.initial_status(mat, seed=2).vec
    ref = oracle.Oracle(mat).rhs(f)
    e = E.Engine(mat)
    try:
        assert rel_l2(e.rhs(f), ref) < TOL
        for c in range(len(mat.channels)):
            e.set_schedule(c, 1, pair=0)
            assert e.schedule(c)["stages"] == 1
        assert rel_l2(e.rhs(f), ref) < TOL
        for c in range(len(mat.channels)):
            e.set_schedule(c, 0, inside_only=True)
        assert rel_l2(e.rhs(f), ref) < TOL
        with pytest.raises(E.TortoiseError):
            e.set_schedule(0, 0, inside_only=False)
        for c in range(len(mat.channels)):
            e.set_channel_amplitude(c, None)
            mat.channels[c].functAmplitude = None
        assert rel_l2(e.rhs(f), oracle.Oracle(mat).rhs(f)) < TOL
    finally:
        e.close()


@pytest.mark.parametrize("shape", ["in_in_out", "in_out_out", "out_in_out", "two_legs", "umklapp", "four_legs",
                                   "four_legs_bosons", "64_points"])
def test_vjp_equals_the_tensor_and_the_list(gpu_lib, shape):
    """grad_f and the amplitude gradients against the moment tensor's transpose, and (one instance or several, one
    channel switched off) against the exact sums over the list."""
    mats = [_material(amp=0.7 + 0.2 * r, **SHAPES[shape]) for r in range(3)]
    fs = [W.initial_status(m, kT=0.1 + 0.05 * r, seed=r).vec for r, m in enumerate(mats)]
    rng = np.random.default_rng(8)
    ths = [rng.standard_normal(f.size) for f in fs]
    rows, tensor = E.Engine(mats[0]), E.Engine(mats[0], layout=E.LAYOUT_T64)
    batch, listed = E.BatchEngine(mats), E.BatchEngine(mats, layout=E.LAYOUT_MC64, deterministic=True)
    try:
        ref = tensor.rhs_vjp(fs[0], ths[0])
        for got in (rows.rhs_vjp(fs[0], ths[0]), rows.rhs_vjp(fs[0], ths[0])):
            assert rel_l2(got[0], ref[0]) < TOL and rel_l2(got[1], ref[1]) < TOL
        for e in (batch, listed):
            e.set_amplitude(0, 0.0)
        a, b = (e.rhs_vjp(np.concatenate(fs), np.concatenate(ths)) for e in (batch, listed))
        assert rel_l2(a[0], b[0]) < TOL and rel_l2(a[1], b[1]) < TOL
        th = ths[0].copy()
        th[3] = np.nan
        got, ref = rows.rhs_vjp(fs[0], th), tensor.rhs_vjp(fs[0], th)
        assert np.array_equal(np.isfinite(got[0]), np.isfinite(ref[0])) or mats[0].channels[0].nlegs == 4
        assert np.array_equal(np.isfinite(got[1]), np.isfinite(ref[1]))
    finally:
        for e in (rows, tensor, batch, listed):
            e.close()


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_coefficients_reach_the_same_elements_as_the_tensor(gpu_lib, value):
    """Also through tuples without a point inside, whose integrand the full quadrature multiplies by 0."""
    mat = _material(**SHAPES["in_in_out"])
    f = W.initial_status(mat, seed=2).vec
    rows, tensor = E.Engine(mat), E.Engine(mat, layout=E.LAYOUT_T64)
    try:
        for k in (4, f.size // 2, f.size - 1):
            g = f.copy()
            g[k] = value
            for call in ("rhs", "scattering_rates"):
                a, b = getattr(rows, call)(g), getattr(tensor, call)(g)
                assert np.array_equal(np.isfinite(a), np.isfinite(b)), (k, call)
                ok = np.isfinite(b)
                assert rel_l2(a[ok], b[ok]) < TOL
    finally:
        rows.close()
        tensor.close()


def test_row_wait_runs_out_and_the_handle_recovers(gpu_lib):
    """The bounded wait for staged rows (see test_gpu_timeout.py)."""
    mat = _material(**SHAPES["in_in_out"])
    f = W.initial_status(mat, seed=2).vec
    e = E.Engine(mat, deterministic=True)
    try:
        ref = e.rhs(f)
        e.set_copy_wait_limit(0)
        with pytest.raises(E.TortoiseError) as ex:
            e.rhs(f)
        assert ex.value.rc == 6
        e.set_copy_wait_limit(1 << 22)
        assert np.array_equal(e.rhs(f), ref)
    finally:
        e.close()

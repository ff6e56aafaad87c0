"""The two passes of the tuple enumeration (tb_enumerate.cu) against the oracle's lists, tuple by tuple: the walk,
and what sends a channel to the pass that evaluates every candidate."""
import numpy as np
import pytest

import oracle
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W
from tortoise_b200.model import BOSON, FERMION, IN, OUT, Material, Mesh, Region

pytestmark = pytest.mark.gpu


def _eph(n_mc=50, nsplit=(6, 5), umklapp=0):
    mat = W.build_material(max(nsplit), ("P", "D"), (0.2,), ee=False, eph=True, n_mc=n_mc, mesh_nsplit=nsplit)
    for c in mat.channels:
        c.findUmklappVectors(umklapp)
    return mat


def _outside_points():
    """A survival table with points outside the reference triangle, which the walk's domain test does not cover."""
    mat = _eph()
    for c in mat.channels:
        c.mc_points_precalc = c.mc_points_precalc * np.array([1.3, 1.4, 1.0]) - np.array([0.2, 0.1, 0.0])
    return mat


def _threshold(t):
    mat = W.parabolic_ee(4, mesh_nsplit=(4, 3))
    for c in mat.channels:
        c.scattElemeThreshold = t
    return mat


def _fine_last_leg():
    """The last leg on a mesh so much finer than the others' that its boxes hold more than 64 candidates."""
    region = Region((-1.0, -1.0), ((2.0, 0.0), (0.0, 2.0)))
    coarse, fine = Mesh(region, (0.0, 0.0), (1.0, 1.0), (3, 3)), Mesh(region, (0.0, 0.0), (1.0, 1.0), (11, 12))
    mat = Material("mixed", region)
    mat.addBand("el:A", -1.0, FERMION, coarse, W.DISPERSIONS["P"])
    mat.addBand("pn:0", 0.0, BOSON, coarse, 0.2)
    mat.addBand("el:B", -1.0, FERMION, fine, W.DISPERSIONS["P"])
    mat.addScatteringChannel(["el:A", "pn:0", "el:B"], [IN, IN, OUT])
    mat.addScatteringChannel(["el:B", "pn:0", "el:A"], [IN, IN, OUT])
    return mat


CASES = {
    "walk": _eph,
    "one_section_wide": lambda: _eph(nsplit=(17, 1)),
    "many_items": lambda: _eph(nsplit=(19, 23)),
    "umklapp": lambda: _eph(nsplit=(5, 4), umklapp=1),
    "64_points": lambda: _eph(n_mc=64),
    "65_points": lambda: _eph(n_mc=65),
    "outside_points": _outside_points,
    "fine_last_leg": _fine_last_leg,
    "four_legs": lambda: W.parabolic_ee(5, mesh_nsplit=(5, 4)),
    "one_point": lambda: _eph(n_mc=1),
    "33_points": lambda: _eph(n_mc=33),
    "high_threshold": lambda: _threshold(2e-6),    # more than one point inside needed
    "negative_threshold": lambda: _threshold(-1.0),   # none needed
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tuples_equal_the_oracle(gpu_lib, name):
    mat = CASES[name]()
    o, e = oracle.Oracle(mat), E.Engine(mat)
    try:
        total = 0
        for ch in range(len(mat.channels)):
            (ids, umk), (ref, ref_umk) = e.tuples(ch), o.tuples(ch)
            assert np.array_equal(ids, ref) and np.array_equal(umk, ref_umk)
            info = e.channel_info(ch)
            assert [info["n_prefilter"], info["n_det"]] == list(o.enum_counts(ch))
            total += len(umk)
        assert total > 0
    finally:
        e.close()


@pytest.mark.parametrize("name", ["walk", "one_point", "33_points", "64_points", "four_legs", "high_threshold",
                                  "negative_threshold"])
def test_streamed_walk_equals_the_stored_list(gpu_lib, name):
    """The streamed operator takes the same decisions: the same bits in the deterministic mode."""
    mat = CASES[name]()
    f = W.initial_status(mat, kT=0.15, seed=6).vec
    stored = E.Engine(mat, layout=E.LAYOUT_MC64, deterministic=True)
    streamed = E.Engine(mat, deterministic=True, stream_legs=2)
    try:
        assert np.array_equal(stored.rhs(f), streamed.rhs(f))
        for ch in range(len(mat.channels)):
            assert streamed.channel_info(ch)["n_tuples"] == stored.channel_info(ch)["n_tuples"]
            if stored.channel_info(ch)["n_tuples"]:
                assert streamed.points_inside(ch) == stored.points_inside(ch)
    finally:
        stored.close()
        streamed.close()

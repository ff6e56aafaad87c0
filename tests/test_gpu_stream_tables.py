"""Streamed channels whose point tables leave the integration domain (free legs' points far outside the reference
triangle): the FP32 pass of the walk has to allow for the size of the coordinates."""
import numpy as np
import pytest

from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.5, 3.0, 40.0])
@pytest.mark.parametrize("legs", [3, 4])
def test_streamed_channels_take_points_far_outside(gpu_lib, legs, scale):
    mat = (W.parabolic_ee(6, mesh_nsplit=(6, 5)) if legs == 4 else
           W.build_material(14, ("P", "D"), (0.2,), ee=False, eph=True, mesh_nsplit=(14, 12)))
    for c in mat.channels:
        for name in ("mc_points", "mc_points_precalc"):
            q = np.array(getattr(c, name))
            q[:, :2 * (legs - 2)] = scale * (q[:, :2 * (legs - 2)] - 0.4)
            setattr(c, name, q)
    f = W.initial_status(mat, kT=0.15, seed=6).vec
    stored = E.Engine(mat, layout=E.LAYOUT_MC64, deterministic=True)
    streamed = E.Engine(mat, deterministic=True, stream_legs=2)
    try:
        a, b = stored.rhs(f, drift=False), streamed.rhs(f, drift=False)
        assert scale > 3 or np.linalg.norm(a) > 0
        assert sum(stored.channel_info(ch)["n_tuples"] for ch in range(len(mat.channels))) > 0
        for ch in range(len(mat.channels)):
            n = stored.channel_info(ch)["n_tuples"]
            assert streamed.channel_info(ch)["n_tuples"] == n
            assert stored.points_inside(ch)[0] < 0 or streamed.points_inside(ch) == stored.points_inside(ch)
        assert np.array_equal(a, b)
    finally:
        stored.close()
        streamed.close()

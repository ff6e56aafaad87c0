"""Operator calls with device pointers under the caller's own stream capture, replayed beside and after other calls of
the handle."""
import numpy as np
import pytest

from conftest import rel_l2
from tortoise_b200 import engine as E
from tortoise_b200 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the suite's bound between FP64 evaluations


class Captured:
    """A graph of one call on the handle's stream, from one device buffer to another."""

    def __init__(self, eng, call, n):
        import torch
        self.x = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.y = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.stream = torch.cuda.ExternalStream(E.lib().tb_get_stream(eng.h))
        self.graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(self.stream):
            self.graph.capture_begin()
            call(self.x.data_ptr(), self.y.data_ptr())
            self.graph.capture_end()

    def __call__(self, f):
        import torch
        self.x.copy_(torch.from_numpy(f))
        torch.cuda.synchronize()
        with torch.cuda.stream(self.stream):
            self.graph.replay()
        torch.cuda.synchronize()
        return self.y.cpu().numpy()


def _material():
    return W.build_material(6, ("P", "D"), (0.2,), ee=True, eph=True, field=(0.1, 0.0), rtol=1e-6, atol=1e-9)


def _calls(e):
    """The captured calls (none of them made before) and the same calls as the test makes them."""
    import ctypes as C
    lib = E.lib()

    def check(rc):
        assert rc == 0, lib.tb_last_error()
    p = C.c_void_p
    return [(lambda x, y: check(lib.tb_rhs(e.h, p(x), p(y), 0)), e.rhs),
            (lambda x, y: check(lib.tb_channel_propagate(e.h, 0, p(x), p(y), 0)), lambda f: e.channel_propagate(0, f)),
            (lambda x, y: check(lib.tb_channel_propagate(e.h, 4, p(x), p(y), 0)), lambda f: e.channel_propagate(4, f)),
            (lambda x, y: check(lib.tb_scattering_rates(e.h, -1, -1, p(x), p(y), 0)), e.scattering_rates),
            (lambda x, y: check(lib.tb_scattering_rates(e.h, 1, 0, p(x), p(y), 0)),
             lambda f: e.scattering_rates(f, 1, 0))]


@pytest.mark.parametrize("deterministic", [False, True])
def test_captured_calls_replay_beside_other_calls(gpu_lib, deterministic):
    mat = _material()
    f = W.initial_status(mat, seed=1).vec
    e, ref = E.Engine(mat, deterministic=deterministic), E.Engine(mat, deterministic=deterministic)
    try:
        e.dp45(f, 0.0, 0.05, 0.05)   # leaves the accumulator to be cleared by the next call
        graphs = [Captured(e, call, f.size) for call, _ in _calls(e)]
        assert rel_l2(e.rhs(f), ref.rhs(f)) < TOL   # captured calls have not run
        for k in (1.0, 0.5):
            for g, (_, call) in zip(graphs, _calls(ref)):
                want = call(k * f)
                assert np.linalg.norm(want) > 0 and rel_l2(g(k * f), want) < TOL
            e.dp45(f, 0.0, 0.05, 0.05)
            e.rhs_vjp(f, f)
        assert rel_l2(e.rhs(f), ref.rhs(f)) < TOL
    finally:
        e.close()
        ref.close()


def test_captured_calls_outlive_a_change_of_schedules(gpu_lib):
    """The row sets that a graph launches stay, although the handle's own calls use others after the change."""
    mat = _material()
    f = W.initial_status(mat, seed=1).vec
    e, ref = E.Engine(mat), E.Engine(mat)
    try:
        graphs = [Captured(e, call, f.size) for call, _ in _calls(e)]
        want = [call(f) for _, call in _calls(ref)]
        legs = [c.nlegs for c in mat.channels]
        three, four = legs.index(3), legs.index(4)
        assert e.schedule(three).get("inside_only") and e.schedule(four).get("inside_only")
        for ch, kw in ((three, {"pair": 0}), (four, {"inside_only": False}), (three, {"inside_only": True})):
            e.set_schedule(ch, 0 if "inside_only" in kw else 1, **kw)
            for (_, call), w, g in zip(_calls(e), want, graphs):
                assert rel_l2(call(f), w) < TOL and rel_l2(g(f), w) < TOL
    finally:
        e.close()
        ref.close()

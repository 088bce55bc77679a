"""Calls that share a context's buffers stay in order whatever their streams
and however they were launched: eager calls after graph replays."""
import numpy as np
import pytest

from helpers import smooth_model, surface_receivers

pytestmark = pytest.mark.gpu

NX, NZ = 150, 90
SHOTS = [(120.0, 0.0), (700.0, 30.0, 10, 120), (1250.0, 80.0)]


def engine(m, arith="reference"):
    from seisfat2d_gb300 import Engine
    e = Engine(NX, NZ, 10.0, 10.0)
    e.set_arithmetic(arith)
    e.set_slowness(m)
    return e


def models():
    return (smooth_model(NX, NZ, 10.0, seed=3, noise=0.02),
            smooth_model(NX, NZ, 10.0, seed=4, vmin=1000.0, vmax=5000.0, noise=0.02))


# the first launches of a context are a graph's: the eager calls after them
# must not take the handoff pairs and progress words the replay left
@pytest.mark.parametrize("arith", ["reference", "compensated"])
@pytest.mark.parametrize("captured", [False, True])
def test_eager_calls_after_a_replay(engine_lib, cuda, arith, captured):
    a, b = models()
    rx, rz = surface_receivers(NX, 10.0, step=3)
    want = engine(b, arith).batch_forward(SHOTS, rx, rz, keep_tape=True)
    e = engine(a, arith)
    e.plan_batch(SHOTS, rx, rz)
    t_obs = cuda.zeros(want.shape, device="cuda")
    picks, grad = cuda.empty_like(t_obs), cuda.empty((e.nxx, e.nzz), device="cuda")
    if captured:
        g, st = cuda.cuda.CUDAGraph(), cuda.cuda.Stream()
        with cuda.cuda.graph(g, stream=st):
            e.plan_iteration(picks, t_obs, grad, stream=st)
        g.replay()
    else:
        e.plan_graph_launch(picks, t_obs, grad)
    cuda.cuda.synchronize()
    e.set_slowness(b)
    for _ in range(3):
        got = e.batch_forward(SHOTS, rx, rz, keep_tape=True)
        assert np.array_equal(got, want, equal_nan=True)
        _, g1 = e.misfit_gradient(np.zeros_like(want))
    e2 = engine(b, arith)
    e2.batch_forward(SHOTS, rx, rz, keep_tape=True)
    assert np.array_equal(g1, e2.misfit_gradient(np.zeros_like(want))[1])

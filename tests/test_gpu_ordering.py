"""Calls that share a context's buffers stay in order whatever their streams
and however they were launched: eager calls after graph replays, streams that
do not wait for the default one."""
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


# a padded device slowness is set while its stream is busy (some 50 ms); the
# calls after it, on a stream that does not wait for that one, use it all the
# same. The second model has values outside the fast updates' range.
@pytest.mark.parametrize("call", ["batch", "table", "plan", "graph", "captured", "autotune", "update", "image"])
def test_slowness_reaches_other_streams(engine_lib, cuda, call):
    a, b = models()
    b[40:60, 30:50] *= 1e-6
    rx, rz = surface_receivers(NX, 10.0, step=3)
    e, ref = engine(a), engine(b)
    pad = lambda m: cuda.from_numpy(np.pad(m, 3, mode="edge")).cuda()
    S = {0: pad(a), 1: pad(b)}
    st = cuda.cuda.Stream()
    t_obs = cuda.zeros((len(SHOTS), len(rx)), device="cuda")
    picks, grad = cuda.empty_like(t_obs), cuda.empty((e.nxx, e.nzz), device="cuda")
    want = cuda.from_numpy(ref.batch_forward(SHOTS, rx, rz)).cuda()
    T = cuda.empty((e.nxx, e.nzz), device="cuda")
    if call in ("plan", "graph", "captured", "autotune"):
        e.plan_batch(SHOTS, rx, rz)
    if call == "captured":
        g = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(g, stream=st):
            e.plan_iteration(picks, t_obs, grad, stream=st)
    if call == "table":
        want = cuda.from_numpy(ref.time_propagation(*SHOTS[0])).cuda()
    if call == "update":
        grad.copy_(cuda.linspace(0.0, 1.0, grad.numel(), device="cuda").view_as(grad))
        ref.update_slowness(grad, 1e-5)
        want = cuda.from_numpy(ref.get_slowness()).cuda()
    if call == "image":
        e.time_propagation(*SHOTS[0], out=T)
        args = (T[None], T[None], np.array([120.0]), np.array([300.0]), cuda.ones((1, 1, 400), device="cuda"), 0.004, 40.0, 1e4)
        want = ref.kirchhoff_image(*args, out=cuda.empty((NX, NZ), device="cuda"))
    cuda.cuda.synchronize()
    for _ in range(3):
        e.set_slowness(S[0], padded=True)
        cuda.cuda.synchronize()
        cuda.cuda._sleep(100_000_000)
        e.set_slowness(S[1], padded=True)
        with cuda.cuda.stream(st):
            if call == "batch":
                got = e.batch_forward(SHOTS, rx, rz, out=picks, stream=st)
            elif call == "table":
                got = e.time_propagation(*SHOTS[0], out=T, stream=st)
            elif call in ("plan", "graph"):
                (e.plan_iteration if call == "plan" else e.plan_graph_launch)(picks, t_obs, grad, stream=st)
                got = picks
            elif call == "captured":
                g.replay()
                got = picks
            elif call == "autotune":
                e.plan_autotune(picks, t_obs, grad, reps=1, stream=st)
                got = picks
            elif call == "update":
                e.update_slowness(grad, 1e-5, stream=st)
                got = cuda.from_numpy(e.get_slowness()).cuda()
            else:
                got = e.kirchhoff_image(*args, out=cuda.empty((NX, NZ), device="cuda"), stream=st)
            st.synchronize()
        assert np.array_equal(got.cpu().numpy(), want.cpu().numpy(), equal_nan=True)


def test_autograd_on_a_side_stream(engine_lib, cuda):
    """The slowness is made on a busy side stream, on which the wrapper runs."""
    from seisfat2d_gb300.autograd import EikonalPicks
    a, b = models()
    rx, rz = surface_receivers(NX, 10.0, step=3)
    want = engine(b).batch_forward(SHOTS, rx, rz)
    e = engine(a)
    S, new = (cuda.from_numpy(np.pad(m, 3, mode="edge")).cuda() for m in (a, b))
    st = cuda.cuda.Stream()
    cuda.cuda.synchronize()
    with cuda.cuda.stream(st):
        cuda.cuda._sleep(100_000_000)
        S.copy_(new)
        got = EikonalPicks.apply(S, e, SHOTS, rx, rz)
        st.synchronize()
    assert np.array_equal(got.cpu().numpy(), want, equal_nan=True)


# calls captured by the user: each replay follows its own pairs and progress
# words, not those of the replay before it on another model
@pytest.mark.parametrize("ani", [False, True])
def test_captured_calls_replay_on_a_new_model(engine_lib, cuda, ani):
    from seisfat2d_gb300.synthetic import thomsen_stiffness
    a, b = models()
    rx, rz = surface_receivers(NX, 10.0, step=3)
    obs = np.zeros((len(SHOTS), len(rx)), np.float32)

    def make(m):
        e = engine(m, "compensated")
        if ani:
            vp = 1.0 / models()[0].astype(np.float64)
            e.set_stiffness([c.astype(np.float32) for c in
                             thomsen_stiffness(vp, vp / np.sqrt(3.0), 1000.0, 0.1 + 0 * vp, 0.05 + 0 * vp)])
        return e

    want = []
    for m in (a, b):
        e = make(m)
        pk = e.batch_forward(SHOTS, rx, rz, ani=ani, keep_tape=True)
        want.append((pk, e.misfit_gradient(obs)[1]))
    e = make(a)
    t_obs = cuda.from_numpy(obs).cuda()
    picks, grad = cuda.empty_like(t_obs), cuda.empty((e.nxx, e.nzz), device="cuda")
    st, g = cuda.cuda.Stream(), cuda.cuda.CUDAGraph()

    def calls():
        e.batch_forward(SHOTS, rx, rz, ani=ani, keep_tape=True, out=picks, stream=st)
        e.misfit_gradient(t_obs, out=grad, stream=st, want_misfit=False)

    calls()
    e.synchronize(st)
    with cuda.cuda.graph(g, stream=st):
        calls()
    for k in (0, 1, 0, 1, 1):
        e.set_slowness((a, b)[k])
        g.replay()
        cuda.cuda.synchronize()
        e.synchronize()
        assert np.array_equal(picks.cpu().numpy(), want[k][0], equal_nan=True)
        assert np.array_equal(grad.cpu().numpy(), want[k][1])

"""The Kirchhoff operators' workspace: blocks of cells and groups of tables
give the bits of one block, and a device without room gets smaller ones."""
import numpy as np
import pytest

from helpers import smooth_model

pytestmark = pytest.mark.gpu

NX, NZ, NS, NR, NT, DT, AP, OFF, ANG, DA = 61, 37, 3, 7, 250, 0.002, 40.0, 1e4, 60.0, 2.0
OPERATORS = ["image", "angle_gathers", "image_forward", "angle_forward"]


def engine():
    from seisfat2d_gb300 import Engine
    e = Engine(NX, NZ, 10.0, 10.0)
    e.set_slowness(smooth_model(NX, NZ, 10.0, seed=2))
    return e


@pytest.fixture(scope="module")
def inputs(oracle, engine_lib, cuda):
    S = oracle.expand_boundary(smooth_model(NX, NZ, 10.0, seed=2))
    xs = np.linspace(55.0, 500.0, NS).astype(np.float32)
    xr = np.linspace(15.0, 560.0, NR).astype(np.float32)
    tab = lambda xx: cuda.from_numpy(np.stack([oracle.solve_f32(S, 10.0, 10.0, float(x), 0.0) for x in xx])).cuda()
    geo = (tab(xs), tab(xr), xs, xr)
    gen = cuda.Generator().manual_seed(5)
    data, img = cuda.randn(NS, NR, NT, generator=gen).cuda(), cuda.randn(NX, NZ, generator=gen).cuda()
    shape = engine().kirchhoff_angle_gathers(*geo, data, DT, AP, OFF, ANG, DA).shape
    return geo, data, img, cuda.randn(*shape, generator=gen).cuda()


def run(name, inputs, e, **kw):
    geo, data, img, gat = inputs
    if name == "image":
        return e.kirchhoff_image(*geo, data, DT, AP, OFF, **kw)
    if name == "angle_gathers":
        return e.kirchhoff_angle_gathers(*geo, data, DT, AP, OFF, ANG, DA, **kw)
    if name == "image_forward":
        return e.kirchhoff_image_forward(*geo, img, NT, DT, AP, OFF, **kw)
    return e.kirchhoff_angle_forward(*geo, gat, NT, DT, AP, OFF, ANG, DA, **kw)


# allocations fail that are larger than: five of the ten tables, three, two, a
# few rows or columns, one; and than the smallest block (24 bytes per table and
# cell, 32 with the gradients that the angle domain needs)
@pytest.mark.parametrize("name", OPERATORS)
def test_smaller_blocks_where_memory_is_short(inputs, name):
    from seisfat2d_gb300 import EngineError
    want = run(name, inputs, engine())
    assert np.abs(want).max() > 0
    cell = 32 if name.startswith("angle") else 24
    table, line = cell * NX * NZ, cell * (NS + NR) * (NX if name == "angle_gathers" else NZ)
    smallest = 2 * table if name.endswith("forward") else line
    for limit in (5 * table, 3 * table, 2 * table, 3 * line + 7, line):
        if limit >= smallest:
            e = engine()
            e.test_workspace_limit(limit)
            assert np.array_equal(run(name, inputs, e), want), limit
    e = engine()
    e.test_workspace_limit(smallest // 2)
    with pytest.raises(EngineError) as err:
        run(name, inputs, e)
    assert err.value.status == 6  # SF_ERR_NOMEM
    e.test_workspace_limit(0)
    assert np.array_equal(run(name, inputs, e), want)


# operators of one context on two streams that do not wait for each other, on
# other tables and inputs, eagerly and from two captured graphs, and many traces
# so that they are in flight together
@pytest.mark.parametrize("captured", [False, True])
def test_operators_on_two_streams(engine_lib, cuda, captured):
    from seisfat2d_gb300 import Engine
    nx, nz, ns, nr, nt = 63, 64, 12, 100, 400
    e = Engine(nx, nz, 10.0, 10.0)
    e.set_slowness(np.full((nx, nz), 1 / 2000.0, np.float32))
    xs, xr = np.linspace(105.0, 500.0, ns).astype(np.float32), np.linspace(15.0, 560.0, nr).astype(np.float32)
    x, z = (np.arange(n) * 10.0 - 30.0 for n in (nx + 6, nz + 6))
    gen = cuda.Generator().manual_seed(6)
    jobs = []
    for k in range(2):
        tab = [cuda.from_numpy((np.hypot(x[None, :, None] - p[:, None, None], z + 25.0) / (1600.0 + 800 * k))
                               .astype(np.float32)).cuda() for p in (xs, xr)]
        data, img = cuda.randn(ns, nr, nt, generator=gen).cuda(), cuda.randn(nx, nz, generator=gen).cuda()
        jobs.append((*tab, data, img, cuda.empty_like(img), cuda.empty_like(data)))

    def call(job, stream=None):
        Ts, Tr, data, img, image, traces = job
        e.kirchhoff_image(Ts, Tr, xs, xr, data, 0.004, 40.0, 1e4, out=image, stream=stream)
        e.kirchhoff_image_forward(Ts, Tr, xs, xr, img, nt, 0.004, 40.0, 1e4, out=traces, stream=stream)

    want = []
    for job in jobs:
        call(job)
        cuda.cuda.synchronize()
        want.append([job[-2].clone(), job[-1].clone()])
        assert all(w.abs().max() > 0 for w in want[-1])
    cuda.cuda.synchronize()
    streams, graphs = [cuda.cuda.Stream() for _ in jobs], [cuda.cuda.CUDAGraph() for _ in jobs]
    if captured:
        for job, st, g in zip(jobs, streams, graphs):
            with cuda.cuda.graph(g, stream=st):
                call(job, st)
    for _ in range(20):
        for job in jobs:
            job[-2].zero_(), job[-1].zero_()
        cuda.cuda.synchronize()
        for job, st, g in zip(jobs, streams, graphs):
            with cuda.cuda.stream(st):
                g.replay() if captured else call(job, st)
        cuda.cuda.synchronize()
        for job, w in zip(jobs, want):
            assert cuda.equal(job[-2], w[0]) and cuda.equal(job[-1], w[1])

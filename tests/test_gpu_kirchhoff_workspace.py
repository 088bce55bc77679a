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

"""The kernels' edges: sizes at and next to the tiles, strips, groups and
thresholds of the dispatch rules, against the oracle. The solver's results and
the FP64 filters and sums are compared bit for bit; the Kirchhoff operators
within the bounds of the tests of their own files."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import smooth_model

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(params=["reference", "ieee", "compensated"])
def arith(request, oracle):
    oracle.set_arith(request.param)
    yield request.param
    oracle.set_arith("ieee")


def engine(m, dx=10.0, dz=10.0, arith="ieee"):
    from seisfat2d_gb300 import Engine
    e = Engine(m.shape[0], m.shape[1], dx, dz)
    e.set_arithmetic(arith)
    e.set_slowness(m)
    return e


def receivers(nx, dx, n=23):
    rx = np.linspace(0.0, (nx - 1) * dx, n).astype(np.float32)
    return rx, np.zeros_like(rx)


def check_gradient(oracle, e, m, dx, dz, shots, ani=None, step=0.01, n=23, nonzero=True):
    """Picks, misfit and gradients of a taped batch equal the oracle's."""
    rx, rz = receivers(m.shape[0], dx, n)
    pk = e.batch_forward(shots, rx, rz, ani=ani is not None, keep_tape=True)
    scale = np.float32(step * np.nanmax(pk))
    tobs = (np.nan_to_num(pk) + scale * np.cos(np.arange(pk.size, dtype=np.float32)).reshape(pk.shape))
    J, g = e.misfit_gradient(tobs)
    o = oracle.batch_misfit_gradient(oracle.expand_boundary(m), dx, dz, shots, rx, rz, tobs, ani=ani)
    assert np.array_equal(pk, o[2], equal_nan=True)
    assert abs(J - o[0]) <= 1e-12 * abs(o[0])
    assert np.array_equal(g, o[1]) and (np.abs(g).max() > 0 or not nonzero)
    if ani is not None:
        g11, g13 = e.stiffness_gradient()
        assert np.array_equal(g11, o[4]) and np.array_equal(g13, o[5])


def vti(oracle, m, seed):
    from seisfat2d_gb300.synthetic import thomsen_stiffness
    rng = np.random.default_rng(seed)
    vp = 1.0 / m.astype(np.float64)
    codes, mm = [], []
    for c in thomsen_stiffness(vp, vp / np.sqrt(3.0), 1000.0, rng.uniform(0.0, 0.25, m.shape),
                               rng.uniform(-0.05, 0.15, m.shape)):
        cd, mn, mx = oracle.compress(oracle.expand_boundary(c.astype(np.float32)))
        codes.append(cd)
        mm += [mn, mx]
    return codes, np.array(mm, np.float32)


# padded sizes nx + 6, nz + 6: strips of 31, 32, 33 and 64, 65 rows (a column
# stride of whole strips), 127 and 128 columns (the interior loops' threshold)
@pytest.mark.parametrize("nx,nz,dz", [(20, 25, 10.0), (121, 26, 10.0), (122, 27, 10.0), (260, 58, 8.0), (130, 59, 10.0)])
def test_strip_and_width_edges(oracle, engine_lib, cuda, arith, nx, nz, dz):
    m = smooth_model(nx, nz, 10.0, seed=nx + nz, noise=0.02)
    x = (nx - 1) * 10.0
    w = min(nx, 37)
    shots = [(0.0, 0.0), (x, 0.0), (round(x / 2), 40.0), (100.0, 0.0, 3, w), (x - 100.0, 16.0, nx + 6 - w, w)]
    check_gradient(oracle, engine(m, 10.0, dz, arith), m, 10.0, dz, shots)


# more warps than strip tasks, fewer, and more shots than gangs (the queue);
# windows of unequal size with many gangs take one body for both directions
@pytest.mark.parametrize("warps,gang,nshots", [(1, 1, 30), (1, 3, 30), (2, 6, 30), (8, 8, 500)])
def test_gangs_and_queue(oracle, engine_lib, cuda, arith, warps, gang, nshots):
    nx, nz = 150, 60
    m = smooth_model(nx, nz, 10.0, seed=5)
    e = engine(m, arith=arith)
    e.set_launch(warps, gang)
    e.set_strip_loop("interior")
    rng = np.random.default_rng(nshots)
    shots = []
    for k in range(nshots):
        n = 156 if k % 3 == 0 else int(rng.integers(40, 150))
        c0 = int(rng.integers(0, 156 - n + 1))
        shots.append((float(10 * rng.integers(c0 + 2, c0 + n - 10)), float(rng.integers(0, 300)), c0, n))
    check_gradient(oracle, e, m, 10.0, 10.0, shots)


# slowness outside the fast range (all of it, one node): the strip loops'
# IEEE form; the qP pass then puts the second solve there too
@pytest.mark.parametrize("outlier", [False, True])
@pytest.mark.parametrize("ani", [False, True])
def test_slowness_outside_fast_range(oracle, engine_lib, cuda, arith, ani, outlier):
    m = smooth_model(140, 40, 10.0, seed=8)
    cij = vti(oracle, m, 8) if ani else None
    if outlier:
        m[70, 20] *= 1e-6
    else:
        m = m * np.float32(2e-6)
    e = engine(m, arith=arith)
    if ani:
        e.set_stiffness_codes(*cij)
    # (stiffnesses over the square of that slowness overflow FP32 and leave no qP slowness, hence no gradient)
    check_gradient(oracle, e, m, 10.0, 10.0, [(300.0, 0.0), (1100.0, 20.0, 30, 116)], ani=cij,
                   nonzero=outlier or not ani)


def test_tables_in_a_row(oracle, engine_lib, cuda):
    """Table copies follow each other, the solve before them and other work on
    their stream in order, eagerly and in a captured graph."""
    m = smooth_model(203, 87, 10.0, seed=6)
    S = oracle.expand_boundary(m)
    shots = [(100.0 * k + 30.0, 0.0) for k in range(12)]
    want = np.stack([oracle.solve_f32(S, 10.0, 10.0, *s) for s in shots])
    e = engine(m)
    none = np.zeros(0, np.float32)
    T = cuda.zeros(want.shape, device="cuda")
    for _ in range(3):
        e.batch_forward(shots, none, none, keep_tables=True)
        for k in range(12):
            e.batch_table(k, e.nxx, out=T[k])
            T[k].mul_(2.0)
        assert np.array_equal(T.cpu().numpy(), 2 * want)
    st, g = cuda.cuda.Stream(), cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(g, stream=st):
        for k in range(12):
            e.batch_table(k, e.nxx, out=T[k], stream=st)
        T.mul_(4.0)
    g.replay()
    assert np.array_equal(T.cpu().numpy(), 4 * want)


# the qP pass's groups of shots: one shot, a partly filled last group
@pytest.mark.parametrize("nshots", [1, 41])
def test_qp_groups(oracle, engine_lib, cuda, nshots):
    m = smooth_model(600, 20, 10.0, seed=3)
    cij = vti(oracle, m, 3)
    e = engine(m)
    e.set_stiffness_codes(*cij)
    shots = [(130.0 * k + 60.0, 0.0, *((0, 606) if k % 4 else (13 * k, 70))) for k in range(nshots)]
    check_gradient(oracle, e, m, 10.0, 10.0, shots, ani=cij)


# the misfit's 1024 sums: below, at and past a row, a thread's eight loads, the rest
@pytest.mark.parametrize("nrec", [5, 1023, 1024, 1025, 8193, 20000])
def test_residual_sums(engine_lib, cuda, nrec):
    m = smooth_model(60, 20, 10.0, seed=2)
    e = engine(m)
    rx = (np.arange(nrec) % 60 * 10.0).astype(np.float32)
    pk = e.batch_forward([(300.0, 0.0)], rx, np.zeros_like(rx), keep_tape=True)
    tobs = pk + np.random.default_rng(nrec).standard_normal(pk.shape).astype(np.float32)
    tobs.ravel()[3::7] = np.nan
    J, _ = e.misfit_gradient(tobs)
    r = np.zeros(-(-nrec // 1024) * 1024)
    r[:nrec] = np.nan_to_num(pk - tobs).ravel()
    part = np.zeros(1024)
    for row in r.reshape(-1, 1024):
        part += row * row  # the square of a binary32 value is exact
    s = 512
    while s:
        part[:s] += part[s:2 * s]
        s //= 2
    assert J == 0.5 * part[0]


# the smoothing's 32 x 32 tiles, a cell or (from a tile per SM on) four cells a
# thread, kernels up to wider than a tile, as an argument (31) or copied (33)
@pytest.mark.parametrize("nx,nz,samples", [(4, 4, 3), (31, 33, 5), (32, 32, 1), (33, 63, 31), (65, 36, 71),
                                           (700, 253, 31), (703, 250, 33)])
def test_smoothing_tiles(oracle, engine_lib, cuda, nx, nz, samples):
    f = np.random.default_rng(nx).standard_normal((nx, nz)).astype(np.float32)
    e = engine(smooth_model(nx, nz, 10.0))
    assert np.array_equal(e.smooth_model(f, 3.0, samples), oracle.model_smoothing(f, 3.0, samples))


# the wavelet filters: traces shorter than, at and past a CTA's samples, and a
# wavelet of more taps than one fetch (a low cut-off at a fine step)
@pytest.mark.parametrize("nt,dt,fmax", [(1, 0.002, 20.0), (255, 0.002, 20.0), (257, 0.002, 20.0), (1024, 0.001, 30.0),
                                        (1300, 0.0005, 3.0)])
def test_filter_lengths(oracle, engine_lib, cuda, nt, dt, fmax):
    e = engine(smooth_model(20, 10, 10.0))
    tr = np.random.default_rng(nt).standard_normal((3, nt)).astype(np.float32)
    assert np.array_equal(e.forward_convolution(tr, dt, fmax), oracle.forward_convolution(tr, dt, fmax))
    assert np.array_equal(e.adjoint_convolution(tr, dt, fmax), oracle.adjoint_convolution(tr, dt, fmax))


# the Kirchhoff operators at cell counts that are no multiple of 32, more
# receivers than one buffer holds, and a cell whose table has no gradient; the
# bounds are those of the tests against the oracle in the operators' own files
@pytest.mark.parametrize("nx,nz,nrec", [(23, 17, 1), (32, 16, 8), (37, 29, 131)])
def test_kirchhoff_edges(oracle, engine_lib, cuda, nx, nz, nrec):
    m = smooth_model(nx, nz, 10.0, seed=4)
    S = oracle.expand_boundary(m)
    xs = np.array([30.0, 150.0], np.float32)
    xr = np.linspace(5.0, (nx - 1) * 10.0 - 5.0, nrec).astype(np.float32)
    tab = lambda xx: np.stack([oracle.solve_f32(S, 10.0, 10.0, float(np.float32(round(x))), 0.0) for x in xx])
    Ts, Tr = tab(xs), tab(xr)
    Tr[0, 9:13, 9:13] = Tr[0, 9, 9]
    rng = np.random.default_rng(nrec)
    nt, dt, ap, off = 300, 0.002, 40.0, 1000.0
    d = rng.standard_normal((2, nrec, nt)).astype(np.float32)
    e = engine(m)
    dTs, dTr = cuda.from_numpy(Ts).cuda(), cuda.from_numpy(Tr).cuda()
    img = e.kirchhoff_image(dTs, dTr, xs, xr, d, dt, ap, off)
    ref = oracle.kirchhoff_image(S, Ts, Tr, xs, xr, d, dt, 10.0, 10.0, ap, off)
    assert np.array_equal(np.isfinite(img), np.isfinite(ref))
    scale = np.nanmax(np.abs(ref))
    assert scale > 0 and np.nanmax(np.abs(img - ref)) <= 1e-4 * scale
    x = rng.standard_normal((nx, nz)).astype(np.float32)
    got = e.kirchhoff_image_forward(dTs, dTr, xs, xr, x, nt, dt, ap, off)
    want = oracle.kirchhoff_image_forward(S, Ts, Tr, xs, xr, x, nt, dt, 10.0, 10.0, ap, off)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.nanmax(np.abs(got - want)) <= 2e-5 * np.nanmax(np.abs(want))


PRIMITIVES = r"""
#include <cstdio>
#include "sf_device.cuh"
using namespace sf;
__global__ void k(unsigned long long* bad)
{
    // every significand at every binary exponent of [2^-100, 2^100]
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 threads
    const float c = __uint_as_float(0x3f800000u | ((m * 2654435761u) & 0x7fffffu));
    for (int e = -100; e <= 99; e++) {
        const float a = __uint_as_float((unsigned)(e + 127) << 23 | m);
        if (fsqrt_k<false>(a) != __fsqrt_rn(a)) atomicAdd(bad, 1ull);
        if (frcp_k(a) != __frcp_rn(a)) atomicAdd(bad + 1, 1ull);
        if (fdiv_k<false>(c, a, frcp_k(a)) != __fdiv_rn(c, a)) atomicAdd(bad + 2, 1ull);
    }
}
int main()
{
    unsigned long long *d, h[3];
    if (cudaMalloc(&d, sizeof(h)) || cudaMemset(d, 0, sizeof(h))) return 2;
    k<<<(1 << 23) / 256, 256>>>(d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost)) return 2;
    printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
"""


def test_fast_root_reciprocal_and_quotient(tmp_path, cuda):
    """fsqrt_k and frcp_k equal IEEE's on every operand of [2^-100, 2^100), and
    fdiv_k by frcp_k IEEE's quotient (one dividend per operand)."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "primitives.cu", tmp_path / "primitives"
    src.write_text(PRIMITIVES)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "-I",
                    os.path.join(ROOT, "seisfat2d_gb300", "csrc"), "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["0", "0", "0"]


@pytest.mark.parametrize("big", [np.inf, 3e38])
def test_infinite_pick_gradients(oracle, engine_lib, cuda, arith, big):
    """An infinite pick gradient, and finite ones whose sums overflow, run
    along their own rays: nodes push an exact zero to the neighbours they did
    not take their value from."""
    m = smooth_model(170, 70, 10.0, seed=7, noise=0.02)
    rx, rz = receivers(170, 10.0)
    rx, rz = rx[2:-2] + np.float32(3.7), rz[2:-2] + np.float32(12.3)  # off the nodes: all 16 weights differ from 0
    shots = [(100.0, 0.0), (1500.0, 20.0), (800.0, 300.0, 20, 140)]
    e = engine(m, arith=arith)
    pk = e.batch_forward(shots, rx, rz, keep_tape=True)
    pg = np.ones_like(pk)
    pg[0, 4], pg[2, 9:11] = big, -big
    g = e.batch_adjoint(pg)
    want, _ = oracle.batch_gradient(oracle.expand_boundary(m), 10.0, 10.0, shots, rx, rz, pg)
    bad = ~np.isfinite(want)
    assert 0 < bad.sum() < 0.5 * bad.size
    assert np.array_equal(g, want, equal_nan=True)


def test_forward_operator_sample_limit(engine_lib, cuda):
    """The most time samples a forward CTA holds, and one more."""
    from seisfat2d_gb300 import EngineError
    e = engine(smooth_model(12, 9, 10.0))
    T = cuda.full((1, e.nxx, e.nzz), 0.1, device="cuda")
    args = (T, T, np.array([30.0]), np.array([60.0]), cuda.ones(12, 9, device="cuda"))
    assert e.kirchhoff_image_forward(*args, 51136, 0.002, 40.0, 1e4).shape == (1, 1, 51136)
    with pytest.raises(EngineError) as err:
        e.kirchhoff_image_forward(*args, 51137, 0.002, 40.0, 1e4)
    assert err.value.status == 4  # SF_ERR_RANGE


def test_negative_times_add_nothing(oracle, engine_lib, cuda):
    """Tables with times before the traces' first sample: those cells read no
    sample, as if the traces were zero there."""
    m = smooth_model(33, 21, 10.0, seed=4)
    S = oracle.expand_boundary(m)
    xs, xr = np.array([30.0, 150.0], np.float32), np.array([20.0, 110.0, 290.0], np.float32)
    tab = lambda xx: np.stack([oracle.solve_f32(S, 10.0, 10.0, float(x), 0.0) for x in xx])
    Ts, Tr = tab(xs), cuda.from_numpy(tab(xr)).cuda()
    d = np.random.default_rng(0).standard_normal((2, 3, 300)).astype(np.float32)
    e = engine(m)
    zero = d.copy()
    zero[0] = 0.0
    for shift in (1.0, 1e6):
        early = Ts.copy()
        early[0] -= np.float32(shift)
        for op, ang in ((e.kirchhoff_image, ()), (e.kirchhoff_angle_gathers, (60.0, 2.0))):
            want = op(cuda.from_numpy(Ts).cuda(), Tr, xs, xr, zero, 0.002, 40.0, 1e4, *ang)
            got = op(cuda.from_numpy(early).cuda(), Tr, xs, xr, d, 0.002, 40.0, 1e4, *ang)
            assert np.abs(want).max() > 0 and np.array_equal(got, want)


@pytest.mark.parametrize("dt", [1e-37, 1e-30, 1e30])
def test_extreme_sample_steps(engine_lib, cuda, dt):
    """Steps at which a time's sample lies past FP32's range, past the trace
    or is the first one."""
    e = engine(smooth_model(20, 15, 10.0))
    T = (500.0 + 1e-3 * cuda.arange(e.nzz, dtype=cuda.float32)).expand(1, e.nxx, -1).contiguous().cuda()
    d, x = cuda.ones(1, 1, 8).cuda(), np.array([100.0])
    img = e.kirchhoff_image(T, T, x, x, d, dt, 40.0, 1e4)
    tr = e.kirchhoff_image_forward(T, T, x, x, np.ones((20, 15), np.float32), 8, dt, 40.0, 1e4)
    assert np.isfinite(img).all() and np.isfinite(tr).all()
    assert np.abs(img).max() > 0 if dt > 1 else not img.any()
    assert np.abs(tr[0, 0, 0]) > 0 if dt > 1 else not tr.any()


def test_fused_gather_default(engine_lib, cuda):
    """An untouched context reports what it does, and setting what it reports
    changes nothing."""
    m = smooth_model(150, 60, 10.0, seed=5)
    rx, rz = receivers(150, 10.0)
    e = engine(m)
    e.set_launch(warps=4)
    for _ in range(2):
        pk = e.batch_forward([(300.0, 0.0)], rx, rz, keep_tape=True)
        e.misfit_gradient(pk + np.float32(0.01))
        assert e.fused_gather() == (False, False)
        e.set_fused_gather(e.fused_gather()[0])


def test_undefined_stiffness_factors(oracle, engine_lib, cuda, arith):
    """Cells without a real qP slowness (C33 below zero) have no derivative:
    their gradients are NaN whether or not a ray passes through them."""
    from seisfat2d_gb300.synthetic import thomsen_stiffness
    m = smooth_model(120, 50, 10.0, seed=9)
    rng = np.random.default_rng(9)
    vp = 1.0 / m.astype(np.float64)
    codes, mm = [], []
    for k, c in enumerate(thomsen_stiffness(vp, vp / np.sqrt(3.0), 1000.0, rng.uniform(0.0, 0.25, m.shape),
                                            rng.uniform(-0.05, 0.15, m.shape))):
        if k == 3:
            c = c.copy()
            c[5, 45], c[60, 30] = -c[5, 45], -c[60, 30]
        cd, mn, mx = oracle.compress(oracle.expand_boundary(c.astype(np.float32)))
        codes.append(cd)
        mm += [mn, mx]
    cij = codes, np.array(mm, np.float32)
    e = engine(m, arith=arith)
    e.set_stiffness_codes(*cij)
    rx, rz = receivers(120, 10.0)
    shots = [(300.0, 0.0), (900.0, 20.0, 30, 90)]
    pk = e.batch_forward(shots, rx, rz, ani=True, keep_tape=True)
    tobs = np.zeros_like(pk)
    J, g = e.misfit_gradient(tobs)
    o = oracle.batch_misfit_gradient(oracle.expand_boundary(m), 10.0, 10.0, shots, rx, rz, tobs, ani=cij)
    assert np.array_equal(pk, o[2], equal_nan=True)
    for got, want in zip((g, *e.stiffness_gradient()), (o[1], o[4], o[5])):
        assert np.isnan(want).sum() == 2 and np.nanmax(np.abs(want)) > 0
        assert np.array_equal(got, want, equal_nan=True)


# cell sizes outside the fast updates' range: too large, too small, too oblong
@pytest.mark.parametrize("dx,dz", [(2000.0, 2000.0), (0.01, 0.0125), (200.0, 10.0)])
def test_cells_outside_fast_range(oracle, engine_lib, cuda, arith, dx, dz):
    m = smooth_model(140, 40, 10.0, seed=8, noise=0.02)
    shots = [(30 * dx, 0.0), (110 * dx, 2 * dz, 30, 116)]
    check_gradient(oracle, engine(m, dx, dz, arith), m, dx, dz, shots)


def test_windows_of_unequal_size_at_once(oracle, engine_lib, cuda, arith):
    """More shots than SMs / 2, every one with a gang of its own: no queue, but
    gangs whose sweeps drift apart share one body for both directions."""
    nx, nz = 200, 60
    m = smooth_model(nx, nz, 10.0, seed=5)
    e = engine(m, arith=arith)
    rng = np.random.default_rng(1)
    shots = []
    for _ in range(100):
        n = int(rng.integers(128, nx + 7))
        c0 = int(rng.integers(0, nx + 7 - n))
        shots.append((float(10 * rng.integers(c0 + 2, c0 + n - 10)), float(rng.integers(0, 300)), c0, n))
    check_gradient(oracle, e, m, 10.0, 10.0, shots)
    assert e.strip_loop()[1]


@pytest.mark.parametrize("dx,scale", [(10.0, 1.0), (10.0, 1e-6), (2000.0, 1.0)])
def test_allocation_free_solve_outside_fast_range(oracle, engine_lib, cuda, dx, scale):
    """The allocation-free solve's own checks of slowness and cell sizes."""
    import ctypes as C
    m = smooth_model(140, 70, 10.0, seed=8, noise=0.02)
    m[70, 20] *= np.float32(scale)
    e = engine(m, dx, dx, "reference")
    want = e.time_propagation(30 * dx, 0.0)
    S = cuda.from_numpy(oracle.expand_boundary(m)).cuda()
    T = cuda.empty_like(S)
    for _ in range(2):
        st = e.L.sf_time_propagation_noalloc(C.c_void_p(S.data_ptr()), 140, 70, dx, dx, 30 * dx, 0.0,
                                             C.c_void_p(T.data_ptr()), None)
        assert st == 0 and np.array_equal(T.cpu().numpy(), want)

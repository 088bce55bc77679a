"""Timed workloads of the engine, through its public Python entry points.

Each case is a plain dict: ``kind`` names the path, the rest are its sizes and
options. ``prepare`` makes what a program holds before the call (an Engine,
device inputs, output buffers) from the seed, ``run`` is one pass, ``work`` its
unavoidable bytes and operations, ``exact`` the same outputs in 64 bits from
plain torch (the discrete scheme written out diagonal by diagonal, the
Kirchhoff sums, the convolutions), without the engine.

Models are a linear velocity gradient with smooth anomalies, or layers; the
observed picks and the migration tables come from the closed-form times of
the unperturbed gradient medium.
"""
import math

import numpy as np
import torch

from seisfat2d_gb300 import Engine

NB = 3            # pad cells of the engine's grid
BIG = 1e6         # time of a node no wave has reached
V0 = 1800.0       # surface velocity of the gradient medium (m/s)
F64 = torch.float64


# ------------------------------------------------------------------- cases

def listed():
    return [
        # one shot at a time, as the drop-in modelling loop calls it: a small
        # survey line, where launch and call latency count
        {"name": "shot_small", "kind": "shot", "nx": 201, "nz": 101, "dx": 10.0, "dz": 10.0, "nrec": 96,
         "arith": "reference", "seed_model": "layers"},
        # the same on the plain isotropic benchmark grid
        {"name": "shot", "kind": "shot", "nx": 1001, "nz": 201, "dx": 10.0, "dz": 10.0, "nrec": 1001,
         "arith": "reference", "seed_model": "gradient"},
        # batched modelling of a survey: picks of 200 shots at 800 receivers
        {"name": "forward", "kind": "forward", "nx": 2001, "nz": 501, "dx": 10.0, "dz": 10.0, "nshots": 200, "nrec": 800,
         "arith": "reference", "seed_model": "layers"},
        # traveltime tables for migration on a ragged grid of oblong cells
        {"name": "tables", "kind": "tables", "nx": 1203, "nz": 187, "dx": 12.5, "dz": 10.0, "nshots": 121,
         "arith": "reference", "seed_model": "gradient"},
        # anisotropic modelling, accurate times
        {"name": "forward_vti", "kind": "forward", "nx": 1601, "nz": 401, "dx": 10.0, "dz": 10.0, "nshots": 100, "nrec": 801,
         "arith": "compensated", "seed_model": "gradient", "vti": True},
        # one tomography iteration: new model in, picks, misfit and gradient out
        {"name": "gradient", "kind": "gradient", "nx": 1701, "nz": 351, "dx": 10.0, "dz": 10.0, "nshots": 100, "nrec": 400,
         "arith": "compensated", "seed_model": "gradient"},
        # a few shots of a small odd-sized line in the default arithmetic
        {"name": "gradient_small", "kind": "gradient", "nx": 333, "nz": 97, "dx": 10.0, "dz": 8.0, "nshots": 7, "nrec": 61,
         "arith": "reference", "seed_model": "gradient"},
        # the planned iteration replayed from its graph: many shots, each on
        # its own aperture window, the launch shape a tuning run found
        {"name": "gradient_windows", "kind": "gradient", "nx": 4001, "nz": 1001, "dx": 5.0, "dz": 5.0, "nshots": 1000,
         "nrec": 801, "arith": "compensated", "seed_model": "gradient", "windows": True, "plan": True},
        # one anisotropic tomography iteration with its stiffness gradients
        {"name": "gradient_vti", "kind": "gradient", "nx": 801, "nz": 201, "dx": 10.0, "dz": 10.0, "nshots": 60, "nrec": 201,
         "arith": "compensated", "seed_model": "gradient", "vti": True},
        # the tomography's model update: smoothed step added to the slowness
        {"name": "update", "kind": "update", "nx": 1701, "nz": 351, "dx": 10.0, "dz": 10.0, "stdv": 5.0, "samples": 11,
         "seed_model": "gradient"},
        # Kirchhoff migration of correlated traces, and its angle gathers
        {"name": "migrate", "kind": "migrate", "nx": 1001, "nz": 201, "dx": 10.0, "dz": 10.0, "nsrc": 20, "nrec": 100,
         "nt": 1000, "dt": 0.004, "fmax": 30.0, "angles": False},
        # modelled traces of the least-squares migration, angle domain
        {"name": "lsm_angles", "kind": "lsm", "nx": 501, "nz": 151, "dx": 10.0, "dz": 10.0, "nsrc": 15, "nrec": 60,
         "nt": 800, "dt": 0.004, "fmax": 30.0, "angles": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["shot", "forward", "forward", "tables", "gradient", "gradient", "gradient", "update", "migrate", "lsm"])
    d = rng.choice([5.0, 8.0, 10.0, 12.5])
    c = {"kind": kind, "nx": _logint(rng, 160, 2001), "nz": _logint(rng, 60, 501), "dx": d,
         "dz": d if rng.random() < 0.6 else rng.choice([5.0, 8.0, 10.0, 12.5])}
    if kind in ("shot", "forward", "tables", "gradient"):
        c["arith"] = rng.choice(["reference", "reference", "ieee", "compensated"])
        c["seed_model"] = rng.choice(["gradient", "layers"])
    if kind == "shot":
        c["nrec"] = _logint(rng, 24, 1001)
    elif kind == "forward":
        c.update(nshots=_logint(rng, 4, 200), nrec=_logint(rng, 24, 1001))
        if rng.random() < 0.35:
            c["vti"] = True
            c["nshots"] = min(c["nshots"], 100)
    elif kind == "tables":
        c.update(nx=_logint(rng, 160, 1203), nz=_logint(rng, 60, 251), nshots=_logint(rng, 8, 121))
    elif kind == "gradient":
        c.update(nshots=_logint(rng, 3, 120), nrec=_logint(rng, 24, 801))
        c["arith"] = rng.choice(["reference", "compensated", "compensated"])
        c["seed_model"] = "gradient"
        form = rng.choice(["eager", "eager", "plan", "windows", "vti"])
        if form == "vti":
            c["vti"] = True
        if form in ("plan", "windows"):
            c["plan"] = True
        if form == "windows":
            c["windows"] = True
            c["nx"] = _logint(rng, 400, 4001)
    elif kind == "update":
        c.update(stdv=float(rng.choice([2.0, 5.0, 8.0])), samples=2 * _logint(rng, 2, 15) + 1, seed_model="gradient")
    else:
        c.update(nx=_logint(rng, 160, 1001), nz=_logint(rng, 60, 251), nsrc=_logint(rng, 3, 24), nrec=_logint(rng, 20, 120),
                 nt=_logint(rng, 300, 1500), dt=rng.choice([0.002, 0.004]), fmax=float(rng.choice([20.0, 30.0, 40.0])),
                 angles=rng.random() < 0.5)
    return c


APERTURE, MAX_OFFSET, MAX_ANGLE, ANGLE_STEP = 40.0, 5000.0, 60.0, 2.0


# ------------------------------------------------------------------ inputs

def _grid(c, padded=False):
    """x (columns, 1) and z (1, rows) of the nodes in metres, 64 bits."""
    n = NB if padded else 0
    x = (torch.arange(c["nx"] + 2 * n, device="cuda", dtype=F64) - n) * c["dx"]
    z = (torch.arange(c["nz"] + 2 * n, device="cuda", dtype=F64) - n) * c["dz"]
    return x[:, None], z[None, :]


def _rate(c):
    """Velocity gradient (1/s) of the medium: 4000 m/s at the grid's floor, at least over 1 km."""
    return 2200.0 / max((c["nz"] - 1) * c["dz"], 1000.0)


def _slowness(c, rng):
    """(nx, nz) float32 slowness on the device."""
    x, z = _grid(c)
    lx, lz = float(x[-1, 0]), float(z[0, -1])
    if c.get("seed_model") == "layers":
        v = torch.full((c["nx"], c["nz"]), 1500.0, device="cuda", dtype=F64)
        for k in range(1, 6):
            top = lz * k / 6 + torch.zeros_like(x)
            for _ in range(3):
                top += rng.uniform(5.0, 20.0) * torch.sin(2 * math.pi * (x / lx * rng.uniform(1, 6) + rng.uniform()))
            v += 600.0 * (z >= top)
    else:
        v = V0 + _rate(c) * z + torch.zeros_like(x)
        for _ in range(5):
            s = rng.uniform(0.08, 0.2) * min(lx, 2 * lz)
            v += rng.uniform(-200.0, 200.0) * torch.exp(-((x - rng.uniform(0, lx)) ** 2 + (z - rng.uniform(0, lz)) ** 2)
                                                         / (2 * s * s))
    return (1.0 / v).float()


def _pad(m):
    """Edge-replicated padding of an (nx, nz) field."""
    return torch.nn.functional.pad(m[None, None], (NB,) * 4, mode="replicate")[0, 0].contiguous()


def _shots(c, rng):
    """[(sx, sz, c0, ncols)], float32 receiver coordinates."""
    n, lx = c.get("nshots", 1), (c["nx"] - 1) * c["dx"]
    nxx = c["nx"] + 2 * NB
    shots = []
    for k in range(n):
        sx = float(np.float32(lx * (k + rng.uniform(0.25, 0.75)) / n))
        sz = float(np.float32(c["dz"] * rng.uniform(0.0, 2.0)))
        lo, hi = 0, nxx
        if c.get("windows"):
            w = rng.uniform(0.1, 0.4) * lx
            lo = max(0, int((sx - w / 2) / c["dx"]) + NB)
            hi = min(nxx, int((sx + w / 2) / c["dx"]) + NB + 8)
        shots.append((sx, sz, lo, hi - lo))
    nrec = c.get("nrec", 0)
    rx = (np.arange(nrec) + 0.3) * (lx - 6 * c["dx"]) / max(nrec, 1) + 2 * c["dx"]
    return shots, rx.astype(np.float32), np.full(nrec, 1.25 * c["dz"], np.float32)


def _times(x, z, xs, zs, g):
    """First arrivals of the gradient medium V0 + g z (closed form)."""
    v, vs = V0 + g * z, V0 + g * zs
    return torch.acosh(1 + g * g * ((x - xs) ** 2 + (z - zs) ** 2) / (2 * v * vs)) / g


def _stiffness(c, rng, m):
    """uint16 codes (6, nxx, nzz) and (min, max) pairs of a VTI medium over the model."""
    x, z = _grid(c)
    vp = 1.0 / m.double()
    u = sum(torch.sin(2 * math.pi * (x / x[-1, 0] * rng.uniform(0.5, 3) + z / z[0, -1] * rng.uniform(0.5, 3) + rng.uniform()))
            for _ in range(4)) / 8 + 0.5
    eps, dlt = 0.25 * u, 0.2 * (1 - u) - 0.05
    c33, c55 = 1000.0 * vp ** 2, 1000.0 * vp ** 2 / 3
    c11 = c33 * (1 + 2 * eps)
    c13 = torch.sqrt((c33 - c55) ** 2 + 2 * dlt * c33 * (c33 - c55)) - c55
    codes, mm = [], []
    for f in (c11, c13, 0 * c33, c33, 0 * c33, c55):
        f = _pad(f.float())
        lo, hi = float(f.min()), float(f.max())
        mm += [lo, hi]
        codes.append(torch.ones_like(f) if hi == lo else 1 + 65534 * (f - lo) / (hi - lo))
    return torch.stack(codes).cpu().numpy().astype(np.uint16), np.array(mm, np.float32)


def _inputs(c, seed):
    """Everything random of a case, the same for prepare() and exact()."""
    rng = np.random.default_rng(seed)
    q = {"g": _rate(c)}
    if c["kind"] in ("migrate", "lsm"):
        x, z = _grid(c, padded=True)
        lx = (c["nx"] - 1) * c["dx"]
        for k, n in (("s", c["nsrc"]), ("r", c["nrec"])):
            pos = (lx * (np.arange(n) + rng.uniform(0.2, 0.8)) / n).astype(np.float32)
            q["x" + k] = pos
            p = torch.from_numpy(pos).cuda().double()[:, None, None]
            q["T" + k] = _times(x, z, p, 0.0, q["g"]).float()
        q["m"] = (1.0 / (V0 + q["g"] * _grid(c)[1] + 0 * _grid(c)[0])).float()
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        ntr, nt = c["nsrc"] * c["nrec"], c["nt"]
        f = torch.fft.rfftfreq(2 * nt, c["dt"]).cuda() / (0.4 * c["fmax"])
        noise = torch.fft.rfft(torch.randn(ntr, 2 * nt, device="cuda", generator=gen))
        q["data"] = torch.fft.irfft(noise * f * f * torch.exp(1 - f * f), 2 * nt)[:, :nt].contiguous()
        if c["kind"] == "lsm":
            shape = (_angle_bins(c, q)[:2] if c["angles"] else (c["nx"],)) + (c["nz"],)
            q["image"] = torch.randn(shape, device="cuda", generator=gen)
        return q
    q["m"] = _slowness(c, rng)
    if c["kind"] == "update":
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        q["grad"] = 1e3 * torch.randn(c["nx"] + 2 * NB, c["nz"] + 2 * NB, device="cuda", generator=gen)
        return q
    q["shots"], q["rx"], q["rz"] = _shots(c, rng)
    if c.get("vti"):
        q["codes"], q["mm"] = _stiffness(c, rng, q["m"])
    if c["kind"] == "gradient":
        sx, sz = (torch.tensor([s[k] for s in q["shots"]], device="cuda", dtype=F64)[:, None] for k in (0, 1))
        rx, rz = (torch.from_numpy(a).cuda().double()[None, :] for a in (q["rx"], q["rz"]))
        noise = torch.from_numpy(rng.standard_normal((len(sx), rx.shape[1]))).cuda()
        q["t_obs"] = (_times(rx, rz, sx, sz, q["g"]) + 0.002 * noise).float().contiguous()
    return q


def prepare(case, seed):
    c, q = case, _inputs(case, seed)
    e = Engine(c["nx"], c["nz"], c["dx"], c["dz"])
    if "arith" in c:
        e.set_arithmetic(c["arith"])
    s = {"case": c, "e": e, "m": q["m"], "S": _pad(q["m"])}
    e.set_slowness(s["S"], padded=True)
    if "codes" in q:
        e.set_stiffness_codes(q["codes"], q["mm"])
    if "shots" in q:
        s.update(shots=q["shots"], tab=Engine.shot_table(q["shots"]), rx=q["rx"], rz=q["rz"])
    dev = {"dtype": torch.float32, "device": "cuda"}
    if c["kind"] == "shot":
        s["T"] = torch.empty((e.nxx, e.nzz), **dev)
    elif c["kind"] == "tables":
        s["T"] = torch.empty((c["nshots"], e.nxx, e.nzz), **dev)
    elif c["kind"] == "gradient":
        s["t_obs"] = q["t_obs"]
        s["picks"] = torch.empty((c["nshots"], c["nrec"]), **dev)
        s["grad"] = torch.empty((e.nxx, e.nzz), **dev)
        if c.get("plan"):
            e.set_launch(warps=4)
            e.plan_batch(s["tab"], s["rx"], s["rz"])
            s["misfit"] = torch.empty(1, dtype=F64, device="cuda")
    elif c["kind"] == "update":
        s["grad"] = q["grad"]
    elif c["kind"] in ("migrate", "lsm"):
        s.update({k: q[k] for k in ("Ts", "Tr", "xs", "xr", "data")})
        s["buf"] = torch.empty_like(q["data"])
        s["out"] = torch.empty_like(q["data"]) if c["kind"] == "lsm" else torch.empty((c["nx"], c["nz"]), **dev)
        if c["kind"] == "lsm":
            s["image"] = q["image"]
    return s


def run(s):
    c, e = s["case"], s["e"]
    kind = c["kind"]
    if kind == "shot":
        sx, sz = s["shots"][0][:2]
        e.time_propagation(sx, sz, out=s["T"])
        picks = e.compute_seismogram(s["T"], s["rx"], s["rz"])
        return {"T": s["T"], "reached": s["T"][1:-1, 1:-1], "picks": picks}  # the outer ring keeps its start value
    if kind == "forward":
        return {"picks": e.batch_forward(s["tab"], s["rx"], s["rz"], ani=bool(c.get("vti")))}
    if kind == "tables":
        none = np.zeros(0, np.float32)
        e.batch_forward(s["tab"], none, none, keep_tables=True)
        for k in range(c["nshots"]):
            e.batch_table(k, e.nxx, out=s["T"][k])
        e.synchronize()
        return {"T": s["T"], "reached": s["T"][:, 1:-1, 1:-1]}
    if kind == "gradient":
        e.set_slowness(s["S"], padded=True)
        if c.get("plan"):
            e.plan_graph_launch(s["picks"], s["t_obs"], s["grad"], s["misfit"])
            e.synchronize()
            return {"picks": s["picks"], "misfit": s["misfit"], "grad": s["grad"]}
        e.batch_forward(s["tab"], s["rx"], s["rz"], ani=bool(c.get("vti")), keep_tape=True, out=s["picks"])
        J, _ = e.misfit_gradient(s["t_obs"], out=s["grad"])
        out = {"picks": s["picks"], "misfit": J, "grad": s["grad"]}
        if c.get("vti"):
            out["c11"], out["c13"] = e.stiffness_gradient()
        return out
    if kind == "update":
        e.set_slowness(s["S"], padded=True)
        dS = e.update_slowness(s["grad"], UPDATE_SCALE, c["stdv"], c["samples"])
        return {"dS": dS, "S": e.get_slowness()}
    shape = (c["nsrc"], c["nrec"], c["nt"])
    geo = (s["Ts"], s["Tr"], s["xs"], s["xr"])
    bins = (MAX_ANGLE, ANGLE_STEP) if c["angles"] else ()
    if kind == "migrate":
        d = e.adjoint_convolution(s["data"], c["dt"], c["fmax"], out=s["buf"]).view(shape)
        args = geo + (d, c["dt"], APERTURE, MAX_OFFSET) + bins
        img = e.kirchhoff_angle_gathers(*args) if c["angles"] else e.kirchhoff_image(*args, out=s["out"])
        return {"traces": s["buf"], "image": img}
    args = geo + (s["image"], c["nt"], c["dt"], APERTURE, MAX_OFFSET) + bins
    fwd = e.kirchhoff_angle_forward if c["angles"] else e.kirchhoff_image_forward
    fwd(*args, out=s["buf"].view(shape))
    return {"traces": e.forward_convolution(s["buf"], c["dt"], c["fmax"], out=s["out"])}


UPDATE_SCALE = -1e-9


# -------------------------------------------------------------------- work

def work(c):
    """Inputs once, outputs once; operations of the scheme: about 45 per node
    and sweep of a solve (one root, three divisions counted as one each),
    12 per node of a reverse sweep, 120 per node of the qP pass, 90 per trace
    and cell of a Kirchhoff sum, 2 per tap of a filter."""
    nx, nz, nt = c["nx"], c["nz"], c.get("nt", 0)
    model, pad = 4.0 * nx * nz, 4.0 * (nx + 6) * (nz + 6)
    kind = c["kind"]
    if kind in ("migrate", "lsm"):
        ntr, cells = c["nsrc"] * c["nrec"], nx * nz
        nw = _wavelet_length(c)
        image = model
        if c["angles"]:
            lx = (nx - 1) * c["dx"]
            step = 0.5 * lx / max(c["nsrc"], c["nrec"])
            image = 4.0 * nz * (int(MAX_ANGLE / ANGLE_STEP) + 1) * (int(lx / step) + 1)
        return {"bytes": pad * (c["nsrc"] + c["nrec"] + 1) + 8.0 * ntr * nt + image, "flops": 90.0 * ntr * cells + 2.0 * ntr * nt * nw}
    if kind == "update":
        return {"bytes": 2 * pad + 2 * model, "flops": 2.0 * nx * nz * c["samples"] ** 2}
    ns, nr = c.get("nshots", 1), c.get("nrec", 0)
    cells = (nx + 6) * (nz + 6) * (0.25 if c.get("windows") else 1.0) * ns
    b, f = pad + 4.0 * ns * nr, 180.0 * cells
    if kind in ("shot", "tables"):
        b += pad * ns
    if c.get("vti"):
        b, f = b + 3 * pad, 2 * f + 120.0 * cells
    if kind == "gradient":
        b, f = b + pad + 4.0 * ns * nr, f + 48.0 * cells
        if c.get("vti"):
            b, f = b + 2 * pad, f + 60.0 * cells
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- the same in 64 bits

def _view(a, n, shape0, stride, at):
    """(shape0, n) strided view of rows of `a` (rows, cells) starting at cell `at`."""
    return torch.as_strided(a, (shape0, n), (a.stride(0) if a.shape[0] > 1 else 0, stride), a.storage_offset() + at)


SWEEPS = ((1, 1), (-1, 1), (1, -1), (-1, -1))


def _diagonals(nzz, nxx, sz, sx):
    """Per anti-diagonal of a sweep, in sweep order: lowest cell, stride, count of its inner cells."""
    st = abs(sz - sx * nzz)
    for d in range(2, nzz + nxx - 3):
        lo, hi = max(1, d - (nxx - 2)), min(nzz - 2, d - 1)  # rows counted along the sweep
        if lo > hi:
            continue
        ends = [(i if sz > 0 else nzz - 1 - i) + (d - i if sx > 0 else nxx - 1 - d + i) * nzz for i in (lo, hi)]
        yield min(ends), st, hi - lo + 1


def _solve(T, S, c, win, tape):
    """The four sweeps on T (shots, cells), in place; S (1 or shots, cells).
    win: (shots, 1) first and last padded column of each shot's window. With
    `tape`, per sweep (code, c1, c2) of every node."""
    nzz, nxx = c["nz"] + 2 * NB, c["nx"] + 2 * NB
    dx, dz = float(np.float32(c["dx"])), float(np.float32(c["dz"]))
    ns, N = T.shape
    a, b = 1 / dz ** 2, 1 / dx ** 2
    D, K, kA, hyp = a + b, a * b, a - b, math.hypot(dx, dz)
    cell = torch.arange(N, device="cuda")[None]
    tapes = []
    for sz, sx in SWEEPS:
        if tape:
            code = torch.zeros((ns, N), dtype=torch.uint8, device="cuda")
            c1, c2 = torch.zeros_like(T), torch.zeros_like(T)
        for p, st, n in _diagonals(nzz, nxx, sz, sx):
            def t(o, f=T):
                return _view(f, n, ns, st, p + o)

            def s(o):
                return _view(S, n, ns, st, p + o)
            at = _view(cell, n, 1, st, p)
            i, j = at % nzz, at // nzz
            jw = j - win[0]
            o1, o2 = (-1 if sz > 0 else 0), (-nzz if sx > 0 else 0)
            told, tv, te, tev = t(0), t(-sz), t(-sx * nzz), t(-sz - sx * nzz)
            s1b, s2b, sref = s(o1), s(o2), s(o1 + o2)
            s1a, s2a = torch.where(jw == 1, s1b, s(o1 - nzz)), torch.where(i == 1, s2b, s(o2 - 1))
            t1, t2 = tv + dz * torch.minimum(s1a, s1b), te + dx * torch.minimum(s2a, s2b)
            dte, dtv = te - tev, tv - tev
            is2d = (tv <= te + dx * sref) & (te <= tv + dz * sref) & (dte >= 0) & (dtv >= 0)
            is4 = ~is2d & (dte <= sref * dz * dz / hyp) & (dte > 0)
            is5 = ~is2d & ~is4 & (dtv <= sref * dx * dx / hyp) & (dtv > 0)
            dd = 2 * (te - tv)
            root = torch.sqrt(4 * sref * sref * D - K * dd * dd)
            q = torch.where(is4, dte / dz, dtv / dx)
            edge = torch.sqrt(sref * sref - q * q)
            t3 = ((tev + tv - te) * a + (tev + te - tv) * b + root) / D
            t45 = torch.where(is4, te + dx * edge, tv + dz * edge)
            cand2 = torch.where(is2d, t3, torch.where(is4 | is5, t45, BIG))
            cand1 = torch.minimum(t1, t2)
            new = torch.minimum(cand1, cand2)
            upd = (new < told) & (jw >= 1) & (j <= win[1] - 1)
            if tape:
                one = cand1 <= cand2
                k1, k2 = one & (t1 <= t2), one & (t1 > t2)
                k3, k4, k5 = ~one & is2d, ~one & is4, ~one & is5
                row = torch.where(k2, torch.where((s2a <= s2b) & (i > 1), 0, 1), 0 if sz > 0 else 1)
                col = torch.where(k1, torch.where((s1a <= s1b) & (jw > 1), 0, 1), 0 if sx > 0 else 1)
                kind = k1 * 1 + k2 * 2 + k3 * 3 + k4 * 4 + k5 * 5
                t(0, code).copy_(torch.where(upd, kind + 8 * row + 16 * col, 0))
                h = torch.where(k4, dx, dz)
                e1 = torch.where(k3, (kA + 2 * K * dd / root) / D, torch.where(k4 | k5, h * q / (torch.where(k4, dz, dx) * edge), 0.0))
                e2 = torch.where(k1, dz, torch.where(k2, dx, torch.where(k3, 4 * sref / root, h * sref / edge)))
                t(0, c1).copy_(torch.where(upd, e1, 0.0))
                t(0, c2).copy_(torch.where(upd, e2, 0.0))
            told.copy_(torch.where(upd, new, told))
        if tape:
            tapes.append((code, c1, c2))
    return tapes


def _reverse(lam, tapes, c):
    """Reverse sweeps of dJ/dT (shots, cells), in place; returns dJ/dS per shot (without the initial values')."""
    nzz, nxx = c["nz"] + 2 * NB, c["nx"] + 2 * NB
    ns = lam.shape[0]
    g = torch.zeros_like(lam)
    for (sz, sx), (code, c1, c2) in reversed(list(zip(SWEEPS, tapes))):
        for p, st, n in reversed(list(_diagonals(nzz, nxx, sz, sx))):
            def t(f, o=0):
                return _view(f, n, ns, st, p + o)
            k, cc = t(code) & 7, t(c1)
            mu = t(lam).clone()
            t(lam).mul_(k == 0)
            pv = torch.where(k == 1, 1.0, torch.where(k == 3, cc, torch.where(k == 5, 1 - cc, 0.0)))
            pe = torch.where(k == 2, 1.0, torch.where(k == 3, -cc, torch.where(k == 4, 1 - cc, 0.0)))
            pev = torch.where(k == 3, 1.0, torch.where(k >= 4, cc, 0.0))
            t(lam, -sz).add_(mu * pv)
            t(lam, -sx * nzz).add_(mu * pe)
            t(lam, -sz - sx * nzz).add_(mu * pev)
            v = mu * t(c2)
            for r in (0, 1):
                for q in (0, 1):
                    t(g, r - 1 + (q - 1) * nzz).add_(torch.where((t(code) >> 3) == r + 2 * q, v, 0.0))
    return g


def _stencils(c, q, win):
    """Cells and weights (receivers, 16) of the receivers' cubic stencils; whether each shot's window holds them."""
    nzz = c["nz"] + 2 * NB
    idx, w, inside = [], [], True
    for pos, h, a in ((q["rx"], c["dx"], 1), (q["rz"], c["dz"], 0)):
        h = float(np.float32(h))
        u = (torch.from_numpy(pos).cuda().double() + 0.5 * h) / h
        t = u - 0.5 - torch.floor(u)
        n = u.long() + NB
        first, last = (win if a else (torch.zeros_like(win[0]), torch.full_like(win[0], nzz - 1)))
        inside = inside & (n[None] - 1 >= first + 1) & (n[None] + 2 <= last - 1)
        idx.append((n[:, None] + torch.arange(-1, 3, device="cuda")).clamp(min=0))
        w.append(torch.stack([-0.5 * t + t * t - 0.5 * t ** 3, 1 - 2.5 * t * t + 1.5 * t ** 3,
                              0.5 * t + 2 * t * t - 1.5 * t ** 3, -0.5 * t * t + 0.5 * t ** 3], 1))
    cells = (idx[0][:, :, None] * nzz + idx[1][:, None, :]).flatten(1).clamp(max=(c["nx"] + 2 * NB) * nzz - 1)
    return cells, (w[0][:, :, None] * w[1][:, None, :]).flatten(1), inside


def _start(c, q, S, win):
    """Initial times (shots, cells); the 3 x 3 source cells and distances, (shots, 9)."""
    nzz, nxx = c["nz"] + 2 * NB, c["nx"] + 2 * NB
    dx, dz = float(np.float32(c["dx"])), float(np.float32(c["dz"]))
    sx, sz = (torch.tensor([s[k] for s in q["shots"]], device="cuda", dtype=F64)[:, None] for k in (0, 1))
    o = torch.arange(-1, 2, device="cuda")
    j = ((sx + 0.5 * dx) / dx).long() + NB + o.repeat_interleave(3)[None]
    i = ((sz + 0.5 * dz) / dz).long() + NB + o.repeat(3)[None]
    cells, dist = i + j * nzz, torch.hypot((j - NB) * dx - sx, (i - NB) * dz - sz)
    T = torch.full((len(q["shots"]), nxx * nzz), BIG, device="cuda", dtype=F64)
    T.scatter_(1, cells, S.expand(len(T), -1).gather(1, cells) * dist)
    return T, cells, dist


def _qp(c, q, S, T, win, src):
    """qP slowness of every shot's window and its derivatives by S, C11, C13 along the rays of T."""
    nzz, nxx = c["nz"] + 2 * NB, c["nx"] + 2 * NB
    ns = len(T)
    codes = torch.from_numpy(q["codes"].astype(np.int64)).cuda().double().view(6, -1)
    mm = torch.from_numpy(q["mm"].astype(np.float64)).cuda().view(6, 2)
    c11, c13, c15, c33, c35, c55 = mm[:, :1] + (codes - 1) * (mm[:, 1:] - mm[:, :1]) / 65534
    f = T.view(ns, nxx, nzz)
    gx, gz = torch.zeros_like(f), torch.zeros_like(f)
    gx[:, 1:-1] = 0.5 * (f[:, 2:] - f[:, :-2]) / c["dx"]
    gz[:, :, 1:-1] = 0.5 * (f[:, :, 2:] - f[:, :, :-2]) / c["dz"]
    gx, gz = gx.view(ns, -1), gz.view(ns, -1)
    n = torch.sqrt(gx * gx + gz * gz)
    px, pz = gx / n, gz / n
    at = torch.arange(nxx * nzz, device="cuda")[None]
    i, j = at % nzz, at // nzz
    use = (i >= NB) & (i < nzz - NB) & (j >= win[0] + NB) & (j <= win[1] - NB) & (at != src) & (n > 0)
    xx = c11 * px * px + c55 * pz * pz + 2 * c15 * px * pz
    zz = c55 * px * px + c33 * pz * pz + 2 * c35 * px * pz
    xz = c15 * px * px + c35 * pz * pz + (c13 + c55) * px * pz
    h = 0.5 * (xx - zz)
    r = torch.sqrt(h * h + xz * xz)
    lam = 0.5 * (xx + zz) + r
    vx, vz = torch.where(h >= 0, h + r, xz), torch.where(h >= 0, xz, r - h)
    nv = torch.sqrt(vx * vx + vz * vz)
    vx, vz = vx / nv, vz / nv
    fs = torch.where(use, torch.sqrt(c33 / lam), 1.0)
    Sq = S * fs
    f11 = torch.where(use, -0.5 * Sq * px * px * vx * vx / lam, 0.0)
    f13 = torch.where(use, -Sq * px * pz * vx * vz / lam, 0.0)
    return Sq, (fs, f11, f13)


def _exact_solve(c, q):
    nzz, nxx = c["nz"] + 2 * NB, c["nx"] + 2 * NB
    S = _pad(q["m"]).double().view(1, -1)
    win = tuple(torch.tensor([[f(s)] for s in q["shots"]], device="cuda") for f in (lambda s: s[2], lambda s: s[2] + s[3] - 1))
    taped = c["kind"] == "gradient"
    T, cells, dist = _start(c, q, S, win)
    slow, factors = S, None
    if c.get("vti"):
        _solve(T, S, c, win, False)
        slow, factors = _qp(c, q, S, T, win, cells[:, 4:5])
        T, cells, dist = _start(c, q, slow, win)
    tapes = _solve(T, slow, c, win, taped)
    if c["kind"] == "tables":
        T = T.view(-1, nxx, nzz)
        return {"T": T, "reached": T[:, 1:-1, 1:-1]}
    at, w, inside = _stencils(c, q, win)
    picks = torch.where(inside, (T[:, at.flatten()].view(len(T), *at.shape) * w).sum(2), math.nan)
    if c["kind"] == "shot":
        T = T.view(nxx, nzz)
        return {"T": T, "reached": T[1:-1, 1:-1], "picks": picks[0]}
    if not taped:
        return {"picks": picks}
    res = torch.where(inside, picks - q["t_obs"].double(), 0.0)
    lam = torch.zeros_like(T)
    lam.index_add_(1, at.flatten(), (res[:, :, None] * w).flatten(1))
    del T
    g = _reverse(lam, tapes, c)
    g.scatter_add_(1, cells, lam.gather(1, cells) * dist)
    misfit = 0.5 * (res * res).sum()
    out = {"picks": picks, "misfit": misfit.view(1) if c.get("plan") else float(misfit)}
    if factors is None:
        return dict(out, grad=g.sum(0).view(nxx, nzz))
    return dict(out, **{k: (g * f).sum(0).view(nxx, nzz) for k, f in zip(("grad", "c11", "c13"), factors)})


def _wavelet_length(c):
    dt = float(np.float32(c["dt"]))
    return 2 * int((2 * math.sqrt(math.pi) / c["fmax"] - 0.5 * dt) / dt)


def _filter(c, d, forward):
    """Wavelet convolution (forward) or correlation of traces (traces, nt)."""
    dt, nw, nt = float(np.float32(c["dt"])), _wavelet_length(c), c["nt"]
    td = torch.arange(nw, device="cuda", dtype=F64) * dt - 2 * math.sqrt(math.pi) / c["fmax"]
    a = math.pi ** 3 * (c["fmax"] / (3 * math.sqrt(math.pi))) ** 2 * td * td
    w = (1 - 2 * a) * torch.exp(-a)
    n = 1 << (nt + nw - 2).bit_length()
    shift = nw // 2 + nw // 10
    W, X = torch.fft.rfft(w, 2 * n), torch.fft.rfft(d.double(), 2 * n)
    y = n * torch.fft.irfft(X * (W if forward else W.conj()), 2 * n)
    if forward:
        return y[:, shift:shift + nt]
    return torch.nn.functional.pad(y, (shift, 0))[:, :nt]


def _angle_bins(c, q):
    """CMP bins, angle bins, and each trace's CMP bin (in the geometry's own 32 bits: midpoints fall on bin edges)."""
    step = np.float32(0.5) * min(q["xs"][1] - q["xs"][0], q["xr"][1] - q["xr"][0])
    cmp = np.float32(0.5) * (q["xs"][:, None] + q["xr"][None])
    bins = ((cmp - cmp.min()) / step).astype(np.int64)
    return int(bins.max()) + 1, int(MAX_ANGLE / ANGLE_STEP) + 1, bins


def _kirchhoff(c, q, data, image):
    """Image or gathers of `data` (traces, nt), or, with `image`, the traces of it."""
    nzz, nxx, nt = c["nz"] + 2 * NB, c["nx"] + 2 * NB, c["nt"]
    dx, dz, dt = (float(np.float32(c[k])) for k in ("dx", "dz", "dt"))
    eps = float(np.float32(1e-6))
    mid = (slice(None), slice(NB, nxx - NB), slice(NB, nzz - NB))

    def at(f, a, b):
        return f[:, NB + a:nxx - NB + a, NB + b:nzz - NB + b]
    x, z = _grid(c)
    S = q["m"].double()
    sigma = math.tan(APERTURE * math.pi / 180) * z + eps
    tab = {}
    for k in "sr":
        f = q["T" + k].double()
        gx, gz = 0.5 * (at(f, 1, 0) - at(f, -1, 0)) / dx, 0.5 * (at(f, 0, 1) - at(f, 0, -1)) / dz
        hxx = (at(f, 1, 0) - 2 * f[mid] + at(f, -1, 0)) / dx ** 2
        hzz = (at(f, 0, 1) - 2 * f[mid] + at(f, 0, -1)) / dz ** 2
        hxz = (at(f, 1, 1) - at(f, 1, -1) - at(f, -1, 1) + at(f, -1, -1)) / (4 * dx * dz)
        n = torch.sqrt(gx * gx + gz * gz) + eps
        det = (hxx * hzz - hxz * hxz).abs() + eps
        tab[k] = (f[mid], gx, gz, n, torch.sqrt(det) / n * torch.sqrt((gz / n).abs()) / torch.sqrt((f[mid] / S).clamp(min=eps)),
                  torch.acos((-gz / n).clamp(-1, 1)))
    if c["angles"]:
        ncmp, nang, bins = _angle_bins(c, q)
    shape = (ncmp, nang, c["nz"]) if c["angles"] else (c["nx"], c["nz"])
    out = torch.zeros((c["nsrc"], c["nrec"], nt) if image is not None else shape, device="cuda", dtype=F64)
    iz = torch.arange(c["nz"], device="cuda")[None].expand(c["nx"], -1)
    for s in range(c["nsrc"]):
        ts = [v[s] for v in tab["s"]]
        for r in range(c["nrec"]):
            if not abs(np.float32(q["xs"][s] - q["xr"][r])) < MAX_OFFSET:
                continue
            cmp = 0.5 * (float(q["xs"][s]) + float(q["xr"][r]))
            tr = [v[r] for v in tab["r"]]
            t = torch.floor((ts[0] + tr[0]) / dt).long()
            wgt = (ts[4] * tr[4] * S * (1 + 0.2 * torch.cos(0.5 * (ts[5] + tr[5])))
                   * torch.exp(-0.5 * ((x - cmp) / sigma) ** 2) / (2 * math.pi))
            use = t < nt
            if c["angles"]:
                a = torch.acos(((ts[1] * tr[1] + ts[2] * tr[2]) / (ts[3] * tr[3])).clamp(max=1))
                a = torch.floor(90 * a / math.pi / ANGLE_STEP).long()
                b = int(bins[s, r])
                use = use & (a < nang)
            t = t.clamp(max=nt - 1)
            wgt = torch.where(use, wgt, 0.0)
            if image is not None:
                val = image[b].double()[a.clamp(max=nang - 1), iz] if c["angles"] else image.double()
                out[s, r].index_add_(0, t.flatten(), (wgt * val).flatten())
            else:
                val = wgt * data[s * c["nrec"] + r][t]
                if c["angles"]:
                    out[b].index_put_((a.clamp(max=nang - 1), iz), val, accumulate=True)
                else:
                    out += val
    return out.view(-1, nt) if image is not None else out


def _exact_update(c, q):
    n, h = c["samples"], c["samples"] // 2
    d2 = torch.arange(-h, h + 1, device="cuda", dtype=F64) ** 2
    k = torch.exp(-d2 / (2 * c["stdv"] ** 2))
    k = k / k.sum()
    f = float(np.float32(UPDATE_SCALE)) * q["grad"].double()[NB:-NB, NB:-NB]
    f = torch.nn.functional.conv2d(f[None, None], k.view(1, 1, n, 1), padding=(h, 0))
    dS = torch.nn.functional.conv2d(f, k.view(1, 1, 1, n), padding=(0, h))[0, 0]
    S = _pad(q["m"]).double()
    S[NB:-NB, NB:-NB] += dS
    return {"dS": dS, "S": S}


def exact(case, seed):
    c = case
    if c["kind"] in ("migrate", "lsm"):
        if c["nsrc"] * c["nrec"] > 20000:  # about a millisecond a trace
            return None
        q = _inputs(c, seed)
        if c["kind"] == "lsm":
            return {"traces": _filter(c, _kirchhoff(c, q, None, q["image"]), True)}
        d = _filter(c, q["data"], False)
        return {"traces": d, "image": _kirchhoff(c, q, d, None)}
    if c["kind"] == "update":
        return _exact_update(c, _inputs(c, seed))
    cells = (c["nx"] + 2 * NB) * (c["nz"] + 2 * NB) * c.get("nshots", 1)
    if cells * (100 if c["kind"] == "gradient" else 40) > 150e9:  # does not fit, or takes minutes
        return None
    return _exact_solve(c, _inputs(c, seed))

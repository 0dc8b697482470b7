"""The work that a program using this framework has it do, as timed cases.

Every case goes through the public Python entry points of fold3dpmm and tomo:
solves of the reference's drift medium (F = 1.1, a = (-0.35, 0.4, 0.7), the
implicit-surface source) from device and host fields, the per-plane step that
the reference's own driver calls, solves of the tilted elliptical (TTI) medium
in its three storage forms (float32 metric, FP64 parameters, float32 field),
winner records with the adjoint, batches of solves, and a whole tomography
gradient through autograd.

listed() holds the cases, draw() gives more of the same ranges, prepare()
makes what a program has in hand before the call (fields, media, a context),
run() is one pass, work() what a pass cannot do without, and exact() the same
result from plain torch in float64 where that takes seconds.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fgcs-openacc-advanced_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

MAXT = 10e15
REF_F, REF_A = 1.1, (-0.35, 0.4, 0.7)
# axis normal to the planes, step sign, local x axis and sign, local y axis and sign, of the six directions
DIRS = ((0, 1, 2, 1, 1, 1), (0, -1, 2, -1, 1, -1), (2, 1, 1, 1, 0, 1), (2, -1, 1, -1, 0, -1), (1, -1, 0, -1, 2, -1),
        (1, 1, 0, 1, 2, 1))


def _drift(name, nx, ny, nz, source, sweeps, tol, how="device", F=REF_F, ax=REF_A[0], ay=REF_A[1], az=REF_A[2]):
    c = {"kind": "drift", "nx": nx, "ny": ny, "nz": nz, "source": source, "sweeps": sweeps, "tol": tol, "how": how,
         "F": F, "ax": ax, "ay": ay, "az": az}
    return dict(c, name=name) if name else c


def _ellip(name, nx, ny, nz, medium, field, sweeps, tol, record=False):
    c = {"kind": "ellip", "nx": nx, "ny": ny, "nz": nz, "medium": medium, "field": field, "sweeps": sweeps, "tol": tol,
         "record": record}
    return dict(c, name=name) if name else c


def _many(name, kind, n, lo, hi, medium):
    c = {"kind": kind, "n": n, "lo": lo, "hi": hi, "medium": medium}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the reference driver's own loop: one call per plane, one sweep at its default size
        _drift("drift_planes_128", 128, 128, 128, "surface", 1, 0.0, how="planes"),
        # the smallest solve worth a GPU: every plane step waits for the last one
        _drift("drift_64", 64, 64, 64, "surface", 8, 0.0),
        # odd sizes, a point source, run until the field stops changing
        _drift("drift_ragged_tol", 121, 87, 150, "point", 200, 1e-6),
        # a caller with host buffers: copy in, solve, copy out
        _drift("drift_host_256", 256, 256, 256, "surface", 8, 0.0, how="host"),
        # the published single-GPU benchmark size
        _drift("drift_512", 512, 512, 512, "surface", 8, 0.0),
        # the default benchmark size (two of its eight sweeps, to fit a pass in two seconds)
        _drift("drift_1280", 1280, 1280, 1280, "surface", 2, 0.0),
        # homogeneous tilted ellipse on a float32 metric, to 1e-10: the accuracy configuration
        _ellip("ellip_128", 128, 128, 128, "metric", "f64", 1000, 1e-10),
        # heterogeneous TTI, FP64 parameters, to 1e-10: the 512^3 configuration
        _ellip("tti_512", 512, 512, 512, "param", "f64", 1000, 1e-10),
        # the float32 build at sizes that end in partial tiles
        _ellip("tti_f32_ragged", 380, 319, 257, "metric", "f32", 40, 1e-4),
        # one source's forward record and adjoint, ragged
        _ellip("gradient_ragged", 161, 143, 127, "param", "f64", 1000, 1e-10, record=True),
        # many independent solves of mixed sizes in one call
        _many("batch_24", "batch", 24, 96, 200, "metric"),
        # tomography: loss and gradient over several sources through autograd
        _many("tomography_8x192", "tomo", 8, 192, 192, "param"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drift", "drift", "drift", "planes", "host", "ellip", "ellip", "record", "batch", "tomo"])
    if kind in ("drift", "planes", "host"):
        hi = {"drift": 520, "planes": 160, "host": 300}[kind]
        n = [_log(rng, 24, hi) for _ in range(3)]
        med = {}
        if rng.random() < 0.4:  # another drift of the same kind, well below F
            med = {"F": round(rng.uniform(0.9, 1.6), 3), "ax": round(rng.uniform(-0.45, 0.45), 3),
                   "ay": round(rng.uniform(-0.45, 0.45), 3), "az": round(rng.uniform(-0.45, 0.45), 3)}
        how = {"drift": "device", "planes": "planes", "host": "host"}[kind]
        sweeps = 1 if kind == "planes" else rng.randint(2, 8)
        return _drift(None, *n, rng.choice(["surface", "point"]), sweeps, 0.0, how=how, **med)
    if kind in ("ellip", "record"):
        n = [_log(rng, 24, 180 if kind == "record" else 400) for _ in range(3)]
        medium, field = rng.choice([("metric", "f64"), ("param", "f64"), ("metric", "f32")])
        return _ellip(None, *n, medium, field, 40, 1e-4 if field == "f32" else 1e-10, record=kind == "record")
    if kind == "batch":
        lo = rng.randint(24, 120)
        return _many(None, "batch", rng.randint(4, 32), lo, lo + rng.randint(1, 60), rng.choice(["metric", "param"]))
    n = rng.randint(48, 160)
    return _many(None, "tomo", rng.randint(2, 8), n, n, rng.choice(["metric", "param"]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dims(case, rng):
    """Grid sizes of a batch's instances (the same for every seed of a case)."""
    return [tuple(int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 3)) for _ in range(case["n"])]


def _smooth(x, sigma):
    k = [torch.fft.fftfreq(n, device=x.device, dtype=x.dtype) for n in x.shape[:2]]
    k.append(torch.fft.rfftfreq(x.shape[2], device=x.device, dtype=x.dtype))
    r2 = k[0].view(-1, 1, 1) ** 2 + k[1].view(1, -1, 1) ** 2 + k[2].view(1, 1, -1) ** 2
    return torch.fft.irfftn(torch.fft.rfftn(x) * torch.exp(r2 * (-2.0 * (math.pi * sigma) ** 2)), s=x.shape)


def _tti(nx, ny, nz, h, seed):
    """(vz, eps, axis) of a heterogeneous TTI medium in the field layout:
    Vz = 1500 + 0.8 depth with 16 Gaussian anomalies of +-15 %, eps in
    [0, 0.25] and the axis's tilt and azimuth smoothed over 8 cells at 512."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    cpu = torch.Generator().manual_seed(seed)
    scale = max(nx, ny, nz) / 512.0
    z = torch.arange(nz, dtype=torch.float64, device=dev).view(nz, 1, 1)
    y = torch.arange(ny, dtype=torch.float64, device=dev).view(1, ny, 1)
    x = torch.arange(nx, dtype=torch.float64, device=dev).view(1, 1, nx)
    pert = torch.ones((nz, ny, nx), dtype=torch.float64, device=dev)
    for _ in range(16):
        u = torch.rand(5, generator=cpu, dtype=torch.float64).tolist()
        s = (20.0 + 40.0 * u[3]) * scale
        g = [torch.exp((c - w * n) ** 2 / (-2.0 * s * s)) for c, w, n in ((z, u[0], nz), (y, u[1], ny), (x, u[2], nx))]
        pert += (0.15 if u[4] < 0.5 else -0.15) * (g[0] * g[1]) * g[2]
    vz = pert.mul_(1500.0 + 0.8 * h * z)
    rand = lambda: torch.rand((nz, ny, nx), generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    sig = max(8.0 * scale, 0.5)
    eps = _smooth(0.25 * rand(), sig).clamp_(0.0, 0.25)
    th, ph = torch.deg2rad(45.0 * rand()), torch.deg2rad(360.0 * rand())
    axis = [_smooth(a, sig) for a in (torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th))]
    nn = torch.sqrt(axis[0] ** 2 + axis[1] ** 2 + axis[2] ** 2)
    sg = torch.where(axis[2] < 0, -1.0, 1.0)
    pad = lambda t: torch.nn.functional.pad(t[None, None], (1,) * 6, mode="replicate")[0, 0].contiguous()  # noqa: E731
    return pad(vz), pad(eps), [pad(sg * a / nn) for a in axis]


def _homogeneous(nx, ny, nz):
    full = lambda v: torch.full((nz + 2, ny + 2, nx + 2), v, dtype=torch.float64, device="cuda")  # noqa: E731
    th, ph = math.radians(30.0), math.radians(45.0)  # Vz 2000, Vx = Vy = 2400
    return full(2000.0), full(0.22), [full(math.sin(th) * math.cos(ph)), full(math.sin(th) * math.sin(ph)),
                                      full(math.cos(th))]


def _medium(kind, vz, eps, axis):
    """Four FP64 parameter arrays, or six float32 metric arrays."""
    if kind == "param":
        return [1.0 / vz, eps, axis[0].clone(), axis[1].clone()]
    a = 1.0 / (vz * vz * (1.0 + 2.0 * eps))
    b = 1.0 / (vz * vz) - a
    x, y, z = axis
    return [m.to(torch.float32) for m in (a + b * x * x, b * x * y, b * x * z, a + b * y * y, b * y * z, a + b * z * z)]


def _point_field(nx, ny, nz, src, dtype=torch.float64):
    T = torch.full((nz + 2, ny + 2, nx + 2), MAXT, dtype=dtype, device="cuda")
    T[src[2], src[1], src[0]] = 0.0
    return T


def _place(rng, *n):
    return tuple(int(rng.integers(1, v + 1)) for v in n)


def _drift_field(case, seed):
    """The initial field: a point source, or the implicit surface with three
    further point sources where the surface left the field unset."""
    import fold3dpmm as f3d

    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    if case["source"] == "point":
        return _point_field(nx, ny, nz, _place(rng, nx, ny, nz))
    T = torch.empty((nz + 2, ny + 2, nx + 2), dtype=torch.float64, device="cuda")
    with f3d.Context(0) as c:
        f3d.init_implicit_device(c, T, _spacing(case), f3d.medium(case["F"], (case["ax"], case["ay"], case["az"])))
    left = 3
    for _ in range(100):  # about half of the cells are unset
        i, j, k = _place(rng, nx, ny, nz)
        if left and float(T[k, j, i]) == MAXT:
            T[k, j, i] = 0.0
            left -= 1
    return T


def _spacing(case):
    return (10.0 / (max(case["nx"], case["ny"], case["nz"]) - 1.0),) * 3


def prepare(case, seed):
    import fold3dpmm as f3d

    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "drift":
        T0 = _drift_field(case, seed)
        s = {"case": case, "f3d": f3d, "h": _spacing(case), "med": f3d.medium(case["F"], (case["ax"], case["ay"], case["az"]))}
        if case["how"] == "host":
            s["T0"] = T0.cpu().pin_memory()
            s["T"] = torch.empty_like(s["T0"]).pin_memory()
        else:
            s["T0"], s["T"] = T0, torch.empty_like(T0)
        if case["how"] != "planes":
            s["ctx"] = f3d.Context(0)
            s["o"] = f3d.opts(max_sweeps=case["sweeps"], fixed=case["tol"] == 0.0, tol=case["tol"])
        return s
    if kind == "ellip":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        homog = case["medium"] == "metric" and case["field"] == "f64" and nx == ny == nz == 128
        M = _medium(case["medium"], *(_homogeneous(nx, ny, nz) if homog else _tti(nx, ny, nz, 10.0, seed)))
        dt = torch.float32 if case["field"] == "f32" else torch.float64
        T0 = _point_field(nx, ny, nz, _place(rng, nx, ny, nz), dt)
        s = {"case": case, "f3d": f3d, "h": 10.0, "M": M, "T0": T0, "T": torch.empty_like(T0), "ctx": f3d.Context(0),
             "o": f3d.opts(max_sweeps=case["sweeps"], tol=case["tol"])}
        if case["record"]:  # receivers on the top face: dL/dT there
            s["W"] = torch.empty(T0.shape, dtype=torch.uint8, device="cuda")
            s["r"] = torch.zeros_like(T0)
            gen = torch.Generator(device="cuda").manual_seed(seed)
            s["r"][1, 1:-1:4, 1:-1:4] = torch.randn(s["r"][1, 1:-1:4, 1:-1:4].shape, generator=gen, device="cuda", dtype=dt)
            s["lam"] = torch.empty_like(T0)
            s["g"] = torch.empty((len(M),) + tuple(T0.shape), dtype=dt, device="cuda")
        return s
    if kind == "batch":
        dims = _dims(case, np.random.default_rng(1))
        T0 = [_point_field(*d, _place(rng, *d)) for d in dims]
        M = [_medium(case["medium"], *_tti(*d, 10.0, 1000 * seed + i)) for i, d in enumerate(dims)]
        return {"case": case, "f3d": f3d, "T0": T0, "T": [torch.empty_like(t) for t in T0], "M": M,
                "ctx": f3d.Context(0), "o": f3d.opts(max_sweeps=1000, tol=1e-10)}
    import tomo

    n, k = case["lo"], case["n"]
    M = _medium(case["medium"], *_tti(n, n, n, 10.0, seed))
    T0 = torch.stack([_point_field(n, n, n, _place(rng, n, n)[:2] + (min(11, n),)) for _ in range(k)])
    step = max(1, n // 32)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    obs = 5.0 + torch.rand(T0[:, 1, 1:-1:step, 1:-1:step].shape, generator=gen, device="cuda", dtype=torch.float64)
    return {"case": case, "tomo": tomo, "T0": T0, "obs": obs, "step": step, "M": [m.requires_grad_() for m in M]}


def _inner(T):
    """The field without its ghost layer, which no call writes."""
    return T[..., 1:-1, 1:-1, 1:-1]


def run(s):
    case = s["case"]
    kind = case["kind"]
    f3d = s.get("f3d")
    if kind == "drift":
        if case["how"] == "host":
            rep = s["ctx"].solve(s["T0"], s["h"], s["med"], s["o"], out=s["T"])
            return _inner(s["T"]), rep.sweeps
        T = s["T"].copy_(s["T0"])
        if case["how"] == "planes":
            st = torch.cuda.current_stream().cuda_stream
            for _ in range(case["sweeps"]):
                for d, (nrm, sg) in enumerate(q[:2] for q in DIRS):
                    n = (case["nx"], case["ny"], case["nz"])[nrm]
                    for src in (range(1, n) if sg > 0 else range(n, 1, -1)):
                        f3d.plane(T, s["h"], d, src, s["med"], st)
            return _inner(T)
        rep = s["ctx"].solve(T, s["h"], s["med"], s["o"], torch.cuda.current_stream().cuda_stream)
        return _inner(T), rep.sweeps
    st = torch.cuda.current_stream().cuda_stream
    if kind == "ellip":
        T = s["T"].copy_(s["T0"])
        if not case["record"]:
            rep = f3d.solve_ellip(s["ctx"], T, s["h"], s["M"], s["o"], st)
            return _inner(T), rep.sweeps
        f3d.solve_ellip_record(s["ctx"], T, s["h"], s["M"], s["W"], s["o"], st)
        f3d.adjoint_ellip(s["ctx"], T, s["h"], s["M"], s["W"], s["r"], s["lam"], s["g"],
                          tol=1e-6 if case["field"] == "f32" else 1e-12, stream=st)
        return _inner(T), s["W"], s["lam"], s["g"]
    if kind == "batch":
        for a, b in zip(s["T"], s["T0"]):
            a.copy_(b)
        reps = f3d.solve_batch(s["ctx"], s["T"], [10.0] * case["n"], s["M"], s["o"], st)
        return [_inner(t) for t in s["T"]], [r.sweeps for r in reps]
    T = s["tomo"].solve_batch(s["T0"], 10.0, s["M"], max_sweeps=1000, tol=1e-10, adj_tol=1e-12)
    res = T[:, 1, 1:-1:s["step"], 1:-1:s["step"]] - s["obs"]
    loss = 0.5 * (res * res).sum()
    return _inner(T.detach()), loss.detach(), torch.autograd.grad(loss, s["M"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: fields, media and records in and out once (a whole solve may
    keep the rest on chip).  Flops: one accepted candidate (about 60) per
    point update, at the sweeps asked for, or 6 where a tolerance ends it."""
    kind = case["kind"]
    if kind in ("drift", "ellip"):
        n = [case["nx"], case["ny"], case["nz"]]
    cells = lambda n: float(n[0] * n[1] * n[2])  # noqa: E731
    med = {"metric": 24.0, "param": 32.0}
    if kind == "drift":
        sweeps = case["sweeps"] if case["tol"] == 0.0 else 6
        return {"bytes": 16.0 * cells(n), "flops": 360.0 * sweeps * cells(n)}
    if kind == "ellip":
        b = 4 if case["field"] == "f32" else 8
        m = med[case["medium"]]
        by = (2 * b + m) * cells(n)
        if case["record"]:  # record out and in; field, dL/dT in; lambda and the gradient out
            by += (2 + 3 * b + (4 if case["medium"] == "param" else 6) * b + m) * cells(n)
        return {"bytes": by, "flops": (2 if case["record"] else 1) * 2160.0 * cells(n)}
    if kind == "batch":
        total = sum(cells(d) for d in _dims(case, np.random.default_rng(1)))
        return {"bytes": (16.0 + med[case["medium"]]) * total, "flops": 2160.0 * total}
    c = cells([case["lo"]] * 3)
    return {"bytes": (case["n"] * (16.0 + 24.0 + 2.0) + 2 * med[case["medium"]] + 32.0) * c,
            "flops": 4320.0 * case["n"] * c}


# ---------------------------------------------------------------------------
# The same results in plain torch, float64
# ---------------------------------------------------------------------------
def _plane(T, nrm, i):
    return T[:, :, i] if nrm == 0 else T[:, i, :] if nrm == 1 else T[i]


def _fan(P, nrm, xa, xs, ya, ys):
    """The nine source values of every interior point of plane P, by offset."""
    rows = {0: (1, 2), 1: (0, 2), 2: (0, 1)}[nrm]  # in-plane axes: faster, slower (dim 1, dim 0)
    v, u = P.shape

    def at(i, j):
        off = {xa: i * xs, ya: j * ys}
        a, b = off[rows[1]], off[rows[0]]
        return P[1 + a:v - 1 + a, 1 + b:u - 1 + b]

    return {(i, j): at(i, j) for i in (-1, 0, 1) for j in (-1, 0, 1)}


RIM = ((1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1))


def _sweeps(T, step, max_sweeps, tol, fixed):
    n = (T.shape[2] - 2, T.shape[1] - 2, T.shape[0] - 2)
    for s in range(max_sweeps):
        T_old = None if fixed else T.clone()
        for d, (nrm, sg, xa, xs, ya, ys) in enumerate(DIRS):
            for src in (range(1, n[nrm]) if sg > 0 else range(n[nrm], 1, -1)):
                step(T, d, src, src + sg)
        if not fixed and float((T - T_old).abs().max()) <= tol:
            return s + 1
    return max_sweeps


def _exact_drift(case, T):
    F, a, h = case["F"], (case["ax"], case["ay"], case["az"]), _spacing(case)
    inf = torch.full((), math.inf, dtype=torch.float64, device=T.device)

    def edge(s0, s1, ax, ay, az, hx, hz):
        mn = torch.minimum(s0, s1)
        g = F * F - ay * ay
        d = (s1 - s0) / hx
        c0 = 1.0 - d * ax
        q = g * (c0 * c0 - d * d * (g - az * az))
        c = (-az * c0 + torch.sqrt(q)) / (g - az * az)
        t = s0 + hz * c
        w = torch.sqrt((d * d + c * c) * F * F / g)
        xe = -hz * (d + ax * w) / (c + az * w)
        body = torch.where((q > 0) & (t > mn) & (xe > 0) & (xe < hx), t, inf)
        k = -hx * ax + hz * az
        gg = hx * hx + hz * hz
        q2 = (F * F - ax * ax - ay * ay - az * az) * gg + k * k
        c2 = k + torch.sqrt(q2)
        back = torch.where((q2 > 0) & (c2 > 0), s1 + gg / c2, inf)
        return torch.where((ax > 0) & (s1 > s0), inf, torch.minimum(body, back))

    def frame(d):
        nrm, sg, xa, xs, ya, ys = DIRS[d]
        hz, hx, hy = h[nrm], h[xa], h[ya]
        out = []
        for sign in (1.0, -1.0):
            ax, ay, az = sign * xs * a[xa], sign * ys * a[ya], sign * sg * a[nrm]
            hxy = math.sqrt(hx * hx + hy * hy)
            sp, dg = [], []
            for i, j in RIM:  # spokes: drift along, across and normal
                if i and j:
                    sp.append(((i * ax * hx + j * ay * hy) / hxy, (-j * ax * hy + i * ay * hx) / hxy, az, hxy, hz))
                else:
                    sp.append((i * ax + j * ay, i * ay - j * ax, az, hx if i else hy, hz))
            for q, (i, j) in enumerate(RIM):  # triangles (st, axis neighbour, corner)
                if i and j:
                    continue
                for o in (1, 7):
                    ci, cj = RIM[(q + o) % 8]
                    if i:
                        dg.append((q, (q + o) % 8, i * ax, cj * ay, hx, hy))
                    else:
                        dg.append((q, (q + o) % 8, j * ay, ci * ax, hy, hx))
            out.append((sp, dg, ax, ay, az))
        col = lambda v: torch.tensor(v, dtype=torch.float64, device=T.device).view(2, -1, 1, 1)  # noqa: E731
        sp = [col([[r[k] for r in o[0]] for o in out]) for k in range(5)]
        dg = [col([[r[k] for r in o[1]] for o in out]) for k in range(2, 6)]
        first, corner = [r[0] for r in out[0][1]], [r[1] for r in out[0][1]]
        az = col([[o[4]] for o in out])
        q = [(F * F - (o[2] ** 2 + o[3] ** 2)) * hz * hz for o in out]
        k1 = [o[4] * hz + math.sqrt(v) if v > 0 else 0.0 for o, v in zip(out, q)]
        k1 = [hz * hz / v if v > 0 else math.inf for v in k1]
        return sp, dg, first, corner, az, hz, k1

    frames = [frame(d) for d in range(6)]

    def step(T, d, src, tgt):
        nrm, sg, xa, xs, ya, ys = DIRS[d]
        (sp, dg, first, corner, az, hz, k1) = frames[d]
        f = _fan(_plane(T, nrm, src).abs(), nrm, xa, xs, ya, ys)
        told = _plane(T, nrm, tgt)[1:-1, 1:-1].clone()
        st = f[(0, 0)]
        rim = torch.stack([f[o] for o in RIM])
        both = []
        for side in range(2):
            ax, ay, hx, hy = (t[side] for t in dg)
            s1, s2 = rim[first], rim[corner]
            dx, dy = (s1 - st) / hx, (s2 - s1) / hy
            dd = dx * dx + dy * dy
            z = az[side]
            g = F * F - z * z
            al = 1.0 - ax * dx - ay * dy
            q = al * al - dd * g
            al = (-z * al + F * torch.sqrt(q)) / g
            t = st + hz * al
            w = torch.sqrt(dd + al * al)
            m = -hz / (F * al + z * w)
            xe, ye = m * (F * dx + ax * w), m * (F * dy + ay * w)
            lo = torch.minimum(torch.minimum(s1, s2), st)
            ok = (q > 0) & (t > lo) & (torch.minimum(xe, ye) >= 0) & (ye * hx <= xe * hy) & (xe <= hx)
            gate = ((ax > 0) & (s1 > st)) | ((ay > 0) & (s2 > s1))
            tri = torch.where(ok & ~gate, t, inf)
            hxz = torch.sqrt(hx * hx + hz * hz)
            rot = ax * hz + z * hx
            nest = edge(s1, s2, ay, rot / hxz, (-ax * hx + z * hz) / hxz, hy, hxz)
            nest = torch.where(gate | ((rot > 0) & (s1 > s2)), inf, nest)
            spoke = edge(st, rim, *(t[side] for t in sp))
            c = torch.minimum(torch.minimum(tri.amin(0), nest.amin(0)), spoke.amin(0))
            both.append(torch.minimum(c, st + k1[side]))
        c = torch.where(told < 0, both[1], both[0])
        t = torch.minimum(told.abs(), c)
        _plane(T, nrm, tgt)[1:-1, 1:-1] = torch.where(told > 0, t, -t)

    T = T.clone()
    return T, _sweeps(T, step, case["sweeps"], case["tol"], case["tol"] == 0.0)


def _exact_ellip(case, T, M):
    T = T.to(torch.float64).clone()
    if case["medium"] == "param":
        s, e, x, y = M
        z = torch.sqrt(((1.0 - x * x) - y * y).clamp_min(0.0))
        a = s * s / (1.0 + 2.0 * e)
        b = s * s - a
        M = [a + b * x * x, b * x * y, b * x * z, a + b * y * y, b * y * z, a + b * z * z]
    pair = {(0, 0): 0, (0, 1): 1, (0, 2): 2, (1, 1): 3, (1, 2): 4, (2, 2): 5}
    h = 10.0
    inf = torch.full((), math.inf, dtype=torch.float64, device=T.device)
    col = lambda v: torch.tensor(v, dtype=torch.float64, device=T.device).view(-1, 1, 1)  # noqa: E731
    pts = ((0, 0),) + RIM
    edges = [(0, r + 1) for r in range(8)] + [(r + 1, (r + 1) % 8 + 1) for r in range(8)]
    e0, e1 = [p for p, _ in edges], [q for _, q in edges]
    t1, t2 = [r + 1 for r in range(8)], [(r + 1) % 8 + 1 for r in range(8)]

    def bf(A, u, v):
        xx, yy, zz, xy, xz, yz = A
        return (u[0] * v[0] * xx + u[1] * v[1] * yy + u[2] * v[2] * zz + (u[0] * v[1] + u[1] * v[0]) * xy
                + (u[0] * v[2] + u[2] * v[0]) * xz + (u[1] * v[2] + u[2] * v[1]) * yz)

    P = [col([p[k] for p in pts]) for k in range(2)]
    to = [(-P[0], -P[1], 1.0)]
    eP = [P[k][e0] for k in range(2)]
    eD = [P[k][e1] - P[k][e0] for k in range(2)]
    aD, bD = [P[k][t1] for k in range(2)], [P[k][t2] for k in range(2)]

    def step(T, d, src, tgt):
        nrm, sg, xa, xs, ya, ys = DIRS[d]
        get = lambda p, q: _plane(M[pair[(min(p, q), max(p, q))]], nrm, tgt)[1:-1, 1:-1].to(torch.float64)  # noqa: E731
        A = [get(xa, xa) * h * h, get(ya, ya) * h * h, get(nrm, nrm) * h * h, xs * ys * get(xa, ya) * h * h,
             xs * sg * get(xa, nrm) * h * h, ys * sg * get(ya, nrm) * h * h]
        f = _fan(_plane(T, nrm, src).abs(), nrm, xa, xs, ya, ys)
        t = torch.stack([f[p] for p in pts])
        told = _plane(T, nrm, tgt)[1:-1, 1:-1].clone()
        q = bf(A, to[0], to[0])
        c = torch.where(q > 0, t + torch.sqrt(q), inf).amin(0)
        u, w = (eD[0], eD[1], 0.0), (-eP[0], -eP[1], 1.0)
        a, b, e = bf(A, u, u), bf(A, u, w), bf(A, w, w)
        dt = t[e1] - t[e0]
        n = torch.sqrt((a * e - b * b) / (a - dt * dt))
        lam = (b - dt * n) / a
        ok = (a - dt * dt > 0) & (a * e - b * b > 0) & (lam > 0) & (lam < 1)
        c = torch.minimum(c, torch.where(ok, t[e0] + lam * dt + n, inf).amin(0))
        ua, ub, uz = (aD[0], aD[1], 0.0), (bD[0], bD[1], 0.0), (0.0, 0.0, 1.0)
        p11, p12, p22, q1, q2 = bf(A, ua, ua), bf(A, ua, ub), bf(A, ub, ub), bf(A, ua, uz), bf(A, ub, uz)
        d1, d2 = t[t1] - t[0], t[t2] - t[0]
        det = p11 * p22 - p12 * p12
        u1, u2, w1, w2 = p22 * d1 - p12 * d2, p11 * d2 - p12 * d1, p22 * q1 - p12 * q2, p11 * q2 - p12 * q1
        s = (d1 * u1 + d2 * u2) / det
        r = A[2] - (q1 * w1 + q2 * w2) / det
        n = torch.sqrt(r / (1.0 - s))
        l1, l2 = (w1 - n * u1) / det, (w2 - n * u2) / det
        ok = (det > 0) & (s < 1) & (r > 0) & (l1 > 0) & (l2 > 0) & (l1 + l2 < 1)
        c = torch.minimum(c, torch.where(ok, t[0] + (l1 * d1 + l2 * d2) + n, inf).amin(0))
        v = torch.minimum(told.abs(), c)
        _plane(T, nrm, tgt)[1:-1, 1:-1] = torch.where(told > 0, v, -v)

    k = _sweeps(T, step, case["sweeps"], case["tol"], False)
    return T, k


def exact(case, seed):
    """run()'s outputs from plain torch in float64, or None where that takes
    long: a step of a plane is about two hundred torch operations."""
    kind = case["kind"]
    if kind not in ("drift", "ellip"):
        return None
    n = (case["nx"], case["ny"], case["nz"])
    sweeps = case["sweeps"] if kind == "drift" and case["tol"] == 0.0 else 16 if kind == "drift" else 8
    if sum(n) * 2 * sweeps > 8000 or n[0] * n[1] * n[2] * sweeps > 2.5e8:
        return None
    s = prepare(case, seed)
    if kind == "drift":
        T, k = _exact_drift(case, s["T0"].cuda())
        return _inner(T) if case["how"] == "planes" else (_inner(T), None)
    T, _ = _exact_ellip(case, s["T0"], s["M"])
    return (_inner(T), None, None, None) if case["record"] else (_inner(T), None)

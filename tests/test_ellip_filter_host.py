"""The elliptical medium's FP64 update with its float filter
(csrc/fold3d_ellip.cuh), built for the host, against the oracle, which computes
every candidate: fields and winner records bit for bit, in heterogeneous media
and tilted ellipses of both storage forms, from point sources, and over fields
of independent values (steep gradients, ties, unset points, infinities) that
no settled field holds."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    import build as pkg_build  # fgcs-openacc-advanced_b200/build.py

    out = str(tmp_path_factory.mktemp("ellip_filter") / "libellip_filter.so")
    cmd = [pkg_build.NVCC, "-O2", "-std=c++17", *pkg_build.ARCH, "--fmad=false", "-shared",
           "-Xcompiler", "-fPIC,-ffp-contract=off,-fno-fast-math", "-I", pkg_build.INCLUDE, "-I", pkg_build.CSRC,
           os.path.join(ROOT, "tests", "ellip_filter_host.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    L.ellip_filter_sweeps.argtypes = [C.c_void_p] * 3 + [C.c_int] * 4 + [C.c_double] * 3 + [C.c_int]
    return L


def _check(orc, host, T0, h, M, sweeps, what):
    nz, ny, nx = (n - 2 for n in T0.shape)
    ref = T0.copy()
    with np.errstate(all="ignore"):
        _, _, Wref = (orc.tti_solve_rec if len(M) == 4 else orc.ell_solve_rec)(ref, M, h, sweeps, tol=-1.0)
    T, W = T0.copy(), np.full(T0.shape, 0xFF, dtype=np.uint8)
    M = [np.ascontiguousarray(m, dtype=np.float64 if len(M) == 4 else np.float32) for m in M]
    ptrs = (C.c_void_p * 6)(*(m.ctypes.data for m in M), *([None] * (6 - len(M))))
    host.ellip_filter_sweeps(T.ctypes.data, W.ctypes.data, ptrs, int(len(M) == 4), nx, ny, nz, *h, sweeps)
    assert np.array_equal(T.view(np.uint64), ref.view(np.uint64)), (what, int((T.view(np.uint64) != ref.view(np.uint64)).sum()))
    assert np.array_equal(W, Wref), what


def _medium(rng, dims, kind, param):
    import media

    nx, ny, nz = dims
    if kind == "seeded":
        vz, eps, ax = media.tti_params(nx, ny, nz, 10.0, seed=int(rng.integers(1000)), pad=True)
    else:  # a tilted ellipse, eps to 0.4 (or 8, beyond the filter's range), any axis; "noise": per cell
        shape = (nz + 2, ny + 2, nx + 2) if kind == "noise" else (1, 1, 1)
        import torch

        u = lambda lo, hi: torch.from_numpy(rng.uniform(lo, hi, shape)).expand(nz + 2, ny + 2, nx + 2).contiguous()
        vz, eps = u(1000.0, 4000.0), u(0.0, 8.0 if kind == "extreme" else 0.4)
        th, ph = u(0.0, np.pi / 2), u(0.0, 2 * np.pi)
        ax = (torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th))
    M = media.params_from(vz, eps, ax) if param else media.metric_from(vz, eps, ax)
    return [m.numpy() for m in M]


@pytest.mark.parametrize("param", [False, True], ids=["metric", "param"])
@pytest.mark.parametrize("kind", ["seeded", "ellipse", "extreme", "noise"])
def test_filter_from_point_sources(orc, host, kind, param):
    rng = np.random.default_rng(5 + len(kind) + param)
    for it in range(8):
        dims = tuple(int(v) for v in rng.integers(5, 24, size=3))
        h = tuple(float(v) for v in (rng.uniform(3.0, 15.0, size=3) if it % 2 else rng.uniform(0.2, 20.0, size=3)))
        T0 = np.full((dims[2] + 2, dims[1] + 2, dims[0] + 2), 1e16)
        src = tuple(int(rng.integers(1, n + 1)) for n in dims)
        T0[src[2], src[1], src[0]] = 0.0
        _check(orc, host, T0, h, _medium(rng, dims, kind, param), 6, (kind, it))


@pytest.mark.parametrize("param", [False, True], ids=["metric", "param"])
@pytest.mark.parametrize("kind", ["plain", "ties", "flat", "inf"])
def test_filter_over_independent_values(orc, host, kind, param):
    rng = np.random.default_rng(17 + len(kind) + param)
    for it in range(16):
        dims = tuple(int(v) for v in rng.integers(2, 14, size=3))
        h = tuple(float(v) for v in rng.uniform(3.0, 15.0, size=3))
        M = _medium(rng, dims, ["ellipse", "noise", "extreme"][it % 3], param)
        scale = min(h) / 2000.0 * rng.choice([0.1, 0.5, 3.0])
        shape = (dims[2] + 2, dims[1] + 2, dims[0] + 2)
        T0 = np.abs(10.0 * scale + scale * rng.normal(size=shape))
        if kind == "ties":
            T0 = scale * rng.integers(1, 4, size=shape).astype(float)
        elif kind == "flat":  # plane waves, so that the stationary points agree
            k = np.meshgrid(*(np.arange(n) for n in shape), indexing="ij")
            T0 = 1.0 + sum(float(rng.uniform(-1, 1)) * scale * q for q in k)
            T0 = np.abs(T0 + 3 * scale * (rng.random(shape) < 0.3))
        T0[rng.random(shape) < 0.3] = 1e16
        if kind == "inf":
            T0[rng.random(shape) < 0.2] = np.inf
            T0[rng.random(shape) < 0.05] = 1e300
        T0 = np.where(rng.random(shape) < 0.3, -T0, T0)
        _check(orc, host, T0, h, M, 2, (kind, it))


def test_filter_with_media_out_of_range(orc, host):
    """Non-finite, zero, negative and indefinite metric entries, and metrics far
    from one in scale: every candidate is then kept."""
    rng = np.random.default_rng(29)
    dims, h = (9, 8, 7), (10.0, 9.0, 11.0)
    for it, v in enumerate((np.nan, np.inf, 0.0, -1e-7, 1e-40, 1e35)):
        M = _medium(rng, dims, "noise", False)
        for m in M:
            m[rng.random(m.shape) < 0.1] = v
        if it == 5:
            M = [m * np.float32(1e12) for m in _medium(rng, dims, "ellipse", False)]
        T0 = np.full((dims[2] + 2, dims[1] + 2, dims[0] + 2), 1e16)
        T0[4, 4, 4] = 0.0
        T0[2, 6, 3] = -0.5
        _check(orc, host, T0, h, M, 4, v)

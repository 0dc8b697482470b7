"""The float filter of the drift medium's point update (csrc/fold3d_fast.cuh,
5.) against the oracle's statement, which gates everything in double: one
sweep of the host build over fields of independent values, in which every gate
and body meets times it never meets in a settled field -- unset points,
near-ties, steep gradients, both signs, huge and tiny scales, infinities."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, assert_bitwise
from oracle import REF_A, REF_F


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    import build as pkg_build  # fgcs-openacc-advanced_b200/build.py

    out = str(tmp_path_factory.mktemp("filter_host") / "libfast_host.so")
    cmd = [pkg_build.NVCC, "-O2", "-std=c++17", *pkg_build.ARCH, "--fmad=false", "-shared",
           "-Xcompiler", "-fPIC,-ffp-contract=off,-fno-fast-math", "-I", pkg_build.INCLUDE, "-I", pkg_build.CSRC,
           os.path.join(ROOT, "tests", "fast_solver_host.cu"), os.path.join(pkg_build.CSRC, "fold3d_tables.cpp"),
           "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    L.fast_host_sweeps.argtypes = [C.c_void_p] + [C.c_int] * 3 + [C.c_double] * 7 + [C.c_int] * 2
    return L


def _field(rng, dims, scale, kind):
    nx, ny, nz = dims
    shape = (nz + 2, ny + 2, nx + 2)
    T = 10.0 * scale + scale * rng.normal(size=shape)
    if kind == "ties":  # few distinct values
        T = scale * rng.integers(1, 5, size=shape).astype(float)
    elif kind == "near":  # differences at float's resolution
        T = scale * (5.0 + rng.integers(-3, 4, size=shape) * 2.0 ** -rng.integers(18, 53, size=shape))
    T = np.abs(T)
    T[rng.random(shape) < 0.3] = 10e15
    if kind == "wide":
        T *= 10.0 ** rng.integers(-6, 7, size=shape)
    elif kind == "inf":
        T[rng.random(shape) < 0.2] = np.inf
        T[rng.random(shape) < 0.05] = 1e300
    return np.where(rng.random(shape) < 0.4, -T, T)


@pytest.mark.parametrize("kind", ["plain", "ties", "near", "wide", "inf"])
@pytest.mark.parametrize("units", [1.0, 1e-5, 2e3, 1e-24, 1e24], ids=lambda u: "F*%g" % u)
def test_filter_drops_nothing(orc, host, kind, units):
    rng = np.random.default_rng(int(np.log10(units) * 7 + 200) * 10 + len(kind))
    for it in range(12):
        dims = tuple(int(v) for v in rng.integers(2, 12, size=3))
        F, a = REF_F, REF_A
        h = tuple(float(v) for v in rng.uniform(0.2, 1.0, size=3))
        if it % 3 == 1:  # drifts up to beyond the filter's limit F^2 = 1.1 |a|^2
            d = rng.normal(size=3)
            F, a = 1.3, tuple(1.3 * rng.uniform(0.0, 0.99) * d / np.linalg.norm(d))
        elif it % 3 == 2:  # spacings beyond the filter's limit of 8
            h = (float(rng.uniform(0.02, 0.2)), 0.5, float(rng.uniform(0.5, 2.0)))
        F, a = F * units, tuple(float(v) * units for v in a)
        T0 = _field(rng, dims, min(h) / F * rng.choice([0.1, 0.5, 3.0]), kind)
        ref, T = T0.copy(), T0.copy()
        with np.errstate(all="ignore"):
            orc.solve(ref, h, 2, F=F, a=a)
        host.fast_host_sweeps(T.ctypes.data, *dims, *h, F, *a, 2, 1)
        assert_bitwise(T, ref, "%s, medium %d" % (kind, it))

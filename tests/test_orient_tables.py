"""Direction tables turned into a plane's own axes (csrc/fold3d_tables.cpp:
orient_table) against the oracle, bit for bit, on the host: all six directions,
whose local axes lie along u or v with either sign, media and spacings that tell
every call from every other, both signs of the field, and the early exit on the
sources that the reference names."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, assert_bitwise


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    import build as pkg_build  # fgcs-openacc-advanced_b200/build.py

    out = str(tmp_path_factory.mktemp("orient") / "liborient.so")
    cmd = [pkg_build.NVCC, "-O2", "-std=c++17", *pkg_build.ARCH, "--fmad=false", "-shared",
           "-Xcompiler", "-fPIC,-ffp-contract=off,-fno-fast-math", "-I", pkg_build.INCLUDE, "-I", pkg_build.CSRC,
           os.path.join(ROOT, "tests", "orient_host.cu"), os.path.join(pkg_build.CSRC, "fold3d_tables.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(out)
    L.orient_sweeps.argtypes = [C.c_void_p] + [C.c_int] * 3 + [C.c_double] * 7 + [C.c_int] * 2
    L.orient_sweeps.restype = None
    return L


@pytest.mark.parametrize("plain", [0, 1], ids=["turned", "local"])
@pytest.mark.parametrize("kind", ["point", "noise"])
def test_turned_tables_match_oracle(orc, host, kind, plain):
    rng = np.random.default_rng(41)
    for it in range(16):
        dims = tuple(int(v) for v in rng.integers(2, 22, size=3))
        h = tuple(float(v) for v in rng.uniform(0.2, 1.2, size=3))
        F, d = 1.3, rng.normal(size=3)
        a = tuple(float(v) for v in F * rng.uniform(0.0, 0.97) * d / np.linalg.norm(d))
        shape = (dims[2] + 2, dims[1] + 2, dims[0] + 2)
        if kind == "point":
            T0 = np.full(shape, 1e16)
            T0[tuple(int(rng.integers(1, n + 1)) for n in reversed(dims))] = 0.0
        else:
            s = min(h) / F * rng.choice([0.1, 0.5, 3.0])
            T0 = np.abs(10.0 * s + s * rng.normal(size=shape))
            T0[rng.random(shape) < 0.3] = 1e16
        T0 = np.where(rng.random(shape) < 0.4, -T0, T0)
        ref, T = T0.copy(), T0.copy()
        orc.solve(ref, h, 3, F=F, a=a)
        host.orient_sweeps(T.ctypes.data, *dims, *h, F, *a, 3, plain)
        assert_bitwise(T, ref, "medium %d" % it)

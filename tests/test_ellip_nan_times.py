"""The elliptical medium's FP64 update over fields that hold NaN: a point whose
sources hold one takes what the oracle's order of comparisons takes, no other
candidate is lost, and points away from it are untouched by it.  Bit for bit
where the result is a number."""
import ctypes as C

import numpy as np
import pytest

from test_ellip_filter_host import _medium, host  # noqa: F401


def _case(rng, it):
    dims = tuple(int(v) for v in rng.integers(5, 40 if it == 0 else 14, size=3))
    h = tuple(float(v) for v in rng.uniform(3.0, 15.0, size=3))
    M = _medium(rng, dims, ["seeded", "ellipse", "noise"][it % 3], it % 2 == 1)
    shape, scale = (dims[2] + 2, dims[1] + 2, dims[0] + 2), min(h) / 2000.0
    T0 = np.abs(10.0 * scale + scale * rng.normal(size=shape))
    T0[rng.random(shape) < 0.3] = 1e16
    T0[rng.random(shape) < 0.05] = np.inf
    T0[rng.random(shape) < 0.08] = np.nan
    return dims, h, M, np.where(rng.random(shape) < 0.3, -T0, T0)


def _reference(orc, T0, h, M):
    ref = T0.copy()
    with np.errstate(all="ignore"):
        _, _, W = (orc.tti_solve_rec if len(M) == 4 else orc.ell_solve_rec)(ref, M, h, 2, tol=-1.0)
    return ref, W


def _same(T, W, ref, Wref, what):
    a, b = np.isnan(T), np.isnan(ref)
    assert np.array_equal(a, b), what
    assert np.array_equal(T.view(np.uint64)[~b], ref.view(np.uint64)[~b]), what
    assert np.array_equal(W[~b], Wref[~b]), what


@pytest.mark.parametrize("it", range(12))
def test_nan_sources_host(orc, host, it):  # noqa: F811
    dims, h, M, T0 = _case(np.random.default_rng(it), it)
    T, W = T0.copy(), np.full(T0.shape, 0xFF, dtype=np.uint8)
    A = [np.ascontiguousarray(m, dtype=np.float64 if len(M) == 4 else np.float32) for m in M]
    ptrs = (C.c_void_p * 6)(*(m.ctypes.data for m in A), *([None] * (6 - len(A))))
    host.ellip_filter_sweeps(T.ctypes.data, W.ctypes.data, ptrs, int(len(M) == 4), *dims, *h, 2)
    _same(T, W, *_reference(orc, T0, h, M), it)


@pytest.mark.gpu
@pytest.mark.parametrize("it", range(4))
def test_nan_sources_gpu(f3d, orc, cuda, it):
    dims, h, M, T0 = _case(np.random.default_rng(it), it)
    T = cuda.from_numpy(T0).cuda()
    W = cuda.empty(T.shape, dtype=cuda.uint8, device="cuda")
    with f3d.Context(0) as c:
        f3d.solve_ellip_record(c, T, h, [cuda.from_numpy(np.ascontiguousarray(m)).cuda() for m in M], W,
                               f3d.opts(max_sweeps=2, fixed=True))
    _same(T.cpu().numpy(), W.cpu().numpy(), *_reference(orc, T0, h, M), it)

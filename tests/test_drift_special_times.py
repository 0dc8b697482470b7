"""The drift medium's point update with its float filter over fields that hold
infinities beside times beyond float's range, in media that have no 1-D
candidate (a drift faster than F), and NaN, whose comparisons decide the
reference's early exit: against the oracle, bit for bit where the result is a
number."""
import numpy as np
import pytest

from test_filter_host import host  # noqa: F401


def _case(kind, it):
    rng = np.random.default_rng(it)
    dims = tuple(int(v) for v in rng.integers(3, 40 if it == 0 else 12, size=3))
    h = tuple(float(v) for v in rng.uniform(0.2, 1.0, size=3))
    F, d = 1.3, rng.normal(size=3)
    a = F * (rng.uniform(0.2, 2.0) if kind == "inf" else rng.uniform(0.0, 0.95)) * d / np.linalg.norm(d)
    shape, scale = (dims[2] + 2, dims[1] + 2, dims[0] + 2), min(h) / F
    T0 = np.abs(10.0 * scale + scale * rng.normal(size=shape) * rng.choice([0.1, 1.0, 3.0]))
    T0[rng.random(shape) < 0.2] = 1e16
    if kind == "inf":
        T0[rng.random(shape) < rng.choice([0.3, 0.7])] = np.inf
        T0[rng.random(shape) < 0.5] = 1e300
    else:
        T0[rng.random(shape) < 0.15] = np.nan
    return dims, h, F, tuple(float(v) for v in a), np.where(rng.random(shape) < 0.4, -T0, T0)


def _same(orc, T, T0, h, F, a, what):
    ref = T0.copy()
    with np.errstate(all="ignore"):
        orc.solve(ref, h, 2, F=F, a=a)
    b = np.isnan(ref)
    assert np.array_equal(np.isnan(T), b), what
    assert np.array_equal(T.view(np.uint64)[~b], ref.view(np.uint64)[~b]), what


KINDS = ["inf", "nan"]


@pytest.mark.parametrize("skip", [1, 2], ids=["searched", "closed-form"])
@pytest.mark.parametrize("kind", KINDS)
def test_special_times_host(orc, host, kind, skip):  # noqa: F811
    for it in range(60):
        dims, h, F, a, T0 = _case(kind, it)
        T = T0.copy()
        host.fast_host_sweeps(T.ctypes.data, *dims, *h, F, *a, 2, skip)
        _same(orc, T, T0, h, F, a, it)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_special_times_gpu(f3d, orc, cuda, kind):
    for it in range(12):
        dims, h, F, a, T0 = _case(kind, it)
        for engine in (f3d.ENGINE_WAVEFRONT, f3d.ENGINE_PLANES):
            T = cuda.from_numpy(T0).cuda()
            with f3d.Context(0) as c:
                c.solve(T, h, f3d.medium(F, a), f3d.opts(max_sweeps=2, fixed=True, engine=engine))
            _same(orc, T.cpu().numpy(), T0, h, F, a, (it, engine))

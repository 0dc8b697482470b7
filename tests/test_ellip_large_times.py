"""The elliptical medium's FP64 update with source times so large that an ulp of
the time reaches the filter's margins (an absolute clock in seconds over cells
of milliseconds and below): fields and winner records against the oracle bit
for bit, the host build up to 1e16 cell times and the device at three of them,
single and batched.  Every candidate is then decided on rounded times, ties
among them, so the filter may drop none that could round lower."""
import numpy as np
import pytest

from test_ellip_filter_host import _check, _medium, host  # noqa: F401


def _sources(rng, dims, h, offset):
    """Three sources within a cell time of offset cell times; unset elsewhere."""
    T0 = np.full((dims[2] + 2, dims[1] + 2, dims[0] + 2), 1e300)
    for _ in range(3):
        i, j, k = (int(rng.integers(1, n + 1)) for n in dims)
        T0[k, j, i] = (offset + rng.uniform(0.0, 1.0)) * min(h) / 2000.0
    return T0


@pytest.mark.parametrize("spacings", [(3.0, 15.0), (0.2, 20.0)], ids=["alike", "apart"])
@pytest.mark.parametrize("offset", [1e7, 1e9, 1e10, 1e11, 1e12, 1e14, 1e16])
def test_large_times_host(orc, host, offset, spacings):  # noqa: F811
    rng = np.random.default_rng(3)
    for it in range(12):
        dims = tuple(int(v) for v in rng.integers(12, 28, size=3))
        h = tuple(float(v) for v in rng.uniform(*spacings, size=3))
        M = _medium(rng, dims, ["seeded", "ellipse", "noise"][it % 3], it % 2 == 1)
        T0 = _sources(rng, dims, h, offset)
        _check(orc, host, -T0 if it % 4 == 0 else T0, h, M, 4, (offset, it))


@pytest.mark.gpu
@pytest.mark.parametrize("param", [False, True], ids=["metric", "param"])
@pytest.mark.parametrize("offset", [1e10, 1e12, 1e15])
def test_large_times_gpu(f3d, orc, cuda, offset, param):
    rng = np.random.default_rng(7)
    dims, h = (45, 38, 33), (10.0, 9.0, 11.0)
    M = _medium(rng, dims, "seeded", param)
    T0 = _sources(rng, dims, h, offset)
    ref = T0.copy()
    with np.errstate(all="ignore"):
        _, _, Wref = (orc.tti_solve_rec if param else orc.ell_solve_rec)(ref, M, h, 4, tol=-1.0)
    Md = [cuda.from_numpy(np.ascontiguousarray(m)).cuda() for m in M]
    T, U = (cuda.from_numpy(T0).cuda() for _ in range(2))
    W = cuda.empty(T.shape, dtype=cuda.uint8, device="cuda")
    o = f3d.opts(max_sweeps=4, fixed=True)
    with f3d.Context(0) as c:
        f3d.solve_ellip_record(c, T, h, Md, W, o)
        f3d.solve_batch(c, [U], [h], [Md], o)
    assert np.array_equal(T.cpu().numpy().view(np.uint64), ref.view(np.uint64))
    assert np.array_equal(W.cpu().numpy(), Wref)
    assert cuda.equal(T, U)

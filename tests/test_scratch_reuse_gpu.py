"""Drift and elliptical solves of one grid taking turns on one context: the
scratch of the first two serves the rest (device memory in use stays as it is),
though the media use other tile heights, and every result is that of a context
of its own, with tiles skipped on the marks that the other medium's passes left
behind."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(200, 190, 180), (1000, 37, 70)], ids=["cube", "long"])
def test_media_take_turns(f3d, cuda, dims):
    import media

    nx, ny, nz = dims
    T0 = cuda.full((nz + 2, ny + 2, nx + 2), 10e15, dtype=cuda.float64, device="cuda")
    T0[nz // 2, ny // 3, nx // 2] = 0.0
    M = media.params_from(*media.tti_params(nx, ny, nz, 10.0, seed=2, device="cuda", pad=True))
    o = f3d.opts(max_sweeps=5, fixed=True)
    solve = {"drift": lambda c, T: c.solve(T, 0.01, None, o), "ellip": lambda c, T: f3d.solve_ellip(c, T, 10.0, M, o)}
    want = {}
    for k in solve:
        want[k] = T0.clone()
        with f3d.Context(0) as c:
            solve[k](c, want[k])
    T = T0.clone()
    left = []
    with f3d.Context(0) as c:
        for k in ("ellip", "drift") * 3:
            T.copy_(T0)
            solve[k](c, T)
            assert cuda.equal(T, want[k]), k
            cuda.cuda.synchronize()
            left.append(cuda.cuda.mem_get_info()[0])
    assert left[1] < left[0]  # the drift medium's tiles are smaller: more flags and marks
    assert left[1:] == [left[1]] * 5

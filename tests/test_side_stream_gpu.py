"""A context's first call on a stream that does not wait for the legacy one (a
torch side stream), while the legacy stream is busy: the scratch of single and
batched solves and of the adjoint is cleared on the caller's stream, so the
results are those of a call with nothing else running."""
import pytest

pytestmark = pytest.mark.gpu


def _run(f3d, cuda, kind, stream):
    import media

    nx, ny, nz = 75, 61, 50
    T = cuda.full((nz + 2, ny + 2, nx + 2), 10e15, dtype=cuda.float64, device="cuda")
    T[20, 30, 40] = 0.0
    vz, eps, axis = media.tti_params(nx, ny, nz, 10.0, seed=4, device="cuda", pad=True)
    M = media.params_from(vz, eps, axis)
    W = cuda.empty(T.shape, dtype=cuda.uint8, device="cuda")
    r, lam = cuda.zeros_like(T), cuda.empty_like(T)
    r[1, 1:-1, 1:-1] = 1.0
    g = cuda.zeros((4,) + tuple(T.shape), dtype=cuda.float64, device="cuda")
    U = T.clone()
    o = f3d.opts(max_sweeps=6, fixed=True)
    if kind == "adjoint":
        with f3d.Context(0) as c:
            f3d.solve_ellip_record(c, T, 10.0, M, W, o)
    cuda.cuda.synchronize()
    s = cuda.cuda.current_stream().cuda_stream
    if stream is not None:
        cuda.cuda._sleep(400_000_000)  # about 0.2 s on the legacy stream
        s = stream.cuda_stream
    with f3d.Context(0) as c:
        if kind == "drift":
            c.solve(T, 0.01, None, o, s)
        elif kind == "ellip":
            f3d.solve_ellip(c, T, 10.0, M, o, s)
        elif kind == "batch":
            f3d.solve_batch(c, [T, U], [10.0, 20.0], [M, M], o, s)
        else:
            f3d.adjoint_ellip(c, T, 10.0, M, W, r, lam, g, tol=1e-12, stream=s)
    cuda.cuda.synchronize()
    return [T, U, lam, g] if kind == "adjoint" else [T, U]


@pytest.mark.parametrize("kind", ["drift", "ellip", "batch", "adjoint"])
def test_first_call_beside_a_busy_legacy_stream(f3d, cuda, kind):
    want = _run(f3d, cuda, kind, None)
    got = _run(f3d, cuda, kind, cuda.cuda.Stream())
    for a, b in zip(got, want):
        if kind == "adjoint":  # its sums run in any order
            assert cuda.allclose(a, b, rtol=1e-12, atol=1e-12 * float(b.abs().max()))
        else:
            assert cuda.equal(a, b)

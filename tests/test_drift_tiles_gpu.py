"""The drift medium's dataflow passes at every tile height that the grid's size
can choose (1, 2 and 4 rows), against the PLANES engine bit for bit: two
sweeps, at sizes whose every axis ends in a partial tile, from a point source
and from the implicit surface, and a converged solve with tile skipping."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    assert torch.cuda.is_available()
    return torch


# (grid, source); mean rows of 32 points per plane step: 3, 47, 12 500, 32 700
@pytest.mark.parametrize("dims,source", [((2, 33, 2), "point"), ((61, 35, 30), "surface"), ((33, 2, 97), "point"),
                                         ((641, 633, 627), "surface"), ((1021, 1027, 1025), "point")])
def test_tile_heights_match_planes(f3d, cuda, dims, source):
    nx, ny, nz = dims
    h = (0.01, 0.012, 0.009)
    T0 = cuda.full((nz + 2, ny + 2, nx + 2), 10e15, dtype=cuda.float64, device="cuda")
    with f3d.Context(0) as ctx:
        if source == "point":
            T0[nz // 2 + 1, ny // 2, nx // 2] = 0.0
        else:
            f3d.init_implicit_device(ctx, T0, h)
        got = {}
        for e in (f3d.ENGINE_WAVEFRONT, f3d.ENGINE_PLANES):
            T = T0.clone()
            ctx.solve(T, h, None, f3d.opts(max_sweeps=2, fixed=True, engine=e))
            got[e] = T
        assert cuda.equal(got[f3d.ENGINE_WAVEFRONT].view(cuda.int64), got[f3d.ENGINE_PLANES].view(cuda.int64))
        if max(dims) < 100:  # and to the end, with skipping
            for e in (f3d.ENGINE_WAVEFRONT, f3d.ENGINE_PLANES):
                T = T0.clone()
                got[e] = (ctx.solve(T, h, None, f3d.opts(max_sweeps=300, tol=0.0, engine=e)).sweeps, T)
            (n0, A), (n1, B) = got.values()
            assert n0 == n1 and cuda.equal(A.view(cuda.int64), B.view(cuda.int64))

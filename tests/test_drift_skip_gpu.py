"""The drift medium's dataflow passes with tiles skipped, at every tile height
(1, 2 and 4 rows), over twelve sweeps: the PLANES engine's bits, with fewer
points evaluated than there were.  An item that follows a skipped one has had
its flags read ahead by nine lanes, and every lane then loads what they promise.
The flat grids are of the sizes at which more than 32 M items raise the tile
height."""
import pytest

pytestmark = pytest.mark.gpu


# 1, 2 and 4 rows by the mean rows of a plane step, then 2 and 4 by the number of items
@pytest.mark.parametrize("dims", [(129, 75, 83), (641, 633, 627), (1021, 1027, 1025), (3, 8200, 4100), (3, 8200, 8200)],
                         ids=lambda d: "x".join(map(str, d)))
def test_skipping_matches_planes(f3d, cuda, dims):
    nx, ny, nz = dims
    h = (0.01, 0.012, 0.009)
    T0 = cuda.full((nz + 2, ny + 2, nx + 2), 10e15, dtype=cuda.float64, device="cuda")
    T0[nz // 2 + 1, ny // 2, nx // 2 + 1] = 0.0
    T0[nz // 3, ny - 1, 1] = 0.05
    got = {}
    with f3d.Context(0) as ctx:
        for e in (f3d.ENGINE_WAVEFRONT, f3d.ENGINE_PLANES):
            T = T0.clone()
            rep = ctx.solve(T, h, None, f3d.opts(max_sweeps=12, fixed=True, engine=e))
            got[e] = T
            if e == f3d.ENGINE_WAVEFRONT:
                assert 0 < rep.evaluated_updates < rep.nominal_updates
    A, B = got.values()
    assert cuda.equal(A.view(cuda.int64), B.view(cuda.int64))

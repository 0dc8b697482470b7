"""Batches whose CTAs claim four items at a time (many tiles per resident CTA: a
grid of one CTA per SM) and two (a grid at the limit): the same bits as solves one
by one, with ragged sizes, instances that converge early and a remainder of the
last claim."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True], ids=["f64", "f32"])
@pytest.mark.parametrize("rows,ctas", [(2, 1), (8, 1), (4, 0)])
def test_claims_equal_one_by_one(f3d, orc, rows, ctas, f32):
    torch = pytest.importorskip("torch")
    import media

    n = 40 if rows < 8 else 120
    rng = np.random.default_rng(5)
    T, M, one = [], [], []
    dt = torch.float32 if f32 else torch.float64
    with f3d.Context(0) as ctx:
        f3d.batch_set_config(ctx, rows, ctas)
        for i in range(n):
            nx, ny, nz = (int(v) for v in rng.integers(57, 75, 3)) if i % 4 else (9, 5, 67)
            vz, eps, axis = media.tti_params(nx, ny, nz, 10.0, seed=i, device="cuda", pad=True)
            M.append(media.metric_from(vz, eps, axis) if f32 else media.params_from(vz, eps, axis))
            T0 = torch.from_numpy(orc.init_point(nx, ny, nz, (nx // 2, 1 + i % 4, nz // 3))).cuda().to(dt)
            T.append(T0.clone())
            one.append(T0)
        opts = f3d.opts(max_sweeps=40, tol=1e-6 if f32 else 1e-10)
        reps = f3d.solve_batch(ctx, T, [10.0] * n, M, opts)
        for i in range(n):
            r = f3d.solve_ellip(ctx, one[i], 10.0, M[i], opts)
            assert r.sweeps == reps[i].sweeps
            assert torch.equal(T[i], one[i]), i

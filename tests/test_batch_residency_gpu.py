"""Batches of every tile height at the limit of resident CTAs keep at least the
warps per SM that the build option stands for (five CTAs of four), so the
autotuner compares the heights on the same footing."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 4, 8])
def test_resident_warps(f3d, cuda, rows):
    import media

    n = 2
    M = media.params_from(*media.tti_params(20, 20, 20, 10.0, seed=1, device="cuda", pad=True))
    T = [cuda.full((22, 22, 22), 10e15, dtype=cuda.float64, device="cuda") for _ in range(n)]
    for t in T:
        t[5, 5, 5] = 0.0
    with f3d.Context(0) as c:
        f3d.batch_set_config(c, rows, 0)
        f3d.solve_batch(c, T, [10.0] * n, [M] * n, f3d.opts(max_sweeps=1, fixed=True))
        used = f3d.batch_get_config(c)
    assert used[0] == rows
    assert used[0] * used[1] >= 20

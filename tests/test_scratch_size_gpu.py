"""Device memory that a context's first drift solve takes for its flags and
change maps: below 100 MB up to the 512^3 grid, on which flags a sector apart
would cost 134 MB and gain nothing."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 400, 512])
def test_scratch_of_a_drift_solve(f3d, cuda, n):
    T = cuda.full((n + 2,) * 3, 10e15, dtype=cuda.float64, device="cuda")
    T[n // 2, n // 2, n // 2] = 0.0
    o = f3d.opts(max_sweeps=1, fixed=True)
    with f3d.Context(0) as c:  # the kernels' own memory is taken before the count
        c.solve(T[:10, :10, :10].contiguous(), 0.01, None, o)
        cuda.cuda.synchronize()
        before = cuda.cuda.mem_get_info()[0]
        c.solve(T, 0.01, None, o)
        assert before - cuda.cuda.mem_get_info()[0] < 100e6

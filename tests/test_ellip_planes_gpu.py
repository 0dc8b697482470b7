"""The FP64 elliptical passes at both plane sizes (a CTA with several items per
step, and fewer), both storage forms of the medium: fields and winner records
against the oracle bit for bit, from a point source and over a field of
independent times of both signs with unset and infinite ones among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("param", [False, True], ids=["metric", "param"])
@pytest.mark.parametrize("source", ["point", "noise"])
@pytest.mark.parametrize("dims", [(1023, 197, 3), (37, 70, 33)], ids=["large", "small"])
def test_planes_match_oracle(f3d, orc, dims, source, param):
    torch = pytest.importorskip("torch")
    import media

    nx, ny, nz = dims
    h = (10.0, 9.0, 11.0)
    vz, eps, axis = media.tti_params(nx, ny, nz, 10.0, seed=3, device="cuda", pad=True)
    M = media.params_from(vz, eps, axis) if param else media.metric_from(vz, eps, axis)
    rng = np.random.default_rng(8)
    T0 = orc.init_point(nx, ny, nz, (nx // 2, ny // 3, 2))
    if source == "noise":
        T0 = np.abs(0.05 + 0.01 * rng.normal(size=T0.shape))
        T0[rng.random(T0.shape) < 0.3] = 10e15
        T0[rng.random(T0.shape) < 0.05] = np.inf
        T0 = np.where(rng.random(T0.shape) < 0.3, -T0, T0)
    ref = T0.copy()
    Mh = [m.cpu().numpy() for m in M]
    with np.errstate(all="ignore"):
        _, _, Wref = (orc.tti_solve_rec if param else orc.ell_solve_rec)(ref, Mh, h, 2, tol=-1.0)
    T = torch.from_numpy(T0).cuda()
    W = torch.empty(T.shape, dtype=torch.uint8, device="cuda")
    with f3d.Context(0) as ctx:
        f3d.solve_ellip_record(ctx, T, h, M, W, f3d.opts(max_sweeps=2, fixed=True))
    assert np.array_equal(T.cpu().numpy().view(np.uint64), ref.view(np.uint64))
    assert np.array_equal(W.cpu().numpy(), Wref)

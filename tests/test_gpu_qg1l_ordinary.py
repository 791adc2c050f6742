"""float64 stages at ordinary points (moderate values: one upwind difference a
direction, no guards) against the general form, which a plan with a beta term of
zeros runs: same step and adjoint over odd sizes, both staging forms (rows a
multiple of 16 or not), land, still water (the derivative's tie), and values that
must take the general form: NaN, infinities, huge and denormal ones. Both forms
round the same terms (in another order where the flow is negative), so they
agree to some roundings of the largest term: 1e-12 of the field's largest value
after two RK2 steps, per field since an infinite one spreads over its own. The field
of huge values squares itself at each stage: one step, 1e-9, and no adjoint (its
velocities far from the spike are rounding noise, whose sign the derivative sees)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


def same(a, b, tols=(1e-12,) * 3):
    a, b = a.cpu().numpy(), b.cpu().numpy()
    for x, y, tol in zip(a, b, tols):
        assert np.array_equal(np.isnan(x), np.isnan(y))
        inf = np.isinf(y)
        assert np.array_equal(x[inf], y[inf]) and np.array_equal(np.isinf(x), inf)
        fin = np.isfinite(y)
        if fin.any():
            assert np.abs(x - y)[fin].max() <= tol * np.abs(y[fin]).max()


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("ny,nx", [(9, 11), (33, 48), (70, 96), (45, 131)])
def test_matches_general_form(ny, nx, special):
    from vardyn_gb300.qg1l import QG1LPlan, build_mask
    rng = np.random.default_rng(ny + nx)
    land = np.where(rng.random((ny, nx)) < 0.01, np.nan, 0.0)
    land[ny // 2, :] = 0.0
    mk = lambda **kw: QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=torch.float64,
                               mask=build_mask(ny, nx, land), **kw)
    plain, general = mk(), mk(beta=np.zeros((ny, nx)))
    h = rng.standard_normal((3, ny, nx)) * 0.1
    h[0, ny // 4:3 * ny // 4, nx // 4:3 * nx // 4] = 0.25      # still water
    h[1] = h[1][:, :1]                                         # no flow along y
    if special:
        h[0, ny // 2, nx // 2] = np.nan
        h[1, ny // 2, nx // 3] = np.inf
        h[2, ny // 3, nx // 2] = 1e35
        h[2, ny // 3 + 1, nx // 2] = 5e-324
    hd = torch.as_tensor(h, device="cuda")
    hb = torch.zeros_like(hd)
    a = torch.as_tensor(rng.standard_normal(h.shape), device="cuda")
    n, k = (1, 2) if special else (2, 3)
    same(plain.step(hd, hb, nstep=n), general.step(hd, hb, nstep=n), (1e-12, 1e-12, 1e-9 if special else 1e-12))
    same(plain.step_adj(a, hd, hb, nstep=n)[:k], general.step_adj(a, hd, hb, nstep=n)[:k])

"""The masked Dirichlet multigrid's tile kernels at the edges of their tiles:
levels one point wider or narrower than a tile, small and large tiles, a
coarsest level too large for the one-block form, strided fields, land reaching
the walls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (n0, n1, modes, batch): 8 x 32 and 32 x 64 tiles with ragged last tiles;
# 63 x 61 coarsens once to 31 x 30 unknowns, 1023 x 7 to a thin column
CASES = [(15, 15, 1, 1), (31, 63, 1, 1), (33, 65, 2, 1), (63, 61, 1, 2), (127, 129, 1, 1), (95, 255, 3, 2),
         (511, 383, 2, 1), (1023, 15, 1, 1)]


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n0,n1,modes,batch", CASES)
def test_solution_satisfies_the_operator(n0, n1, modes, batch, dtype):
    from vardyn_gb300.helmholtz_mg import MaskedDirichletMG
    rng = np.random.default_rng(n0 * n1)
    k = np.fft.fftfreq(n0)[:, None] ** 2 + np.fft.fftfreq(n1)[None, :] ** 2
    w = np.real(np.fft.ifft2(np.exp(-k / 0.004) * np.fft.fft2(rng.standard_normal((n0, n1)))))
    mask = (w < np.quantile(w, 0.85)).astype(float)
    lam = np.array([0.0, 1e-9, 6e-9])[:modes]
    d0, d1 = 5e3, 4e3
    tol = 1e-10 if dtype == torch.float64 else 2e-5
    mg = MaskedDirichletMG(n0, n1, d0, d1, lam, mask=mask, dtype=dtype, tol=tol, max_cycles=60)
    b = torch.as_tensor(rng.standard_normal((modes, batch, n0, n1)), dtype=dtype, device="cuda")
    u = mg.solve(b).double().cpu().numpy()
    bd = b.double().cpu().numpy() * mask
    assert np.all(u[..., mask == 0] == 0)
    up = np.pad(u, ((0, 0), (0, 0), (1, 1), (1, 1)))
    Au = (up[..., 2:, 1:-1] + up[..., :-2, 1:-1] - 2 * u) / d0 ** 2 + (up[..., 1:-1, 2:] + up[..., 1:-1, :-2] - 2 * u) / d1 ** 2
    Au = mask * (Au - lam[:, None, None, None] * u)
    res = np.linalg.norm(bd - Au, axis=(2, 3)) / np.linalg.norm(bd, axis=(2, 3))
    # the recurred residual met tol; the true one drifts from it by rounding
    # (float32: eps times the operator's norm times the solution's)
    eps = np.finfo(np.float64 if dtype == torch.float64 else np.float32).eps
    drift = 60 * eps * (4 / d0 ** 2 + 4 / d1 ** 2) * np.linalg.norm(u, axis=(2, 3)) / np.linalg.norm(bd, axis=(2, 3))
    assert np.all(mg.rel.cpu().numpy() <= tol)
    assert np.all(res <= tol + drift)
    # strided form: the interior of padded fields, bit for bit
    pb = torch.full((modes * batch, n0 + 3, n1 + 5), 3.0, dtype=dtype, device="cuda")
    pb[:, 1:n0 + 1, 2:n1 + 2] = b.reshape(-1, n0, n1)
    pu = torch.full_like(pb, 9.0)
    ld, fs = n1 + 5, (n0 + 3) * (n1 + 5)
    mg.solve_strided(batch, pb[0, 1:, 2:], ld, fs, pu[0, 1:, 2:], ld, fs)
    assert np.array_equal(pu[:, 1:n0 + 1, 2:n1 + 2].double().cpu().numpy(), u.reshape(-1, n0, n1))
    assert float((pu[:, 0] - 9.0).abs().max()) == 0.0 and float((pu[:, :, :2] - 9.0).abs().max()) == 0.0

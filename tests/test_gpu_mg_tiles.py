"""The multigrid levels' forms against the float64 oracle at the sizes where they
change: levels run as tile kernels whose rows and columns leave remainders of every
tile size (8 x 8 to 16 x 32), levels too large for them, the one-block coarse levels
as clusters of 8, 4 and 2 blocks and as one block (by the number of systems), the
bottom by matrices, by sweeps and by pseudo-inverse. float64: 1e-11, the bound of
the solver's other oracle tests; float32: 2e-4, a rounding of 6e-8 times the
problem's condition number (coefficients up to 8 over the smallest lambda, 2e-3)."""
import numpy as np
import pytest
import torch

from oracle.helmholtz_mg import MGOracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-11), (torch.float32, 2e-4)])
@pytest.mark.parametrize("n0,n1,nsys,niter_bottom", [(104, 72, 1, 20), (200, 136, 1, -1), (336, 304, 1, 20),
                                                     (144, 176, 2, 3), (80, 48, 16, 20), (48, 32, 40, 20),
                                                     (40, 24, 70, -1)])
def test_levels_vs_oracle(n0, n1, nsys, niter_bottom, dtype, tol):
    from vardyn_gb300.helmholtz_mg import MG_Helmholtz
    rng = np.random.default_rng(n0 * 1000 + n1 + nsys)
    mask = np.ones((n0, n1))
    mask[n0 // 3:n0 // 2, n1 // 4:n1 // 2] = 0
    mask[:5, :7] = mask[n0 - 3:, n1 // 2:] = 0
    mask[15:17, 31:33] = 0
    cu = 1.0 + 0.3 * rng.random((n0 + 1, n1))
    cv = 1.0 + 0.3 * rng.random((n0, n1 + 1))
    lam = np.linspace(2e-3, 0.5, nsys)
    rhs = rng.standard_normal((nsys, n0, n1)) * mask
    g = MG_Helmholtz(1.0, 1.3, n0, n1, cu, cv, lambd=lam, mask=mask, niter_bottom=niter_bottom, max_ite=4,
                     dtype=dtype)
    f = g.solve(torch.tensor(rhs, dtype=dtype, device="cuda")).double().cpu().numpy()
    pick = sorted({0, nsys // 2, nsys - 1})
    o = MGOracle(1.0, 1.3, n0, n1, cu, cv, lam[pick], mask=mask, niter_bottom=niter_bottom, max_ite=4)
    want = o.solve(rhs[pick])
    assert np.linalg.norm(f[pick] - want) <= tol * np.linalg.norm(want)

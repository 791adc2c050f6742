"""Gaussian bases over the range of lattices, against the dense products of their windows:
centres closer than the grid columns, a few columns and hundreds of columns a centre
(every number of lanes of the transposed x pass), runs of centres that end inside and at
a block's, more than 64 centres reached by a block of columns, one column and one row."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


def window(s):
    return np.where(np.abs(s) <= 1, np.cos(0.5 * np.pi * s) ** 2, 0.0)


# sigma_D / facns and the grid: lanes a centre 1, 2, 4, 8, 16, 32 and mixed ones
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
@pytest.mark.parametrize("ny,nx,B,comps", [
    (40, 300, 1, [(4.0, 2.0)]), (37, 129, 2, [(8.0, 1.5)]), (30, 260, 1, [(25.0, 1.0)]), (33, 300, 2, [(60.0, 1.2)]),
    (20, 400, 1, [(150.0, 1.0)]), (25, 700, 1, [(600.0, 0.8)]), (1, 128, 1, [(12.0, 1.0)]), (50, 1, 2, [(30.0, 2.0)]),
    (40, 257, 2, [(5.0, 1.5), (300.0, 0.85), (40.0, 1.5), (5.0, 1.5)])])
def test_dense_products(ny, nx, B, comps, dtype, tol):
    from vardyn_gb300.basis import BasisPlan, Gauss3dParams
    rng = np.random.default_rng(ny * nx)
    xc, yc = np.arange(nx) * 5.0, np.arange(ny) * 6.0
    land = rng.random((ny, nx)) < 0.1
    cs = [Gauss3dParams(sd, 3.0 + c, facns=fn, facnlt=1.5) for c, (sd, fn) in enumerate(comps)]
    plan = BasisPlan(xc, yc, np.arange(0.0, 8.1, 0.5), cs, land=land, dtype=dtype)
    k = 5
    X, phi = rng.standard_normal((B, plan.nbasis)), rng.standard_normal((B, ny, nx))
    X, phi = (torch.as_tensor(a, dtype=dtype, device="cuda") for a in (X, phi))
    G, GT = plan.project(k, X).double().cpu().numpy(), plan.project_T(k, phi, torch.zeros_like(X)).double().cpu().numpy()
    Xn, pn = X.double().cpu().numpy(), phi.double().cpu().numpy() * ~land
    exp, expT = np.zeros((B, ny, nx)), np.zeros((B, plan.nbasis))
    for c, (sd, _) in enumerate(comps):
        o, nt, ns = plan.component(c)
        _, lat, lon = plan.lattice(c)
        W = (window((yc[:, None] - lat) / sd)[:, None, :] * window((xc[:, None] - lon) / sd)[None, :, :]).reshape(-1, ns)
        for it, w in plan.time_weights(k, c):
            sl = slice(o + it * ns, o + (it + 1) * ns)
            exp += w * (Xn[:, sl] @ W.T).reshape(B, ny, nx)
            expT[:, sl] += w * (pn.reshape(B, -1) @ W)
    exp *= ~land
    assert np.linalg.norm(G - exp) <= tol * np.linalg.norm(exp)
    assert np.linalg.norm(GT - expT) <= tol * np.linalg.norm(expT)

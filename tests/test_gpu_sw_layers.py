"""Shallow-water right-hand side kernels over the layer counts and the grid
edges: every layer count's pressure sum (1 to the largest), grids below, at
and above the thread block, land next to each edge, against the float64
oracle. The float64 tolerance is the other model tests' 1e-11 (a few hundred
roundings of 1e-16 a step over three steps, amplified by the differences of
pressures that nearly cancel)."""
import numpy as np
import pytest
import torch

from oracle.sw import SWOracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("nx,ny,nl,land", [(8, 32, 1, False), (9, 33, 2, True), (7, 31, 3, True), (6, 6, 5, False),
                                           (12, 65, 8, True)])
def test_steps_vs_oracle(nx, ny, nl, land):
    from vardyn_gb300.sw import SWPlan
    rng = np.random.default_rng(nx * 100 + ny + nl)
    dx = 2e3 * (1 + 0.15 * rng.random((nx, ny)))
    dy = 2.5e3 * (1 + 0.15 * rng.random((nx, ny)))
    f = 1e-4 + 2e-11 * np.arange(ny + 1)[None, :] * 2.5e3 + np.zeros((nx + 1, 1))
    H = 100.0 + 50.0 * np.arange(nl).reshape(nl, 1, 1)
    gp = np.r_[9.81, 0.02 + 0.0 * np.arange(nl - 1)]
    mask = np.ones((nx, ny))
    if land:
        mask[0, 3:6] = mask[nx // 2, ny // 2] = mask[nx - 1, 0] = 0
        mask[1:3, ny - 1] = 0
    opt = dict(slip_coef=0.7, bottom_drag_coef=2e-6, visc_coef=5.0, diff_coef=2.0, taux=0.04, tauy=-0.02)
    o = SWOracle(dict(nx=nx, ny=ny, nl=nl, dx=dx, dy=dy, H=H, g_prime=gp, f=f, dt=10.0, mask=mask, **opt))
    m = o.masks
    u = 0.05 * rng.standard_normal((2, nl, nx + 1, ny)) * m.u
    v = 0.05 * rng.standard_normal((2, nl, nx, ny + 1)) * m.v
    h = 0.4 * rng.standard_normal((2, nl, nx, ny)) * m.h
    v[0] *= rng.random(v[0].shape) < 0.8          # faces at rest
    want = o.step(u, v, h, nstep=3)
    for dtype, tol in ((torch.float64, 1e-11), (torch.float32, 2e-4)):
        pl = SWPlan(nx, ny, nl, dx, dy, f, H, gp, 10.0, mask=mask, dtype=dtype, **opt)
        got = pl.step(*(torch.tensor(a, dtype=dtype, device="cuda") for a in (u, v, h)), nstep=3)
        for a, b, k in zip(got, want, "uvh"):
            assert np.abs(a.cpu().numpy() - b).max() <= tol * np.abs(b).max(), (k, dtype)

"""The tiled adjoint of the shallow-water tendency at the edges of its tiles
(24 x 32 and 32 x 32 targets): one below, at and above a tile's rows and columns,
grids inside one tile, land on a tile's boundary, more than one member. The
adjoint is held against the tangent by dot products (the tangent runs the
forward kernels on dual numbers and shares no code with the tiles): 1e-12 in
float64 and 1e-4 in float32, the bounds of the other dot-product tests. The
sums are in a fixed order: two runs are equal in every bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-4)])
@pytest.mark.parametrize("nx,ny,nl,B", [(6, 6, 2, 1), (22, 30, 1, 2), (23, 31, 3, 1), (24, 32, 1, 1), (25, 33, 2, 2),
                                        (30, 64, 1, 1), (31, 63, 2, 1), (32, 65, 1, 1), (49, 34, 8, 1)])
def test_dot_product(nx, ny, nl, B, dtype, tol):
    from vardyn_gb300.sw import SWPlan
    rng = np.random.default_rng(1000 * nx + 10 * ny + nl)
    dx = 2e3 * (1 + 0.15 * rng.random((nx, ny)))
    dy = 2.5e3 * (1 + 0.15 * rng.random((nx, ny)))
    f = 1e-4 + 2e-11 * np.arange(ny + 1)[None, :] * 2.5e3 + np.zeros((nx + 1, 1))
    H = 100.0 + 50.0 * np.arange(nl).reshape(nl, 1, 1)
    gp = np.r_[9.81, 0.02 + 0.0 * np.arange(nl - 1)]
    mask = np.ones((nx, ny))
    if nx > 8:
        mask[nx // 2, 3:9] = mask[min(nx - 1, 23):min(nx, 25), ny - 3] = 0
    pl = SWPlan(nx, ny, nl, dx, dy, f, H, gp, 10.0, mask=mask, dtype=dtype, slip_coef=0.7, bottom_drag_coef=2e-6,
                visc_coef=5.0, diff_coef=2.0, taux=0.04, tauy=-0.02)
    m = pl.masks
    t = lambda a: torch.tensor(a, dtype=dtype, device="cuda")
    shp = ((B, nl, nx + 1, ny), (B, nl, nx, ny + 1), (B, nl, nx, ny))
    mk = (np.asarray(m.u), np.asarray(m.v), np.asarray(m.h))
    x = [t(s * rng.standard_normal(n) * k) for s, n, k in zip((0.05, 0.05, 0.4), shp, mk)]
    d = [t(s * rng.standard_normal(n) * k) for s, n, k in zip((0.01, 0.01, 0.1), shp, mk)]
    a = [t(rng.standard_normal(n)) for n in shp]
    tl = pl.step_tgl(*x, *d, nstep=2)
    g1 = pl.step_adj(*x, *a, nstep=2)
    g2 = pl.step_adj(*x, *a, nstep=2)
    g1, g2 = ([v for v in (g.values() if isinstance(g, dict) else g) if v is not None][:3] for g in (g1, g2))
    for p, q in zip(g1, g2):
        assert torch.equal(p, q)
    dot = lambda p, q: sum(float((c.double() * e.double()).sum()) for c, e in zip(p, q))
    size = sum(float((c.double() * e.double()).abs().sum()) for c, e in zip(tl, a))
    lhs, rhs = dot(tl, a), dot(d, g1)
    assert abs(lhs - rhs) <= tol * max(abs(lhs), 1e-2 * size)

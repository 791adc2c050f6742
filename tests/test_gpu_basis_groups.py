"""Gaussian bases with components on the same space lattice (projected as one
group) against the sum of their components' own plans; rows of more than 64
centres, more than 128 table entries, lon/lat rows, land, two windows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


def comps_of(kind):
    from vardyn_gb300.basis import Gauss3dParams
    if kind == "interleaved":
        return [Gauss3dParams(sd, st, facns=fn, facnlt=st / 2.0, sigma_Q=0.01)
                for st in (3.0, 7.0) for sd, fn in ((60.0, 0.9), (120.0, 1.0), (60.0, 2.0))]
    if kind == "long rows":        # 100 centres a row, one group of three
        return [Gauss3dParams(20.0, st, facns=1.0, facnlt=1.0) for st in (2.0, 4.0, 9.0)]
    # dense lattices: 12 or more rows over a point in each of 7 groups, and many time centres
    return [Gauss3dParams(200.0 + 10 * (c % 7), 4.0, facns=6.0, facnlt=8.0) for c in range(9)]


@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("kind", ["interleaved", "long rows", "dense"])
def test_groups_equal_the_sum_of_components(kind, geographic):
    from vardyn_gb300.basis import BasisPlan
    rng = np.random.default_rng(5)
    ny, nx = (40, 201) if kind == "long rows" else (45, 70)
    xc, yc = np.arange(nx) * 10.0, np.arange(ny) * 10.0
    if geographic:
        xc, yc = -20.0 + xc / 110.0, 30.0 + yc / 110.0
    times = np.arange(0.0, 5.1, 0.5)
    land = rng.random((ny, nx)) < 0.1
    cs = comps_of(kind)
    kw = dict(land=land, geographic=geographic, dtype=torch.float64)
    plan = BasisPlan(xc, yc, times, cs, **kw)
    k, B = 4, 2
    X = torch.as_tensor(rng.standard_normal((B, plan.nbasis)), device="cuda")
    phi = torch.as_tensor(rng.standard_normal((B, ny, nx)), device="cuda")
    G, adX = plan.project(k, X), plan.project_T(k, phi, torch.zeros_like(X))
    out, ad = torch.zeros_like(G), torch.zeros_like(X)
    for c, p in enumerate(cs):
        one = BasisPlan(xc, yc, times, [p], **kw)
        o = plan.component(c)[0]
        sl = slice(o, o + one.nbasis)
        out += one.project(k, X[:, sl].contiguous())
        ad[:, sl] = one.project_T(k, phi, torch.zeros(B, one.nbasis, dtype=torch.float64, device="cuda"))
    assert float((G - out).norm() / out.norm()) < 1e-13
    # the space products of a group are formed once, with the same sums
    assert float((adX - ad).norm() / ad.norm()) < 1e-14
    assert float((plan.project(k, X, out=G.clone(), accumulate=True) - 2 * G).abs().max()) < 1e-14 * float(G.abs().max())

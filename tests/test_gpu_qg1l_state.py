"""float32 model state: the PV pair evaluated in float64 (integer conversions,
NaN guard), and background fields that are zero for some windows only."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


def plans(ny, nx, **kw):
    from vardyn_gb300.qg1l import QG1LPlan
    return [QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=d, **kw) for d in (torch.float32, torch.float64)]


@pytest.mark.parametrize("special", [False, True])
def test_pv_pair_equals_float64(special):
    from vardyn_gb300.qg1l import build_mask
    ny, nx, B = 45, 70, 2
    rng = np.random.default_rng(3)
    mask = build_mask(ny, nx, np.where(rng.random((ny, nx)) < 0.01, np.nan, 0.0))
    p, p64 = plans(ny, nx, mask=mask)
    h = (10.0 ** rng.uniform(-6, 3, (B, ny, nx)) * rng.choice([-1, 1], (B, ny, nx))).astype(np.float32)
    hb = rng.standard_normal((B, ny, nx)).astype(np.float32)
    h[0, 5:9, 5:9] = 0.0
    if special:
        h[0, 20, 20], h[0, 30, 31], h[0, 31, 31] = np.nan, np.inf, -np.inf
        h[1, 10, 10], h[1, 11, 12] = 1e-42, -3e-41           # denormal
    hd, hbd = (torch.as_tensor(a, device="cuda") for a in (h, hb))
    q, qb, qlo = torch.empty_like(hd), torch.empty_like(hd), torch.empty_like(hd)
    p.init_state(hd, hbd, q, qb, qlo)
    exp = p64.h2pv(hd.double(), hbd.double()).cpu().numpy()
    got = (q.double() + qlo.double()).cpu().numpy()
    fin = np.isfinite(exp)
    # (the low part of an infinite value is inf - inf)
    hi = q.cpu().numpy()
    assert np.array_equal(np.isnan(exp), np.isnan(hi)) and np.array_equal(fin, np.isfinite(hi))
    scale = np.maximum(np.abs(exp), 1e-30)
    # a pair of floats holds 48 bits; both sides round the same float64 terms
    # (of at most (4/dx^2 + 4/dy^2) g/f |h| around a point) a few times
    lim = 2.0 ** -47 * scale + 8 * 2.0 ** -53 * 9.81e4 * (4 / 5e3 ** 2 + 4 / 4e3 ** 2) * 1e3
    assert np.all(np.abs(got - exp)[fin] <= lim[fin])


@pytest.mark.parametrize("ny,nx", [(40, 66), (200, 131)])
def test_zero_backgrounds_are_skipped_exactly(ny, nx):
    B, n = 4, 3
    p, _ = plans(ny, nx)
    g = torch.Generator(device="cuda").manual_seed(2)
    h0 = 0.1 * torch.randn(B, ny, nx, generator=g, device="cuda")
    hb = torch.zeros_like(h0)
    hb[1] = 0.1 * torch.randn(ny, nx, generator=g, device="cuda")
    hb[3, ny // 2, nx // 2] = 0.05
    out = p.step(h0, hb, nstep=n)
    # the state-level calls take the fields as given, without looking at them
    traj = p.new_traj(B, n)
    tv = p.traj_view(traj, B, n)
    tv[0, 0] = h0
    qb, qlo = torch.empty_like(h0), p.new_qlo(B)
    p.init_state(tv[0, 0], hb, tv[0, 1], qb, qlo)
    p.advance(B, traj, n, 0, n, hb, qb, qlo)
    exp = torch.empty_like(h0)
    p.finalize(B, tv[n * p.nstage, 0], hb, exp)
    assert torch.equal(out, exp)
    assert torch.equal(p.step(h0, hb, nstep=n, traj=p.new_traj(B, n)), exp)
    assert torch.equal(p.step(h0, hb, nstep=0)[:, 1:-1, 1:-1], h0[:, 1:-1, 1:-1])
    # in place, and the tangent
    h = h0.clone()
    assert torch.equal(p.step(h, hb, nstep=n, out=h), exp)
    dh = torch.randn(B, ny, nx, generator=g, device="cuda")
    d = p.step_tgl(dh, h0, hb, nstep=n)
    for b in range(B):
        one = p.step_tgl(dh[b], h0[b], hb[b], nstep=n)[0]
        assert float((d[b] - one).norm() / one.norm()) < 1e-5

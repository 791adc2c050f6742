"""The reverse sweep doesn't depend on memory that nothing writes: the wall ring of a
stored state's SSH (the forward sweep writes the interior) and the workspace. Equal in
every bit whatever these hold, in both staging forms and for one and several tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("scheme", ["rk2", "rk4"])
@pytest.mark.parametrize("ny,nx", [(12, 16), (33, 48), (70, 96), (45, 131)])
def test_ring_and_workspace_contents(ny, nx, scheme, dtype):
    from vardyn_gb300.qg1l import QG1LPlan
    B, n = 2, 2
    p = QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=dtype, time_scheme=scheme)
    g = torch.Generator(device="cuda").manual_seed(ny * nx)
    rnd = lambda: torch.randn(B, ny, nx, generator=g, device="cuda", dtype=dtype)  # noqa: E731
    h, hb, adh, adq = 0.1 * rnd(), 0.01 * rnd(), rnd(), 1e3 * rnd()
    traj = torch.zeros((n * p.nstage + 1) * 2 * B * ny * nx, dtype=dtype, device="cuda")
    t0 = p.traj_view(traj, B, n)
    t0[0, 0] = h
    qb, qlo = torch.empty_like(h), torch.zeros_like(h) if dtype == torch.float32 else None
    p.init_state(t0[0, 0], hb, t0[0, 1], qb, qlo)
    p.advance(B, traj, n, 0, n, hb, qb, qlo)
    ring = torch.ones(ny, nx, dtype=torch.bool, device="cuda")
    ring[1:-1, 1:-1] = False
    res = []
    for v in (0.0, float("nan"), 1e40 if dtype == torch.float64 else 1e30):
        t = traj.clone()
        p.traj_view(t, B, n)[:, 0][..., ring] = v
        a, q = adh.clone(), adq.clone()
        ws = p.workspace(B)
        ws.view(-1)[:ws.numel() // 8 * 8].view(torch.float64).fill_(v)
        p.advance_adj(B, t, n, 0, n, a, q)
        res.append((a, q))
    for a, q in res[1:]:
        assert torch.equal(a, res[0][0]) and torch.equal(q, res[0][1])

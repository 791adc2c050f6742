"""The tensor-core inversion (forward pass with the tridiagonal solve in its
epilogue, inverse pass) in every launch shape: fields of one to eight row blocks
and beyond, rows that end at, before and behind a block, odd transform lengths,
one and two groups of modes, unaligned rows, clusters with padding, background,
boundary field and mask."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (ny, nx, batch)
CASES = [(10, 10, 1), (34, 67, 1), (35, 130, 3), (66, 258, 2), (130, 260, 1), (131, 301, 5), (258, 64, 1),
         (259, 515, 1), (200, 516, 7), (514, 100, 2), (1026, 70, 1), (1100, 90, 1), (64, 1030, 2)]


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("ny,nx,B", CASES)
def test_every_shape_solves(ny, nx, B):
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan, build_mask
    rng = np.random.default_rng(ny * nx + B)
    mask = build_mask(ny, nx, np.where(rng.random((ny, nx)) < 0.01, np.nan, 0.0))
    kw = dict(mask=mask)
    p64 = QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=torch.float64, **kw)
    p = QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=torch.float32, **kw)
    dev = lambda a: torch.as_tensor(a, dtype=torch.float32, device="cuda")  # noqa: E731
    q, qb = dev(1e-6 * rng.standard_normal((B, ny, nx))), dev(1e-6 * rng.standard_normal((B, ny, nx)))
    hb, add = dev(rng.standard_normal((B, ny, nx))), dev(1e-6 * rng.standard_normal((B, ny, nx)))
    exp = p64.pv2h(q.double(), hb.double(), qb.double()).cpu().numpy()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    spec = torch.zeros(_lib.load().vd_qg1l_spec_bytes(p.handle, B) // 4, device="cuda")
    spec64 = torch.zeros(_lib.load().vd_qg1l_spec_bytes(p64.handle, B) // 8, dtype=torch.float64, device="cuda")
    a64 = torch.empty_like(q, dtype=torch.float64)
    _lib.call("vd_qg1l_dst_x", p64.handle, B, ptr(q.double()), ptr(spec64), 0, None, st)
    _lib.call("vd_qg1l_dst_x", p64.handle, B, ptr(add.double()), ptr(spec64), 2, ptr(a64), st)
    flag = ctypes.c_int(0)
    for grp in (0, 1, 2, 4, 8):
        p.set_schedule(tc_group_fwd=grp, tc_group_inv=grp)
        h = p.pv2h(q, hb, qb).cpu().numpy()
        # 3xTF32 with fp32 accumulation, two transforms and the solve: 5e-6 at
        # the largest lengths for smooth fields; white noise keeps the bound
        assert rel(h, exp) < 1e-5, grp
        # the pass alone and its adjoint epilogue (interior; the ring is not written)
        out = torch.full_like(q, 7.0)
        _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(q), ptr(spec), 0, None, st)
        _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(add), ptr(spec), 2, ptr(out), st)
        o = out.cpu().numpy()
        e = a64.cpu().numpy()[:, 1:-1, 1:-1]
        assert rel(o[:, 1:-1, 1:-1], e) < 1e-5, grp
        assert np.all(o[:, 1:-1, 1:-1][:, mask[1:-1, 1:-1] != 3] == 0)
        assert np.all(o[:, 0] == 7.0) and np.all(o[:, -1] == 7.0)
        assert np.all(o[:, :, 0] == 7.0) and np.all(o[:, :, -1] == 7.0)
        _lib.call("vd_device_error", ctypes.byref(flag), 1)
        assert flag.value == 0


def test_unaligned_fields_match_aligned():
    """Fields that start 4 bytes into an allocation take the scalar stores."""
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan
    ny, nx, B = 70, 132, 2
    p = QG1LPlan(ny, nx, 5e3, 5e3, 900.0, 1e-4, 2.7, dtype=torch.float32)
    g = torch.Generator(device="cuda").manual_seed(1)
    q, hb = (torch.randn(B, ny, nx, generator=g, device="cuda") for _ in range(2))
    ref = torch.zeros_like(q)
    shifted = [torch.zeros(q.numel() + 1, device="cuda")[1:].view(B, ny, nx) for _ in range(3)]
    shifted[0].copy_(q)
    shifted[1].copy_(hb)
    ws = p.workspace(B)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.call("vd_qg1l_pv2h", p.handle, B, ptr(q), ptr(hb), None, ptr(ref), ptr(ws), ws.numel(), st)
    _lib.call("vd_qg1l_pv2h", p.handle, B, ptr(shifted[0]), ptr(shifted[1]), None, ptr(shifted[2]), ptr(ws),
              ws.numel(), st)
    assert torch.equal(ref, shifted[2])

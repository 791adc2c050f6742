"""The float64 x-direction DST-I pass at lengths of every form: dense products
(one, two and several column groups, 1, 2 and 4 rows a warp), direct odd
radices as first and as later stages, with odd row counts and batches."""
import ctypes

import numpy as np
import pytest
import scipy.fft
import torch

pytestmark = pytest.mark.gpu

# (ny, nx, batch): nx - 1 = 127, 61, 29 and 383 prime; 63 = 3^2 7, 77 = 7 11,
# 255 = 3 5 17, 511 = 7 73, 343 = 7^3, 1023 = 3 11 31, 26 = 2 13
CASES = [(9, 30, 1), (130, 62, 1), (9, 128, 1), (128, 128, 1), (130, 128, 9), (66, 384, 1), (200, 384, 8),
         (34, 64, 1), (33, 78, 2), (258, 256, 1), (37, 512, 3), (20, 344, 1), (19, 1024, 1), (12, 27, 1)]


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("ny,nx,B", CASES)
def test_f64_dst_passes(ny, nx, B):
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan, build_mask
    rng = np.random.default_rng(ny * nx + B)
    land = np.where(rng.random((ny, nx)) < 0.02, np.nan, 0.0)
    p = QG1LPlan(ny, nx, 5e3, 5e3, 900.0, 1e-4, 2.7, dtype=torch.float64, mask=build_mask(ny, nx, land))
    n, st = nx - 2, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    f = torch.as_tensor(rng.standard_normal((B, ny, nx)), device="cuda")
    spec = torch.zeros(_lib.load().vd_qg1l_spec_bytes(p.handle, B) // 8, dtype=torch.float64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def rel(a, b):
        return np.linalg.norm(a - b) / np.linalg.norm(b)

    x = f.cpu().numpy()
    _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(f), ptr(spec), 0, None, st)
    y = scipy.fft.dst(x[:, 1:-1, 1:-1], type=1, norm="ortho", axis=-1)
    exp = np.concatenate([y[..., 0::2], y[..., 1::2]], axis=-1)
    got = spec.view(B, ny - 2, -1)[..., :n].cpu().numpy()
    # sums of n terms of unit size: n eps relative at most
    assert rel(got, exp) < 1e-12
    out = torch.full_like(f, 7.0)
    _lib.call("vd_qg1l_dst_x", p.handle, B, None, ptr(spec), 1, ptr(out), st)
    assert rel(out.cpu().numpy()[:, 1:-1, 1:-1], x[:, 1:-1, 1:-1]) < 1e-12
    add = torch.as_tensor(rng.standard_normal((B, ny, nx)), device="cuda")
    _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(add), ptr(spec), 2, ptr(out), st)
    ref = np.where(p.mask == 3, x + add.cpu().numpy(), 0.0)[:, 1:-1, 1:-1]
    assert rel(out.cpu().numpy()[:, 1:-1, 1:-1], ref) < 1e-12
    # the pass with a background field subtracted, through the whole solve
    hb = torch.as_tensor(rng.standard_normal((B, ny, nx)), device="cuda")
    q, qb = 1e-6 * f, 1e-6 * add
    h = p.pv2h(q, hb, qb)
    h2 = p.pv2h(q - qb, hb, torch.zeros_like(qb))
    assert rel(h.cpu().numpy(), h2.cpu().numpy()) < 1e-12

"""The float64 FFT form of the x-direction DST-I over half stages: lengths of radix 4,
2, 3 and 5 alone, with odd and even numbers of rows left at the last stages, and after
a direct odd radix; both directions against scipy, at the bound of the other lengths'
test (sums of n terms of unit size: n eps relative at most)."""
import ctypes

import numpy as np
import pytest
import scipy.fft
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


# nx - 1 = 8, 9, 15, 16, 45, 60, 64, 81, 96, 125, 512 and 17 * 8, 17 * 45
@pytest.mark.parametrize("nx", [9, 10, 16, 17, 46, 61, 65, 82, 97, 126, 513, 137, 766])
def test_passes(nx):
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan
    ny, B, n = 12, 3, nx - 2
    rng = np.random.default_rng(nx)
    p = QG1LPlan(ny, nx, 5e3, 5e3, 900.0, 1e-4, 2.7, dtype=torch.float64)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    f = torch.as_tensor(rng.standard_normal((B, ny, nx)), device="cuda")
    spec = torch.zeros(_lib.load().vd_qg1l_spec_bytes(p.handle, B) // 8, dtype=torch.float64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    x = f.cpu().numpy()[:, 1:-1, 1:-1]
    _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(f), ptr(spec), 0, None, st)
    y = scipy.fft.dst(x, type=1, norm="ortho", axis=-1)
    exp = np.concatenate([y[..., 0::2], y[..., 1::2]], axis=-1)
    got = spec.view(B, ny - 2, -1)[..., :n].cpu().numpy()
    assert np.linalg.norm(got - exp) < 1e-12 * np.linalg.norm(exp)
    out = torch.full_like(f, 7.0)
    _lib.call("vd_qg1l_dst_x", p.handle, B, None, ptr(spec), 1, ptr(out), st)
    back = out.cpu().numpy()[:, 1:-1, 1:-1]
    assert np.linalg.norm(back - x) < 1e-12 * np.linalg.norm(x)

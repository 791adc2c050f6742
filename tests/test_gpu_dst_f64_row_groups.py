"""The float64 dense x-transform of few rows: one row a CTA (up to 152 CTAs) and the
next count above, with half lengths of every remainder of 8 (the prefetched loop's tail
of 4, 2 and 1), forward and inverse against scipy at the other lengths' 1e-12."""
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


# nx - 1 prime (dense form), or the length too short for the FFT to pay
@pytest.mark.parametrize("ny,nx,B", [(8, 30, 1), (10, 32, 1), (12, 38, 2), (9, 42, 1), (78, 44, 1), (79, 44, 2),
                                     (153, 54, 1), (154, 60, 1), (155, 62, 1), (40, 68, 2), (78, 72, 2), (79, 74, 2),
                                     (80, 80, 2), (40, 104, 1), (153, 128, 1), (155, 132, 1)])
def test_passes(ny, nx, B):
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan
    n = nx - 2
    rng = np.random.default_rng(nx + ny)
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

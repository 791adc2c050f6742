"""The float64 x-transform at lengths that have an FFT, on both sides of the row count
up to which the dense form runs (152 one-row blocks, by column groups of 64) and of the
length up to which it does (120 half modes): forward and inverse against scipy at the
other lengths' 1e-12, and the two forms of one length against each other."""
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


def passes(p, x):
    from vardyn_gb300 import _lib
    B, ny, nx = x.shape
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    spec = torch.zeros(_lib.load().vd_qg1l_spec_bytes(p.handle, B) // 8, dtype=torch.float64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.call("vd_qg1l_dst_x", p.handle, B, ptr(x), ptr(spec), 0, None, st)
    s = spec.view(B, ny - 2, -1)[..., :nx - 2].cpu().numpy()
    out = torch.full_like(x, 7.0)
    _lib.call("vd_qg1l_dst_x", p.handle, B, None, ptr(spec), 1, ptr(out), st)
    return s, out.cpu().numpy()[:, 1:-1, 1:-1]


# nx - 1 = 9, 16, 45, 60, 64, 96, 125, 128, 240, 250: rows 152 or 76 a field, then twice
@pytest.mark.parametrize("nx,ny", [(10, 154), (17, 154), (46, 154), (61, 154), (65, 154), (97, 154), (126, 154),
                                   (129, 154), (241, 78), (251, 78)])
def test_both_sides(nx, ny):
    from vardyn_gb300.qg1l import QG1LPlan
    rng = np.random.default_rng(nx)
    p = QG1LPlan(ny, nx, 5e3, 5e3, 900.0, 1e-4, 2.7, dtype=torch.float64)
    x = torch.as_tensor(rng.standard_normal((2, ny, nx)), device="cuda")
    xi = x.cpu().numpy()[:, 1:-1, 1:-1]
    y = scipy.fft.dst(xi, type=1, norm="ortho", axis=-1)
    exp = np.concatenate([y[..., 0::2], y[..., 1::2]], axis=-1)
    few, many = passes(p, x[:1].contiguous()), passes(p, x)
    for b, (s, back) in ((1, few), (2, many)):
        assert np.linalg.norm(s - exp[:b]) < 1e-12 * np.linalg.norm(exp[:b])
        assert np.linalg.norm(back - xi[:b]) < 1e-12 * np.linalg.norm(xi[:b])
    assert np.linalg.norm(few[0][0] - many[0][0]) < 1e-12 * np.linalg.norm(exp[0])

"""The float64 dense x-transform of more row tiles than a launch has blocks in y: each of
its column layouts just above 65535 tiles. A row's sums don't depend on the batch: the
first and the last field give what they give alone, to rounding (1e-13)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


# (ny, nx, fields): transforms of 42, 66 and 138 (n + 1 = 43, 67, 139: prime, dense),
# tiles of 16, 8 and 4 rows
@pytest.mark.parametrize("ny,nx,B", [(1026, 44, 1025), (1026, 68, 513), (260, 140, 1017)])
def test_pass_over_many_rows(ny, nx, B):
    from vardyn_gb300 import _lib
    from vardyn_gb300.qg1l import QG1LPlan
    p = QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=torch.float64)
    g = torch.Generator(device="cuda").manual_seed(ny + nx)
    x = torch.randn(B, ny, nx, generator=g, device="cuda", dtype=torch.float64)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    size = lambda n: _lib.load().vd_qg1l_spec_bytes(p.handle, n) // 8  # noqa: E731

    def passes(f):
        """Spectra and their inverse transform (the transform is its own inverse)."""
        n = f.shape[0]
        spec, out = torch.zeros(size(n), dtype=torch.float64, device="cuda"), torch.zeros_like(f)
        _lib.call("vd_qg1l_dst_x", p.handle, n, ptr(f), ptr(spec), 0, None, st)
        _lib.call("vd_qg1l_dst_x", p.handle, n, None, ptr(spec), 1, ptr(out), st)
        return spec.view(n, -1), out

    spec, out = passes(x)
    for k in (0, B - 1):
        s1, o1 = passes(x[k:k + 1].contiguous())
        assert float((spec[k] - s1[0]).norm() / s1.norm()) < 1e-13
        assert float((out[k] - o1[0]).norm() / o1.norm()) < 1e-13
    inner = x[:, 1:-1, 1:-1]
    assert float((out[:, 1:-1, 1:-1] - inner).norm() / inner.norm()) < 1e-13

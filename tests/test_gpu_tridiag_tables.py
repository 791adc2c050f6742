"""The float64 tridiagonal kernel with tables against the general one (another piece
length, through the schedule) at heights around its pieces, warps and its tallest
field, with several fields, and with values that are not finite. Both solve the same
recurrences with pieces joined at other rows: a few roundings, 1e-13 of the largest."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


# interior rows 6, 7, 8, 9, 31, 32, 33, 64, 130, 511, 512, 513
@pytest.mark.parametrize("ny,nx,B", [(8, 20, 1), (9, 27, 2), (10, 40, 1), (11, 33, 3), (33, 18, 1), (34, 20, 2),
                                     (35, 47, 1), (66, 64, 4), (132, 30, 2), (513, 24, 1), (514, 41, 2), (515, 24, 1)])
def test_equals_general_kernel(ny, nx, B):
    from vardyn_gb300.qg1l import QG1LPlan
    rng = np.random.default_rng(ny + nx)
    p = QG1LPlan(ny, nx, 5e3, 4e3, 900.0, 1e-4, 2.7, dtype=torch.float64)
    q = torch.as_tensor(1e-6 * rng.standard_normal((B, ny, nx)), device="cuda")
    z = torch.zeros_like(q)
    got = p.pv2h(q, z, z)
    p.set_schedule(tridiag_rows=32)
    want = p.pv2h(q, z, z)
    assert float((got - want).abs().max()) <= 1e-13 * float(want.abs().max())
    q[0, ny // 2, nx // 2] = np.nan
    bad = p.pv2h(q, z, z)
    p.set_schedule(tridiag_rows=0)
    assert torch.equal(torch.isnan(p.pv2h(q, z, z)), torch.isnan(bad))

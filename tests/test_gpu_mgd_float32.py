"""The float32 masked Dirichlet solve against the float64 one: the operator that the
iteration applies keeps the small eigenvalues of the smoothest modes, also where
lambda is 0 or far below the diagonal's rounding and the spacings are unequal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# The float32 iteration stops at 1e-6, which between coasts leaves a few times that in
# the solution (the float64 iteration's own stopping error); c0, c1 and lambda rounded
# to float32 move it by 1e-7, the float32 updates of x and r by up to 5e-6.
TOL, BOUND = 1e-6, 1e-5


@pytest.fixture(scope="module", autouse=True)
def built():
    from vardyn_gb300 import build
    build.build()


@pytest.mark.parametrize("land", [0.0, 0.1])
@pytest.mark.parametrize("n0,n1,d0,d1", [(511, 767, 9.1e3, 6.9e3), (1023, 767, 9.1e3, 6.9e3), (511, 767, 5e3, 5e3),
                                         (1023, 767, 5e3, 5e3), (127, 255, 3e3, 1.1e4)])
def test_float32_solution_is_the_float64_one(n0, n1, d0, d1, land):
    from vardyn_gb300.helmholtz_mg import MaskedDirichletMG
    rng = np.random.default_rng(n0 + n1)
    k = np.fft.fftfreq(n0)[:, None] ** 2 + np.fft.fftfreq(n1)[None, :] ** 2
    w = np.real(np.fft.ifft2(np.exp(-k / 0.0005) * np.fft.fft2(rng.standard_normal((n0, n1)))))
    mask = (w <= np.quantile(w, 1 - land)).astype(float)
    lam = np.array([0.0, 2.6e-13, 1.1e-9])
    b = torch.as_tensor(rng.standard_normal((3, 1, n0, n1)), device="cuda")
    ref = MaskedDirichletMG(n0, n1, d0, d1, lam, mask=mask, tol=1e-11, max_cycles=60)
    mg = MaskedDirichletMG(n0, n1, d0, d1, lam, mask=mask, dtype=torch.float32, tol=TOL, max_cycles=60)
    b32 = b.float()
    e = ref.solve(b32.double())
    u = mg.solve(b32).double()
    assert bool((mg.rel <= TOL).all())
    err = (u - e).flatten(1).norm(dim=1) / e.flatten(1).norm(dim=1)
    assert float(err.max()) <= BOUND, err

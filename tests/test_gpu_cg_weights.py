"""CG with Jacobi weights that are not positive numbers: the same outcome resident and streaming (the
scaled streaming form, from which the weight cancels, is for positive ones)."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import csr_solve
from test_gpu_resident_cg import seven_point

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(13, 11, 12), (80, 80, 101)])
@pytest.mark.parametrize("omega,want", [(0.0, 2), (float("nan"), 4), (float("inf"), 4), (-1.3, 0), (1e-30, 0)])
def test_weights(shape, omega, want):
    rp, c, v, x, b = seven_point(*shape, seed=8)
    y, it, res, status = csr_solve(rp, c, v, b, method="CG", maxit=1000, eps=1e-10, omega=omega)
    assert status == want
    if want == 2:  # z = 0: no direction
        assert it == 1 and res == 1.0 and not y.any()
    if want == 0:  # cond(A) <= 100
        assert res < 1e-10 and np.linalg.norm(y - x) <= 100 * 1e-10 * np.linalg.norm(x)

"""Mixed BiCGSTAB of one system beyond the shared memory that holds its FP32 matrix (from 520,000 rows
of 7 entries), odd sizes, and its neighbour on chip: the reported residual is the true one."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import csr_solve, csr_spmv
from test_gpu_mixed_bicgstab import _convection_diffusion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(80, 80, 80), (84, 84, 84), (101, 99, 103), (160, 160, 163)])
@pytest.mark.parametrize("precond", ["Jacobi", "none"])
def test_large_systems(shape, precond):
    rp, cl, vl, b = _convection_diffusion(*shape, 4.0, seed=3)
    eps = 1e-10
    x, it, res, status = csr_solve(rp, cl, vl, b, method="BiCGSTAB-mixed", precond=precond, maxit=5000, eps=eps)
    assert status == 0 and res < eps
    r = b - csr_spmv(rp, cl, vl, x)
    true = np.linalg.norm(r) / np.linalg.norm(b)
    assert true < eps and abs(true - res) <= 1e-3 * res + 1e-18
    y, it2, res2, _ = csr_solve(rp, cl, vl, b, method="BiCGSTAB-mixed", precond=precond, maxit=5000, eps=eps)
    assert it2 == it and res2 == res and np.array_equal(x, y)  # runs are bit-identical

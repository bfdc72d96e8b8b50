"""BiCGSTAB, FP64 and mixed, on long rows: just below and above 64 entries on average (from where the
kernels for wide rows run), 24 in FP64 beyond shared memory, rows of a number of entries that no
group divides, and one long row among short ones.

b = A x*, cond(A) <= 100 (see test_gpu_cg_wide_rows), so ||x - x*|| <= 100 eps ||x*||.
"""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import csr_bicgstab3, csr_solve
from test_gpu_cg_wide_rows import banded

pytestmark = pytest.mark.gpu
EPS = 1e-10


@pytest.mark.parametrize("n,couplings,wide", [(300, 31, 0), (300, 32, 0), (301, 99, 0), (3001, 33, 0), (20003, 37, 0),
                                              (90013, 11, 0), (90013, 12, 0), (120007, 35, 0), (5000, 3, 900)])
def test_long_rows(n, couplings, wide):
    rp, c, v, _, x, b = banded(n, range(1, couplings + 1), 5, wide)
    for method in ("BiCGSTAB", "BiCGSTAB-mixed"):
        y, it, res, status = csr_solve(rp, c, v, b, method=method, maxit=1000, eps=EPS)
        assert status == 0 and res < EPS and it > 0, method
        assert np.linalg.norm(y - x) <= 100 * EPS * np.linalg.norm(x), method
        r = b - np.add.reduceat(v * y[c], rp[:-1])
        assert np.linalg.norm(r) <= 2 * EPS * np.linalg.norm(b), method
    z, its, _, status, _ = csr_bicgstab3(rp, c, v, [b, x, -b], maxit=1000, eps=EPS)
    one = [csr_solve(rp, c, v, t, method="BiCGSTAB", maxit=1000, eps=EPS) for t in (b, x, -b)]
    assert status == [0, 0, 0] and its == [o[1] for o in one]
    assert all(np.array_equal(z[k], one[k][0]) for k in range(3))  # three together as one after another

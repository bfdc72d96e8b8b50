"""The stopping test ||r|| / ||b|| < eps of FP64 BiCGSTAB and the allocation-free CG where eps^2 ||b||^2
is no normal number, and with an eps that nothing is below.

b = A x*, cond(A) <= 100 (see test_gpu_resident_cg), so ||x - x*|| <= 100 eps ||x*||.
"""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import csr_bicgstab3, csr_solve
from test_gpu_cg_small_numbers import noalloc
from test_gpu_resident_cg import seven_point

pytestmark = pytest.mark.gpu


def bicgstab(rp, c, v, b, maxit, eps, x0=None):
    return csr_solve(rp, c, v, b, x0, method="BiCGSTAB", maxit=maxit, eps=eps)


def bicgstab3(rp, c, v, b, maxit, eps, x0=None):
    """The first of three right-hand sides solved together: b, 2 b, -b."""
    x, it, res, status, _ = csr_bicgstab3(rp, c, v, [b, 2.0 * b, -b], None if x0 is None else [x0, 2.0 * x0, -x0],
                                      maxit=maxit, eps=eps)
    assert status == [status[0]] * 3
    return x[0], it[0], res[0], status[0]


FORMS = {
    "BiCGSTAB": (bicgstab, (13, 11, 12)),
    "BiCGSTAB, matrix streamed": (bicgstab, (80, 80, 101)),
    "three BiCGSTAB": (bicgstab3, (13, 11, 12)),
    "CG, cluster": (noalloc, (13, 11, 12)),
    "CG, whole GPU": (noalloc, (23, 21, 20)),
}


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("scale", [-510, -500, 0, 490])
def test_scaled_right_hand_sides(form, scale):
    solve, shape = FORMS[form]
    rp, c, v, x, b = seven_point(*shape, seed=6)
    f = 2.0 ** scale
    y, it, res, status = solve(rp, c, v, b * f, 1000, 1e-8)
    assert status == 0 and res < 1e-8 and 0 < it < 1000
    assert np.linalg.norm(y / f - x) <= 100 * 1e-8 * np.linalg.norm(x)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("scale,eps", [(0, 1e-8), (0, 1e-170), (-520, 1e-8), (-530, 1e-30)])
def test_started_at_the_solution(form, scale, eps):
    """Whole numbers times a power of two: the residual of x0 = x* is exactly 0, below any eps."""
    solve, shape = FORMS[form]
    rp, c, v, x, _ = seven_point(*shape, seed=6)
    v, x = np.round(8 * v), np.round(8 * x) * 2.0 ** scale
    b = np.add.reduceat(v * x[c], rp[:-1])
    y, it, res, status = solve(rp, c, v, b, 10, eps, x)
    assert status == 0 and it == 0 and res == 0 and np.array_equal(y, x)
    y, it, res, status = solve(rp, c, v, np.zeros_like(b), 10, eps)
    assert status == 0 and it == 0 and res == 0 and not y.any()


@pytest.mark.parametrize("form", [f for f in FORMS if f != "three BiCGSTAB"])  # which takes eps > 0 only
@pytest.mark.parametrize("eps,want", [(-1.0, 1), (float("nan"), 1), (float("inf"), 0)])
def test_any_eps(form, eps, want):
    solve, shape = FORMS[form]
    rp, c, v, x, b = seven_point(*shape, seed=6)
    _, it, res, status = solve(rp, c, v, b, 5, eps)
    assert status == want and it == (5 if want else 0) and np.isfinite(res)

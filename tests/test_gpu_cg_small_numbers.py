"""CG in every form where the scalars of the recurrence become tiny: a fixed number of iterations
(eps 0), which goes on until r.z underflows, and right-hand sides scaled down to where it is below
2^-1021 before the solve has converged, so that its reciprocal is infinite.

b = A x* for a 7-point operator whose diagonal exceeds its row's off-diagonal sum by 10 %:
cond(A) <= 100, so ||x - x*|| <= 100 (eps + n-term rounding, below 1e-13) ||x*||.  Scaled by 2^-500,
r stops at 2^-537, where its squares underflow: relative to b 2^-37, 1e-11.
"""
import ctypes as C

import numpy as np
import pytest

from sysu_cfd_heat_gb300._lib import LIB_PATH
from sysu_cfd_heat_gb300.solver import csr_solve
from test_gpu_resident_cg import seven_point

pytestmark = pytest.mark.gpu


def noalloc(rp, c, v, b, maxit, eps, x0=None, omega=1.3):
    torch = pytest.importorskip("torch")
    f = C.CDLL(LIB_PATH).sysu_csr_cg_noalloc
    f.argtypes = [C.c_int] + [C.c_void_p] * 5 + [C.c_int, C.c_double, C.c_double] + [C.c_void_p] * 4
    d = [torch.from_numpy(t).cuda() for t in (rp, c, v, b)]
    x = torch.from_numpy(np.zeros(len(b)) if x0 is None else x0.copy()).cuda()
    torch.cuda.synchronize()
    it, res, st = C.c_int(), C.c_double(), C.c_int()
    assert f(len(b), *(t.data_ptr() for t in d), x.data_ptr(), maxit, eps, omega, None, C.addressof(it),
             C.addressof(res), C.addressof(st)) == 0
    return x.cpu().numpy(), it.value, res.value, st.value


FORMS = {
    "resident": ("CG", (13, 11, 12)),
    "streaming": ("CG", (80, 80, 101)),
    "resident mixed": ("CG-mixed", (13, 11, 12)),
    "streaming mixed": ("CG-mixed", (80, 80, 101)),
    "device, cluster": (noalloc, (13, 11, 12)),
    "device, whole GPU": (noalloc, (23, 21, 20)),
}


def run(form, scale, maxit, eps):
    method, shape = FORMS[form]
    rp, c, v, x, b = seven_point(*shape, seed=6)
    f = 2.0 ** scale
    if method is noalloc:
        got = noalloc(rp, c, v, b * f, maxit, eps)
    else:
        got = csr_solve(rp, c, v, b * f, method=method, maxit=maxit, eps=eps, omega=1.3)
    if not np.isfinite(np.dot(b * f, b * f)):  # 646,400 rows scaled by 2^500
        assert got[1:] == (0, got[2], 4) and not np.isfinite(got[2])
        pytest.skip("||b||^2 is beyond FP64's range: reported as not finite")
    y = got[0] / f
    return np.linalg.norm(y - x) / np.linalg.norm(x), *got[1:]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("scale,tol", [(0, 1e-11), (-480, 1e-11), (-500, 1e-8)])
def test_fixed_number_of_iterations(form, scale, tol):
    err, it, res, _ = run(form, scale, 2000, 0.0)
    # the mixed forms count the iterations of the FP64 solve that takes over from them as well
    assert err <= tol and np.isfinite(res) and it <= (4000 if "mixed" in form else 2000)


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("scale", [-480, -490, -500, 480, 500])
def test_scaled_right_hand_sides(form, scale):
    err, it, res, status = run(form, scale, 1000, 1e-8)
    assert status == 0 and res < 1e-8 and err <= 100 * 1e-8

"""FP64 BiCGSTAB with the matrix in shared memory and the vectors in registers against the general
form (which the three-matrix solve runs): the same sums in the same order, so the same bits.  Row
counts at the edges of one to four rows a thread and of two blocks a CTA, one and three right-hand
sides, and a row too wide for the resident form."""
import ctypes as C

import numpy as np
import pytest

from sysu_cfd_heat_gb300 import _lib
from sysu_cfd_heat_gb300.solver import csr_bicgstab3, csr_solve

pytestmark = pytest.mark.gpu


def _system(n, wide, rng):
    lo, up = -rng.uniform(0.5, 1.5, n), -rng.uniform(0.2, 0.8, n)
    rows = [[i] + [j for j in (i - 1, i + 1) if 0 <= j < n] for i in range(n)]
    vals = [[3.0] + [lo[i] if j < i else up[i] for j in rows[i][1:]] for i in range(n)]
    if wide:
        rows[n // 2] = [n // 2] + [j for j in range(n) if j != n // 2]
        vals[n // 2] = [2.0 * n] + list(rng.uniform(-1.0, 1.0, n - 1))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    return rp, np.concatenate(rows), np.concatenate(vals)


def _general(rp, cl, vl, B, maxit, eps):
    """The same matrix three times through the three-matrix solve."""
    dp, ip = C.POINTER(C.c_double), C.POINTER(C.c_int)
    f = _lib.lib().sysu_csr_bicgstab_batched3
    f.argtypes = [C.c_int, ip, ip, C.POINTER(dp), C.POINTER(dp), C.POINTER(dp), C.c_int, C.c_double, ip, dp, ip]
    rp, cl = np.ascontiguousarray(rp, np.int32), np.ascontiguousarray(cl, np.int32)
    X = np.zeros_like(B)
    it, res, status = (C.c_int * 3)(), (C.c_double * 3)(), (C.c_int * 3)()
    p3 = dp * 3
    at = lambda a: a.ctypes.data_as(dp)  # noqa: E731
    code = f(B.shape[1], rp.ctypes.data_as(ip), cl.ctypes.data_as(ip), p3(*[at(vl)] * 3), p3(*[at(b) for b in B]),
             p3(*[at(x) for x in X]), maxit, eps, it, res, status)
    assert code == 0 and list(status) == [0, 0, 0]
    return X, list(it)


@pytest.mark.parametrize("n,wide", [(1, 0), (33, 0), (257, 0), (38912, 0), (38913, 0), (77825, 0), (155648, 0),
                                    (155649, 0), (311297, 0), (400, 1)])
def test_same_bits_as_the_general_form(n, wide):
    rng = np.random.default_rng(n)
    rp, cl, vl = _system(n, wide, rng)
    B = rng.standard_normal((3, n))
    ref = _general(rp, cl, vl, B, 200, 1e-10)
    three = csr_bicgstab3(rp, cl, vl, B, maxit=200, eps=1e-10)
    for c in range(3):
        x, it, _, status = csr_solve(rp, cl, vl, B[c], method="BiCGSTAB", maxit=200, eps=1e-10)
        assert status == 0
        assert it == ref[1][c] == three[1][c]
        assert np.array_equal(x, ref[0][c])
        assert np.array_equal(x, three[0][c])

"""Streaming CG kernels on rows so wide that a tile holds fewer slices than there are consumer
warps (FP64: 9 of 19 from 16 entries a row, 4 from 31; FP32: 11 of 23 from 19, 5 from 38), one slice
a tile, and rows too wide for a slot; sizes beyond the shared memory of the resident kernels.

b = A x* for a matrix whose diagonal exceeds its row's off-diagonal sum by 10 %, so
||x - x*|| <= cond(A) eps ||x*|| with cond(A) <= 21 max(d) / min(d) <= 100.
"""
import numpy as np
import pytest

from oracle.simple_np import cg as oracle_cg
from sysu_cfd_heat_gb300.solver import csr_solve

pytestmark = pytest.mark.gpu
EPS = 1e-10


def banded(n, offsets, seed, wide=0):
    """Symmetric couplings at the given distances on a ring of n rows (so that all rows are equally
    long); wide: row n // 3 is coupled to that many more, far from it."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    rows, cols, vals = [], [], []
    for o in offsets:
        w = -rng.uniform(0.8, 1.2, n)
        j = (i + o) % n
        rows += [i, j]
        cols += [j, i]
        vals += [w, w]
    if wide:
        far = n // 2 + np.arange(wide)
        w = -rng.uniform(0.8, 1.2, wide) / wide
        rows += [np.full(wide, n // 3), far]
        cols += [far, np.full(wide, n // 3)]
        vals += [w, w]
    r, c, v = (np.concatenate(a) for a in (rows, cols, vals))
    diag = 1.1 * np.bincount(r, -v, n)
    r, c, v = np.concatenate([i, r]), np.concatenate([i, c]), np.concatenate([diag, v])
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order].astype(np.int32), v[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    x = rng.standard_normal(n)
    return rp, c, v, diag, x, np.add.reduceat(v * x[c], rp[:-1])


NEAR = [1, 2, 3, 31, 32, 33, 700, 1500, 9001, 20011, 41, 43, 47, 53, 59, 61, 67, 71, 73]
SYSTEMS = {
    "15 a row": (200013, NEAR[:7], 0),       # the widest rows of a full FP64 tile
    "17 a row": (200013, NEAR[:8], 0),
    "21 a row": (200013, NEAR[:10], 0),
    "39 a row": (200013, NEAR, 0),
    "one of 260": (200013, NEAR[:3], 250),   # one slice a tile
    "one of 900": (70001, NEAR[:3], 893),    # no slot holds it
}


@pytest.mark.parametrize("system", SYSTEMS)
@pytest.mark.parametrize("method,precond", [("CG", "Jacobi"), ("CG", "none"), ("CG-mixed", "Jacobi")])
def test_wide_rows(system, method, precond):
    """Jacobi: the scaled form; no preconditioner: the form with M^-1."""
    n, offsets, wide = SYSTEMS[system]
    rp, c, v, _, x, b = banded(n, offsets, 3, wide)
    y, it, res, status = csr_solve(rp, c, v, b, method=method, precond=precond, maxit=1000, eps=EPS, omega=1.3)
    assert status == 0 and res < EPS and it > 0
    assert np.linalg.norm(y - x) <= 100 * EPS * np.linalg.norm(x)
    r = b - np.add.reduceat(v * y[c], rp[:-1])
    assert np.linalg.norm(r) <= 2 * EPS * np.linalg.norm(b)
    z, it2, res2, _ = csr_solve(rp, c, v, b, method=method, precond=precond, maxit=1000, eps=EPS, omega=1.3)
    assert it2 == it and res2 == res and np.array_equal(y, z)  # runs are bit-identical


@pytest.mark.parametrize("system", ["15 a row", "17 a row", "39 a row", "one of 900"])
@pytest.mark.parametrize("method,tol", [("CG", 1e-11), ("CG-mixed", 1e-5)])
@pytest.mark.parametrize("sign", ["one", "mixed"])
def test_wide_rows_first_iterates(system, method, tol, sign):
    """Three iterations against the oracle's; sign mixed: one diagonal entry is of the other sign, so
    the form with M^-1 runs behind the scaled one.  tol: rounding of three steps in the precision of
    the recurrences (2^-53 and 2^-24 times some 100)."""
    n, offsets, wide = SYSTEMS[system]
    rp, c, v, d, x, b = banded(n, offsets, 4, wide)
    if sign == "mixed":
        at = rp[n // 2] + int(np.where(c[rp[n // 2]:rp[n // 2 + 1]] == n // 2)[0][0])
        v[at] = -v[at]
        d = d.copy()
        d[n // 2] = -d[n // 2]
    want, _, want_res = oracle_cg((rp, c, v, d), b, np.zeros(n), 3, EPS, 1.3)
    y, it, res, status = csr_solve(rp, c, v, b, method=method, maxit=3, eps=EPS, omega=1.3)
    assert it == 3 and status == 1
    assert np.linalg.norm(y - want) <= tol * np.linalg.norm(want)
    assert abs(res - want_res) <= 10 * tol * want_res

"""A host CSR matrix laid out on the device (csr_device.cu): every form of row list that the calls
take gives the product and the solution that the plain row lists give."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import SysuError, csr_solve, csr_spmv

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _rows(n, form, rng):
    """Row lists (columns, values) of one of the accepted forms."""
    out = []
    for i in range(n):
        c = rng.permutation(n)[:rng.integers(0, min(n, 9) + 1)]
        c = c[c != i]
        if form == "empty" and i % 3 == 0:
            c = c[:0]
        if form not in ("no diagonal", "empty"):
            c = np.insert(c, rng.integers(0, len(c) + 1), i)
        if form == "repeated":
            c = np.concatenate([c, [i], c[:1]])
        out.append((c, rng.standard_normal(len(c))))
    if form == "one long row":
        out[n // 2] = (np.arange(n), rng.standard_normal(n))
    return out


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 1000])
@pytest.mark.parametrize("form", ["sorted", "no diagonal", "repeated", "empty", "one long row", "offset", "backwards"])
def test_row_lists(n, form):
    rng = np.random.default_rng(n)
    rows = _rows(n, form, rng)
    if form == "sorted":
        rows = [(c[np.argsort(c)], v) for c, v in rows]
    rp = np.concatenate([[0], np.cumsum([len(c) for c, _ in rows])])
    cl = np.concatenate([c for c, _ in rows]).astype(np.int64)
    vl = np.concatenate([v for _, v in rows])
    if form == "offset":  # the lists begin behind the arrays' start
        rp, cl, vl = rp + 3, np.concatenate([[-7, n + 9, 0], cl]), np.concatenate([[np.nan] * 3, vl])
    if form == "backwards" and n > 2:  # a row that ends before it begins is empty
        rp[1] = rp[2] + min(2, rp[-1] - rp[2])
    x = rng.standard_normal(n)
    y = np.array([np.dot(vl[rp[i]:max(rp[i], rp[i + 1])], x[cl[rp[i]:max(rp[i], rp[i + 1])]]) for i in range(n)])
    size = np.array([np.abs(vl[rp[i]:max(rp[i], rp[i + 1])] * x[cl[rp[i]:max(rp[i], rp[i + 1])]]).sum()
                     for i in range(n)])
    count = np.array([max(0, rp[i + 1] - rp[i]) + 2 for i in range(n)])
    got = csr_spmv(rp, cl, vl, x)
    assert np.all(np.abs(got - y) <= 2 * count * EPS * size)


@pytest.mark.parametrize("column", [-1, 40, 2 ** 31 - 1])
def test_column_out_of_range(column):
    rp, cl = np.arange(41) * 2, np.repeat(np.arange(40), 2)
    cl[37] = column
    with pytest.raises(SysuError, match="out of range"):
        csr_spmv(rp, cl, np.ones(80), np.ones(40))


@pytest.mark.parametrize("method", ["CG", "BiCGSTAB", "CG-mixed", "BiCGSTAB-mixed", "GMRES"])
def test_solves_with_unsorted_rows(method):
    """Shuffled row lists, the diagonal anywhere: the solution of the system, to its tolerance times
    the condition number (a diagonally dominant matrix, below 10)."""
    rng = np.random.default_rng(3)
    n = 700
    a = np.zeros((n, n))
    i = np.arange(n - 1)
    a[i, i + 1] = a[i + 1, i] = -rng.uniform(0.5, 1.0, n - 1)
    a[np.arange(n), np.arange(n)] = 1.3 + np.abs(a).sum(1)
    rp, cl, vl = [0], [], []
    for r in range(n):
        c = rng.permutation(np.flatnonzero(a[r]))
        cl += list(c)
        vl += list(a[r, c])
        rp.append(len(cl))
    x = rng.standard_normal(n)
    got, _, _, status = csr_solve(rp, cl, vl, a @ x, method=method, eps=1e-10)
    assert status == 0
    assert np.linalg.norm(got - x) <= 10 * 1e-10 * np.linalg.norm(a @ x)

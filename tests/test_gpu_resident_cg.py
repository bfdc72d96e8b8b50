"""The CG kernels that keep the system on chip (csrc/cg_resident.cuh), at the sizes where their
launch changes: one CTA, the rows a thread holds (1, 2, 4, 6 or 8 for 152 CTAs of 512 threads),
the last size that fits and the first that goes to the streaming kernel.

b = A x* for a 7-point operator whose diagonal exceeds its row's off-diagonal sum by 10 %, so
||x - x*|| <= ||A^-1|| ||r|| <= cond(A) eps ||x*|| with cond(A) <= 21 max(d) / min(d) <= 100.
"""
import numpy as np
import pytest

from sysu_cfd_heat_gb300.solver import csr_solve

pytestmark = pytest.mark.gpu
EPS = 1e-10


def seven_point(nx, ny, nz, seed):
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    idx = np.arange(n).reshape(nz, ny, nx)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.zeros(n)]
    diag = np.zeros(n)
    for ax in range(3):
        a = np.take(idx, range(idx.shape[ax] - 1), axis=ax).ravel()
        b = np.take(idx, range(1, idx.shape[ax]), axis=ax).ravel()
        w = rng.uniform(0.8, 1.2, a.size)
        rows += [a, b]
        cols += [b, a]
        vals += [-w, -w]
        diag += np.bincount(a, w, n) + np.bincount(b, w, n)
    vals[0] = 1.1 * np.maximum(diag, 2.0)
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order].astype(np.int32), v[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    x = rng.standard_normal(n)
    return rp, c, v, x, np.add.reduceat(v * x[c], rp[:-1])


SIZES = [
    (1, 1, 1), (31, 1, 1), (33, 1, 1), (7, 5, 139),     # one slice, two, a ragged 153rd
    (64, 38, 32), (64, 38, 33),                         # 77,824 rows: one row a thread, then two
    (64, 76, 33), (64, 76, 64), (64, 76, 65),           # four; the last with four, the first with six
    (80, 70, 66), (80, 70, 71), (80, 80, 101),          # beyond FP64's shared memory; beyond FP32's
]


@pytest.mark.parametrize("shape", SIZES)
@pytest.mark.parametrize("method", ["CG", "CG-mixed"])
def test_resident_cg(shape, method):
    rp, c, v, x, b = seven_point(*shape, seed=sum(shape))
    x0 = np.random.default_rng(1).standard_normal(len(x)) if shape[0] % 2 else None
    y, it, res, status = csr_solve(rp, c, v, b, x0, method=method, maxit=1000, eps=EPS, omega=1.3)
    assert status == 0 and res < EPS and it > 0
    assert np.linalg.norm(y - x) <= 100 * EPS * np.linalg.norm(x)
    z, it2, res2, _ = csr_solve(rp, c, v, b, x0, method=method, maxit=1000, eps=EPS, omega=1.3)
    assert it2 == it and res2 == res and np.array_equal(y, z)  # runs are bit-identical


@pytest.mark.parametrize("shape", [(13, 17, 19), (80, 80, 101), (128, 100, 82)])
@pytest.mark.parametrize("method", ["CG", "CG-mixed"])
@pytest.mark.parametrize("kind", ["negative", "spread", "one_negative"])
def test_cg_diagonals(shape, method, kind):
    """Streaming solves run on the scaled system where the diagonal has one sign (a negative
    definite matrix among them); with a single entry of the other sign (capped: it need not
    converge) the form with M^-1 runs; row scales spread over 12 decades leave the answer."""
    rp, c, v, x, b = seven_point(*shape, seed=5)
    n = len(x)
    rows = np.repeat(np.arange(n), np.diff(rp))
    if kind == "spread":  # D A D with D over 6 decades: Jacobi removes it
        d = 10.0 ** np.random.default_rng(2).uniform(-3, 3, n)
        v, b, x = v * d[rows] * d[c], d * b, x / d
    elif kind == "negative":
        v, b = -v, -b
    else:
        v = v.copy()
        at = rp[n // 2] + int(np.where(c[rp[n // 2]:rp[n // 2 + 1]] == n // 2)[0][0])
        v[at] = -v[at]
        _, it, res, status = csr_solve(rp, c, v, b, method=method, maxit=3, eps=EPS)
        assert it == 3 and status == 1 and np.isfinite(res)
        return
    y, it, res, status = csr_solve(rp, c, v, b, method=method, maxit=1000, eps=EPS)
    assert status == 0 and res < EPS
    r = b - np.add.reduceat(v * y[c], rp[:-1])
    assert np.linalg.norm(r) <= 2 * EPS * np.linalg.norm(b)
    if kind == "negative":
        assert np.linalg.norm(y - x) <= 100 * EPS * np.linalg.norm(x)


def test_resident_cg_cap_breakdown_and_no_preconditioner():
    rp, c, v, x, b = seven_point(20, 19, 18, seed=3)
    _, it, res, status = csr_solve(rp, c, v, b, method="CG", maxit=5, eps=1e-14)
    assert it == 5 and status == 1 and res > 1e-14
    y, _, res, status = csr_solve(rp, c, v, b, method="CG", precond="none", maxit=1000, eps=EPS)
    assert status == 0 and np.linalg.norm(y - x) <= 100 * EPS * np.linalg.norm(x)
    y, it, res, status = csr_solve(rp, c, v, np.zeros_like(b), method="CG", maxit=10, eps=EPS)
    assert it == 0 and status == 0 and not y.any()
    bad = b.copy()
    bad[7] = np.nan
    _, it, _, status = csr_solve(rp, c, v, bad, method="CG", maxit=10, eps=EPS)
    assert it == 0 and status == 4


@pytest.mark.parametrize("n", [1, 32, 33, 4864, 77824, 77857, 155680, 262144])
@pytest.mark.parametrize("wide", [0, 20000])
def test_noalloc_cg_sizes(n, wide):
    """sysu_csr_cg_noalloc at the sizes where its launch changes (one CTA, 1, 2 and 4 rows a
    thread, the largest), and with one row so long that its CTA reads the caller's arrays."""
    torch = pytest.importorskip("torch")
    import ctypes as C

    from sysu_cfd_heat_gb300._lib import LIB_PATH

    if wide and n < 2 * wide:
        pytest.skip("the row needs more columns")
    rng = np.random.default_rng(n)
    a = np.arange(n - 1)
    w = rng.uniform(0.5, 1.5, n - 1)
    far = np.arange(n - wide, n) if wide else np.zeros(0, np.int64)  # couplings of row 0
    g = rng.uniform(0.5, 1.0, far.size) / max(wide, 1)
    rows = np.concatenate([a, a + 1, np.zeros(far.size, np.int64), far])
    cols = np.concatenate([a + 1, a, far, np.zeros(far.size, np.int64)])
    off = np.concatenate([w, w, g, g])
    diag = 1.1 * np.maximum(np.bincount(rows, off, n), 1.0)
    r, c = np.concatenate([np.arange(n), rows]), np.concatenate([np.arange(n), cols])
    v = np.concatenate([diag, -off])
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order].astype(np.int32), v[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    x = rng.standard_normal(n)
    b = np.add.reduceat(v * x[c], rp[:-1])
    fn = C.CDLL(LIB_PATH).sysu_csr_cg_noalloc
    fn.argtypes = [C.c_int] + [C.c_void_p] * 5 + [C.c_int, C.c_double, C.c_double] + [C.c_void_p] * 4
    d = [torch.from_numpy(t).cuda() for t in (rp, c, v, b)]
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    it, res, st = C.c_int(), C.c_double(), C.c_int()
    assert fn(n, *(t.data_ptr() for t in d), y.data_ptr(), 1000, EPS, 1.3, None, C.addressof(it), C.addressof(res),
              C.addressof(st)) == 0
    assert st.value == 0 and res.value < EPS
    # cond(A) <= 21 max(d) / min(d) <= 21 * 3.3 / 1.1
    assert np.linalg.norm(y.cpu().numpy() - x) <= 100 * EPS * np.linalg.norm(x)

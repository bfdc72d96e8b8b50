"""Allocation-free CG on one thread-block cluster (up to 8,192 rows) and just beyond: row counts at
the edges of warps, CTAs and cluster sizes, short and dense rows (dense: the matrix stays in the
caller's memory), rows in any column order."""
import ctypes as C

import numpy as np
import pytest

from sysu_cfd_heat_gb300._lib import LIB_PATH

pytestmark = pytest.mark.gpu


def _system(n, dense, rng):
    if dense:
        a = -rng.uniform(0.0, 1.0, (n, n))
        a = a + a.T
        np.fill_diagonal(a, 0.0)
        np.fill_diagonal(a, 1.3 * np.abs(a).sum(1) + 0.1)
        cols = np.argsort(rng.random((n, n)), axis=1)
        return np.arange(n + 1) * n, cols.ravel(), np.take_along_axis(a, cols, 1).ravel()
    step = [1, 33, max(2, n // 2)]  # neighbours in the warp, the CTA, the cluster
    rows = [dict() for _ in range(n)]
    for s in step:
        for i in range(n - s):
            w = rng.uniform(0.2, 1.0)
            rows[i][i + s] = rows[i + s][i] = -w
    rp, cl, vl = [0], [], []
    for i, r in enumerate(rows):
        r[i] = 0.1 + 1.3 * sum(map(abs, r.values()))
        keys = list(r)
        rng.shuffle(keys)
        cl += keys
        vl += [r[k] for k in keys]
        rp.append(len(cl))
    return np.array(rp), np.array(cl), np.array(vl)


@pytest.mark.parametrize("n,dense", [(1, 0), (2, 0), (31, 0), (33, 0), (128, 0), (129, 0), (257, 0), (1716, 0), (2049, 0),
                                     (8160, 0), (8191, 0), (8192, 0), (8193, 0), (300, 1), (700, 1)])
def test_against_the_known_solution(n, dense):
    """Diagonally dominant by 1.3: condition below 10, so x is within 10 eps ||x|| of the solution
    whose right-hand side was formed in FP64."""
    torch = pytest.importorskip("torch")
    f = C.CDLL(LIB_PATH).sysu_csr_cg_noalloc
    p = C.c_void_p
    f.argtypes = [C.c_int, p, p, p, p, p, C.c_int, C.c_double, C.c_double, p, p, p, p]
    rng = np.random.default_rng(n)
    rp, cl, vl = _system(n, dense, rng)
    x = rng.standard_normal(n)
    b = np.array([np.dot(vl[rp[i]:rp[i + 1]], x[cl[rp[i]:rp[i + 1]]]) for i in range(n)])
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (rp.astype(np.int32), cl.astype(np.int32), vl, b)]
    x0 = rng.standard_normal(n)
    got = torch.from_numpy(x0).cuda()
    it, res, status = C.c_int(), C.c_double(), C.c_int()
    for cap, want in ((1, None), (500, 0)):  # the second call starts from the first one's x
        rc = f(n, *(v.data_ptr() for v in d), got.data_ptr(), cap, 1e-10, 1.0, torch.cuda.current_stream().cuda_stream,
               C.addressof(it), C.addressof(res), C.addressof(status))
        assert rc == 0 and it.value <= cap
        assert want is None or status.value == want
    assert res.value < 1e-10
    assert np.linalg.norm(got.cpu().numpy() - x) <= 10 * 1e-10 * np.linalg.norm(x)

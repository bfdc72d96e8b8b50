"""Allocation-free CG of systems small enough in rows for one cluster whose matrix its CTAs' shared
memory does not hold (17,066 entries a CTA): every CTA beyond it, the first, a middle or the last one,
and the largest that fits."""
import numpy as np
import pytest

from test_gpu_cg_small_numbers import noalloc

pytestmark = pytest.mark.gpu
EPS = 1e-10


def system(n, dense_rows, width, seed):
    """A chain, and symmetric couplings of the given rows to `width` rows each."""
    rng = np.random.default_rng(seed)
    a = {(i, i + 1): -rng.uniform(0.5, 1.0) for i in range(n - 1)}
    for r in dense_rows:
        for j in rng.permutation(n)[:width]:
            if j != r:
                a[(min(r, j), max(r, j))] = -rng.uniform(0.0, 1.0) / width
    ij = np.array(list(a), np.int64)
    w = np.array(list(a.values()))
    r, c, v = np.concatenate([ij[:, 0], ij[:, 1]]), np.concatenate([ij[:, 1], ij[:, 0]]), np.concatenate([w, w])
    i = np.arange(n)
    r, c, v = np.concatenate([r, i]), np.concatenate([c, i]), np.concatenate([v, 1.3 * np.bincount(r, -v, n)])
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order].astype(np.int32), v[order]
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    x = rng.standard_normal(n)
    return rp, c, v, x, np.add.reduceat(v * x[c], rp[:-1])


@pytest.mark.parametrize("n,rows,width", [
    (2048, range(0, 2048, 1), 90), (2048, range(0, 12), 2000), (2048, range(1000, 1012), 2000),
    (2048, range(2036, 2048), 2000), (2048, range(0, 2048, 128), 1000), (100, range(100), 99), (130, range(130), 129),
    (8192, range(8180, 8192), 8000), (129, [], 0)])
def test_wide_systems(n, rows, width):
    """Diagonally dominant by 1.3: condition below 21 max(d) / min(d) <= 200."""
    rp, c, v, x, b = system(n, rows, width, n + len(rows))
    for x0 in (None, np.ones(n)):
        y, it, res, status = noalloc(rp, c, v, b, 2000, EPS, x0)
        assert status == 0 and res < EPS and 0 < it < 2000
        assert np.linalg.norm(y - x) <= 200 * EPS * np.linalg.norm(x)

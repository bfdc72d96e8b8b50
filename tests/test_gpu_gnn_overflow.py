"""Features that overflow stay with the rows that the graph connects to them: a row past whose last
neighbour the kernel reads on is not touched by another row's infinities."""
import numpy as np
import pytest

from sysu_cfd_heat_gb300 import learned as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [70, 1000, 9728, 9729])  # 32-row tiles, and the first size with 128-row tiles
def test_an_infinite_row(n):
    i = np.arange(n)
    rp = np.concatenate([[0], np.cumsum(np.where((i == 0) | (i == n - 1), 2, 3))])
    col = np.concatenate([[j for j in (k - 1, k, k + 1) if 0 <= j < n] for k in range(n)])
    val = np.where(col == np.repeat(i, np.diff(rp)), 2.5, -1.0)
    prm = np.zeros(G.NPARAM, np.float32)
    prm[G.OFF_ENC:G.OFF_ENC + 32] = 1.0                            # h0 = u
    prm[G.OFF_LAYER:G.OFF_LAYER + 32 * 32] = 1e38                  # layer 1: overflows where |u| > 1e-1
    b2 = G.OFF_LAYER + G.LAYER_STRIDE + 64 * 32
    prm[b2:b2 + 32] = 1.0                                          # layer 2: adds 1 wherever it can
    r = np.zeros(n)
    r[0] = 1.0
    with G.LearnedPreconditioner(rp, col, val) as net:
        net.params = prm
        h1, h2 = net.hidden(r, 1), net.hidden(r, 2)
    assert not np.isfinite(h1[0]).any() and np.isfinite(h1[1:]).all()
    # layer 2 (weights 0) takes its neighbours' features: only rows 0 and 1 meet the infinities
    assert np.array_equal(h1[2:], np.zeros((n - 2, 32))) and np.array_equal(h2[2:], np.ones((n - 2, 32)))

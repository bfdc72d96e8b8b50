"""Tiles of the learned preconditioner's network kernels against the oracle (oracle/gnn_np.py):
row counts at the edges of the 32- and 128-row tiles and of the rule between them.  Bounds: BF16
operands (2^-9) through four layers with FP32 sums, as for the network's other tests."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import gnn_np as G  # noqa: E402

from sysu_cfd_heat_gb300.learned import LearnedPreconditioner  # noqa: E402

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("shape", [(1, 1, 31), (3, 11, 1), (1, 1, 127), (3, 43, 1), (16, 19, 32), (3, 47, 69)])
def test_tile_edges(shape):
    rp, cl, vl = G.laplacian_3d(*shape, seed=4)
    g = G.Graph(rp, cl, vl)
    rng = np.random.default_rng(5)
    r, e = rng.standard_normal(g.n), rng.standard_normal(g.n)
    p = G.init_params(6)
    p[G.OFF_DEC:G.OFF_DEC + 33] = rng.uniform(-0.3, 0.3, 33)
    z, _ = G.forward(p, g, r, exact=False)
    lo, go, _ = G.loss_and_grad(p, g, r, e, kind=0, exact=False)
    with LearnedPreconditioner(rp, cl, vl) as net:
        net.params = p
        assert _rel(net.apply(r), z) < 5e-3
        net.add_pair(r, e)
        loss, grad = net.loss_grad(0, 0)
    assert abs(loss - lo) <= 2e-3 * abs(lo), (loss, lo)
    blocks = [slice(0, G.OFF_LAYER), slice(G.OFF_DEC, G.NPARAM)]
    blocks += [slice(G.OFF_LAYER + l * G.LAYER_STRIDE, G.OFF_LAYER + l * G.LAYER_STRIDE + 2048) for l in range(G.LAYERS)]
    assert max(_rel(grad[s], go[s]) for s in blocks) < 2e-2

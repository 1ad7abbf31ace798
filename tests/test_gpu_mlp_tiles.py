"""The surrogate's products where their tiles change shape: rows, hidden and output sizes around multiples of 64, inner
sizes that are multiples of 8 but not of 16 (the input gradient sums over n_out), one hidden layer, more stages than are
in flight.  Against the oracle with the same bfloat16 rounding points, at the bars of test_gpu_mlp.py."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,n_in,n_hidden,n_layers,n_out,E", [
    (1, 3, 16, 1, 8, 1), (63, 6, 48, 2, 24, 2), (64, 16, 64, 1, 64, 1), (65, 17, 80, 3, 72, 3), (300, 6, 320, 2, 136, 2), (700, 5, 112, 2, 384, 1)])
def test_tiles(q, n, n_in, n_hidden, n_layers, n_out, E):
    net = q.mlp_ensemble(n_in, n_out, n_hidden, n_layers, E, seed=5)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, n_in)).astype(np.float32)
    Y = rng.standard_normal((n, n_out)).astype(np.float32)
    loss, grad = net.loss_grad(X, Y)
    pred = net.predict(X)
    for e in range(E):
        params = mo.unflatten(net.get_params(e), n_in, n_hidden, n_layers, n_out)
        ref_loss, ref_grad = mo.loss_grad(params, X.astype(np.float64), Y.astype(np.float64), n_in)
        assert abs(loss[e] - ref_loss) <= 1e-4 * ref_loss
        o = 0
        for W, b in params:
            assert rel(grad[e][o:o + W.size], ref_grad[o:o + W.size]) < 2e-2
            assert rel(grad[e][o + W.size:o + W.size + b.size], ref_grad[o + W.size:o + W.size + b.size]) < 2e-2
            o += W.size + b.size
        assert rel(pred[e], mo.predict(params, X.astype(np.float64), n_in)) < 1e-3

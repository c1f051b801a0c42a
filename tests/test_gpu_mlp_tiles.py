"""The network's GEMM at the edges of its tiles (128 rows, 64 columns, 256 of
K per block): gradients of batches around them against the numpy oracle, and
training of batch sizes that change from call to call."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_ref
from test_gpu_mlp import TOL_FORWARD, TOL_GRAD, _inputs, _layer_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 17, 127, 129, 256, 257, 515])
def test_gradients_of_ragged_batches(n):
    from optimisation2forme_b200.warmstart import Network
    with Network(max_batch=600, seed=9) as net:
        x = _inputs(n, n)
        t = np.random.default_rng(n).standard_normal((n, 8)).astype(np.float32)
        loss, g = net.gradients(x, t)
        p, f = net.params()
        lo, go = mlp_ref.gradients(p, f, x, t)
        assert abs(loss - lo) <= 1e-3 * lo
        for s in _layer_slices():
            den = np.linalg.norm(go[s])
            assert np.linalg.norm(g[s] - go[s]) <= TOL_GRAD * den + (den == 0.0) * 1e-12
        y = net.predict(x)
        yo, _ = mlp_ref.forward(p, f, x)
        assert np.linalg.norm(y - yo) <= TOL_FORWARD * np.linalg.norm(yo)


def test_training_continues_over_calls_of_other_sizes():
    from optimisation2forme_b200.warmstart import Network
    x = _inputs(3000, 2)
    t = np.tanh(x[:, :1] * np.arange(1, 9)).astype(np.float32)
    with Network(max_batch=512, seed=1) as net:
        net.set_data(x, t)
        first = net.train(40, batch=300, lr=2e-3, seed=0)
        net.train(3, batch=1, lr=1e-3, seed=1)
        last = net.train(300, batch=512, lr=2e-3, seed=2)
        assert np.all(np.isfinite(first)) and np.all(np.isfinite(last))
        assert last[-20:].mean() < 0.3 * first[:5].mean()
        net.set_data(x[:700], t[:700])  # fewer points, then more: the step follows
        net.train(5, batch=64, lr=1e-3, seed=3)
        net.set_data(np.concatenate([x, x]), np.concatenate([t, t]))
        again = net.train(20, batch=512, lr=1e-3, seed=4)
        assert again.mean() < 0.3 * first[:5].mean()

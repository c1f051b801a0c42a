"""The gradients' sums over the batch have a fixed order: the same inputs give
the same bits, and training the same weights.  (Batches above 4,096 add three
and more parts of a weight gradient in the order they come in; their bias
gradients are fixed like the others.)"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_mlp import TOL_GRAD, _inputs, _layer_slices

pytestmark = pytest.mark.gpu


# around the parts of an accumulator (2,048 rows), its chunks (64 rows, a ring
# of eight) and the bias sums' slices (an eighth of the batch)
@pytest.mark.parametrize("n", [7, 65, 511, 513, 577, 1000, 2048, 2049, 3001, 4095, 4096, 4097])
def test_gradients_are_the_same_every_time(n):
    from optimisation2forme_b200.warmstart import Network
    x = _inputs(n, 5)
    t = np.random.default_rng(6).standard_normal((n, 8)).astype(np.float32)
    fixed = _layer_slices() if n <= 4096 else _layer_slices()[1::2]
    with Network(max_batch=4224, seed=3) as net:
        first = net.gradients(x, t)[1]
        for _ in range(12):
            g = net.gradients(x, t)[1]
            for s in fixed:
                assert np.array_equal(g[s].view(np.int32), first[s].view(np.int32))


def test_training_gives_the_same_weights_every_time():
    from optimisation2forme_b200.warmstart import Network
    x = _inputs(9000, 1)
    t = np.tanh(x[:, :1] * np.arange(1, 9)).astype(np.float32)
    runs = []
    for _ in range(3):
        with Network(max_batch=4096, seed=2) as net:
            net.set_data(x, t)
            net.train(30, batch=4096, lr=1e-3, seed=4)
            net.train(20, batch=1500, lr=1e-3, seed=5)
            runs.append(net.params()[0])
    assert np.array_equal(runs[0].view(np.int32), runs[1].view(np.int32))
    assert np.array_equal(runs[0].view(np.int32), runs[2].view(np.int32))


# parts of one, two and three accumulators, with ragged last chunks
@pytest.mark.parametrize("n", [577, 2047, 2049, 2177, 4096, 4111])
def test_gradients_of_large_batches_match_the_oracle(n):
    from optimisation2forme_b200.warmstart import Network
    from oracle import mlp_ref
    x = _inputs(n, n)
    t = np.random.default_rng(n).standard_normal((n, 8)).astype(np.float32)
    with Network(max_batch=4224, seed=9) as net:
        loss, g = net.gradients(x, t)
        p, f = net.params()
    lo, go = mlp_ref.gradients(p, f, x, t)
    assert abs(loss - lo) <= 1e-3 * lo
    for s in _layer_slices():
        den = np.linalg.norm(go[s])
        assert np.linalg.norm(g[s] - go[s]) <= TOL_GRAD * den + (den == 0.0) * 1e-12

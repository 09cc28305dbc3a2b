"""Training steps that follow one another on the GPU: each step's kernels start
under the tail of the step before (dependent launches), so many steps in one call
must give the bits of single steps with a synchronisation after each."""
import numpy as np
import pytest

from test_gpu_surrogate import random_params

pytestmark = pytest.mark.gpu


def trained(marl, batch, calls):
    rng = np.random.default_rng(batch)
    raw = np.zeros((6000, 112), np.float32)
    raw[:, :109] = rng.integers(0, 1024, (6000, 109)) / np.float32(1024)
    s = marl.Surrogate(max_pairs=6000, batch=batch, seed=9, lr=1e-3)
    s.upload_pairs(raw)
    s.set_weights(random_params(rng))
    s.prepare(6000)
    loss = []
    for k in calls:
        loss += list(s.train(k))
        s.get_weights()
    params = s.get_weights()[0]
    s.close()
    return np.asarray(loss, np.float32), params


@pytest.mark.parametrize("batch", [128, 640, 8192])
def test_one_call_equals_single_steps(marl, batch):
    loss, params = trained(marl, batch, [1] * 24)
    for calls in ([24], [24], [5, 19]):
        again = trained(marl, batch, calls)
        np.testing.assert_array_equal(again[0], loss)
        np.testing.assert_array_equal(again[1], params)

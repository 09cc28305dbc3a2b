"""The training step's kernels at sizes the gradient test does not reach, and
the batch rows a step draws, against the float64 restatement."""
import numpy as np
import pytest

import mlp_ref
from test_gpu_surrogate import identity_norm, normwise, random_params

pytestmark = pytest.mark.gpu

PARTS = [mlp_ref.OFF_W1, mlp_ref.OFF_B1, mlp_ref.OFF_W2, mlp_ref.OFF_B2, mlp_ref.OFF_W3, mlp_ref.OFF_B3,
         mlp_ref.N_PARAMS]


@pytest.mark.parametrize("batch", [256, 1152, 2432, 8192])
def test_gradients_over_many_splits(marl, batch):
    """Less than one split of 512 rows, a partial last split, the default batch."""
    rng = np.random.default_rng(batch)
    s = marl.Surrogate(max_pairs=128, batch=128)
    params = random_params(rng)
    s.set_weights(params, identity_norm())
    x = rng.normal(0, 1, (batch, 128)).astype(np.float32)
    x[:, 93:] = 0
    xb, t = mlp_ref.bf16_bits(x), rng.normal(0, 1, (batch, 16)).astype(np.float32)
    g, loss, y = s.gradients(xb, t)
    loss_ref, g_ref, y_ref = mlp_ref.loss_and_gradients(params, xb, t)
    assert normwise(y, y_ref) < 2e-3 and abs(loss - loss_ref) <= 2e-3 * abs(loss_ref)
    for a, b in zip(PARTS, PARTS[1:]):
        assert normwise(g[a:b], g_ref[a:b]) < 2e-3, (a, b)
    s.close()


def mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


@pytest.mark.parametrize("batch", [128, 640])
def test_steps_train_on_the_drawn_rows(marl, batch):
    """The losses of two steps equal those of gradients() on the rows the
    draws name (a wrong row set of this size is off by several percent), and
    the step's update is Adam's on gradients()'s gradient."""
    rng = np.random.default_rng(batch)
    n, seed = 1500, 77
    raw = np.zeros((n, 112), np.float32)
    raw[:, :109] = rng.random((n, 109), dtype=np.float32)
    s = marl.Surrogate(max_pairs=n, batch=batch, seed=seed, lr=1e-3)
    params = random_params(rng)
    s.upload_pairs(raw)
    s.set_weights(params)
    s.prepare(n)
    norm = s.get_weights()[1]
    f = raw[:, :93].copy()
    logs = [29 + 4 * r + i for r in range(16) for i in range(3)]
    f[:, logs] = np.log(np.abs(f[:, logs]) + np.float32(1e-3))
    x = np.zeros((n, 128), np.float32)
    x[:, :93] = (f - norm[:93]) / norm[93:186]
    t = (raw[:, 93:109] - norm[186:202]) / norm[202:218]
    ref = marl.Surrogate(max_pairs=128, batch=128)
    for step in range(2):
        with np.errstate(over="ignore"):
            at = mix64(np.uint64(seed) ^ mix64(np.uint64(step) * np.uint64(0x100000001B3) +
                                               np.arange(batch, dtype=np.uint64))) % np.uint64(n)
        before = s.get_weights()[0]
        ref.set_weights(before, norm)
        g, loss, _ = ref.gradients(mlp_ref.bf16_bits(x[at]), t[at])
        got = s.train(1)[0]
        assert abs(got - loss) <= 1e-4 * loss
        if step == 0:  # first step: m = (1 - b1) g, v = (1 - b2) g^2, so the update is lr g / (|g| + eps)
            big = np.abs(g) > 1e-4 * np.abs(g).max()  # where rounding cannot turn the sign
            moved = before - s.get_weights()[0]
            np.testing.assert_allclose(moved[big], 1e-3 * g[big] / (np.abs(g[big]) + 1e-8), rtol=2e-3)
    s.close()
    ref.close()

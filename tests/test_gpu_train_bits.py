"""The training step's roundings, bit for bit.

Up to 512 rows a weight gradient is one partial sum, so its bits say whether any
BF16 rounding of h1, h2, dY, dZ2 or dZ1 differs; the weights after steps from the
same parameters (the moments are carried over) add Adam's.  The fingerprints in
golden/train_step_bits.json were recorded from the step as a kernel per layer and
direction, gelu and its derivative as two functions, gradients added by atomics
(which makes the biases' bits vary there: they are left out).
"""
import hashlib
import json
import os

import numpy as np
import pytest

import mlp_ref
from test_gpu_surrogate import identity_norm, random_params

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "train_step_bits.json")
WEIGHTS = {"W1": (mlp_ref.OFF_W1, mlp_ref.OFF_B1), "W2": (mlp_ref.OFF_W2, mlp_ref.OFF_B2),
           "W3": (mlp_ref.OFF_W3, mlp_ref.OFF_B3)}


def sha(flat: np.ndarray) -> dict:
    return {k: hashlib.sha256(np.ascontiguousarray(flat[a:b]).tobytes()).hexdigest()[:16]
            for k, (a, b) in WEIGHTS.items()}


def gradients(marl, batch: int) -> list:
    rng = np.random.default_rng(batch)
    s = marl.Surrogate(max_pairs=128, batch=128)
    out = []
    for _ in range(6):
        s.set_weights(random_params(rng), identity_norm())
        x = rng.normal(0, 1.5, (batch, 128)).astype(np.float32)
        x[:, 93:] = 0
        t = rng.normal(0, 1, (batch, 16)).astype(np.float32)
        out.append(sha(s.gradients(mlp_ref.bf16_bits(x), t)[0]))
    s.close()
    return out


def steps(marl, batch: int) -> list:
    rng = np.random.default_rng(batch)
    raw = np.zeros((4000, 112), np.float32)
    raw[:, :109] = rng.integers(0, 1024, (4000, 109)) / np.float32(1024)
    s = marl.Surrogate(max_pairs=4000, batch=batch, seed=5, lr=1e-3)
    s.upload_pairs(raw)
    params, out = random_params(rng), []
    s.set_weights(params)
    s.prepare(4000)
    for _ in range(5):
        s.set_weights(params)
        s.train(1)
        out.append(sha(s.get_weights()[0]))
    s.close()
    return out


@pytest.mark.parametrize("batch", [128, 384, 512])
def test_gradients(marl, batch):
    assert gradients(marl, batch) == json.load(open(GOLDEN))["gradients"][str(batch)]


@pytest.mark.parametrize("batch", [128, 512])
def test_steps(marl, batch):
    assert steps(marl, batch) == json.load(open(GOLDEN))["steps"][str(batch)]

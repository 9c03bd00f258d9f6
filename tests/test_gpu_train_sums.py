"""The sums of the training step, bit for bit: a bias gradient is the FP32 sum of
its column over the samples of a 64-sample chunk, rounded after each sample, and
the batch's gradient the FP32 sum of its chunks.

A sample's own terms do not depend on its place in a batch, and the mean's 1/n is
an exact factor for n a power of two, so gradients of one sample give the terms of
larger batches and no tolerance is needed."""
import os

import numpy as np
import pytest

import mcx
from mcx.gain import init_weights

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "train_batch128.npz")
B1 = slice(32 * 64, 32 * 64 + 64)
B2 = slice(B1.stop + 64 * 64, B1.stop + 64 * 64 + 64)
B3 = slice(B2.stop + 64 * 8, B2.stop + 64 * 8 + 8)


def _samples(n, seed):
    """Ordered neighbourhoods: six neighbours and the director, T (columns 0..21)."""
    r = np.random.default_rng(seed)
    v = r.normal(0, 0.6, (n, 7, 3)) + r.normal(0, 1, 3)
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    s = np.zeros((n, 22))
    s[:, :18] = v[:, :6].reshape(n, 18)
    s[:, 18] = r.uniform(0.9, 1.2, n)
    s[:, 19:22] = v[:, 6]
    return s.astype(np.float32)


def _engine():
    eng = mcx.Engine([mcx.replica(nx=8, ny=8, nz=8, T=1.1, seed=5)])
    eng.set_mlp(init_weights(3))
    return eng


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_bias_gradients_round_after_every_sample(seed):
    n = 64
    s = _samples(n, seed)
    with _engine() as eng:
        one = np.stack([eng.mlp_grad(s[i:i + 1])[1] for i in range(n)]) / np.float32(n)
        _, g = eng.mlp_grad(s)
    for b in (B1, B2, B3):
        want = np.zeros(one[:, b].shape[1], np.float32)
        for row in one[:, b]:
            want = want + row
        assert np.array_equal(g[b], want)


@pytest.mark.parametrize("n", [128, 512, 8192, 16384])
def test_gradient_adds_its_chunks_in_order(n):
    """One chunk per CTA (at most 256 of them), added in FP32 one after another."""
    s = _samples(n, 7)
    with _engine() as eng:
        want = np.zeros(mcx.MLP_PARAMS, np.float32)
        for c in range(0, n, 64):
            want = want + eng.mlp_grad(s[c:c + 64])[1] * np.float32(64 / n)
        assert np.array_equal(eng.mlp_grad(s)[1], want)


def record(path):
    """Weights after training with batches of at most two chunks, whose sum does
    not depend on which chunk is added first (recorded with atomic additions)."""
    out = {}
    for batch, seed in ((128, 1), (64, 2), (100, 3)):
        with _engine() as eng:
            eng.mlp_grad(_samples(4096, seed))  # held as the training samples
            loss = eng.train_mlp(samples=0, batch=batch, steps=100, lr=1e-3, seed=seed)
            out["weights%d" % batch], out["loss%d" % batch] = eng.get_mlp(), loss
    if path:
        np.savez_compressed(path, **out)
    return out


def test_trained_weights_are_the_recorded_ones():
    got, want = record(None), np.load(GOLD)
    for batch in (128, 64, 100):
        assert np.array_equal(got["weights%d" % batch], want["weights%d" % batch])
        # a step's loss is a sum of 4 or 8 warp sums in any order: 8 roundings
        assert np.allclose(got["loss%d" % batch], want["loss%d" % batch], rtol=8 * 2.0 ** -24, atol=1e-7)

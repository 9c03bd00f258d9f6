"""The training step's batch draw, partial sums and determinism: batches at the
edges of the 64-sample chunks and of a CTA's share of them."""
import numpy as np
import pytest

import mcx
from mcx.gain import init_weights
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _engine(n=12, reps=2):
    eng = mcx.Engine([mcx.replica(nx=n, ny=n, nz=n, T=1.1, seed=5 + q, stream=q) for q in range(reps)])
    eng.sweep(50)
    eng.set_mlp(init_weights(3))
    return eng


def _batch(n, nsamples, seed, step):
    return np.array([(int(O.philox((i, step, 0xBA7C, 0xC011), (seed, 0x7EA1))[0]) * nsamples) >> 32
                     for i in range(n)])


@pytest.mark.parametrize("batch", [1, 63, 64, 65, 1000, 64 * 304 + 1])
def test_first_step_is_the_drawn_batch(batch):
    """The loss of the first step is mlp_grad's over the samples the step's
    Philox counters draw.  Both are sums of FP32 terms below 4 in groups of 64:
    2e-6 relative covers their order."""
    nsamples = 777
    with _engine() as eng:
        s = eng.collect_samples(nsamples, seed=9, augment=mcx.AUG_FLIP)
        want, g = eng.mlp_grad(s[_batch(batch, nsamples, 9, 1)])
        w0 = eng.get_mlp()
        loss = eng.train_mlp(samples=nsamples, batch=batch, steps=1, lr=1e-3, seed=9, augment=mcx.AUG_FLIP)
        assert loss[0] == pytest.approx(want, rel=2e-6)
        # Adam's first step moves a weight by the learning rate against its gradient's sign
        d, big = eng.get_mlp() - w0, np.abs(g) > 1e-4 * np.abs(g).max()
        assert np.allclose(d[big], -1e-3 * np.sign(g[big]), atol=2e-5)


def test_training_does_not_depend_on_timing():
    """Fixed-order sums: two trainings from the same state give the same bits."""
    out = []
    for _ in range(2):
        with _engine() as eng:
            loss = eng.train_mlp(samples=5000, batch=3000, steps=60, lr=2e-3, seed=4, augment=mcx.AUG_FLIP)
            out.append((loss, eng.get_mlp()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

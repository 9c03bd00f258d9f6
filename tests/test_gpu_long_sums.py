"""Measured sums of deep chunks against FP64: the energy of one measured sweep of an
unmasked lattice is that of its final state.

A thread adds its n terms of a chunk in FP32 one by one.  An addition is off by an
ulp / sqrt(12) of its result (rms; 0.42 x 2^-24 of it, averaged over mantissas), so a
chain of n equal terms by 0.42 x 2^-24 sqrt(n / 3) of itself, and N terms in N / n
independent chains by 0.42 x 2^-24 n / sqrt(3 N).  The plain z-march's chains are 16
terms (8 planes of two sites of colour 1, which count the bonds), the learned one's at
most 64 (32 planes); what follows keeps two parts.  The bound is six times that."""
import numpy as np
import pytest

import mcx
from mcx.gain import init_weights

pytestmark = pytest.mark.gpu


def _energy(v, n):
    v = v.astype(np.float64).reshape(n, n, n, 3)
    return sum(2 * float((-1.5 * (v * np.roll(v, -1, ax)).sum(-1) ** 2).sum()) for ax in range(3)) / n ** 3


@pytest.mark.parametrize("n,reps,learned", [(96, 6, False), (64, 8, False), (96, 8, True)])
def test_energy_of_deep_chunks(n, reps, learned):
    with mcx.Engine([mcx.replica(nx=n, ny=n, nz=n, T=1.0, seed=3 + q, stream=q) for q in range(reps)]) as eng:
        if learned:
            eng.set_mlp(init_weights(3))
            eng.set_proposal("vmf_mlp")
        eng.sweep(30)
        eng.sweep(1, measure=True)
        terms = 64 if learned else 16
        tol = 6 * 0.42 * 2.0 ** -24 * terms / np.sqrt(3 * n ** 3 / 2)
        for q in range(reps):
            want = _energy(eng.get_state(q), n)
            assert abs(eng.stats(q)[mcx.ST_E1] - want) <= tol * abs(want)

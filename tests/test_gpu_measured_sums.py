"""The masked z-march's measured sums against the direct pass: the same chain
bit for bit, and the same sums up to the FP32 order of a pass's partial sums
(1e-7 relative per sweep for E and the E of active sites, 1e-8 for S; the
bounds are three times that)."""
import numpy as np
import pytest

import mcx
from oracle import oracle as O
from helpers import desc_from_model

pytestmark = pytest.mark.gpu

HOM, FG = O.Surface("homeotropic", 4.0), O.Surface("fg", 1.0)
MODELS = {
    "ll_16": dict(nx=16, ny=16, nz=16, potential="ll"),
    "ll_min": dict(nx=4, ny=2, nz=2, potential="ll"),
    "ll_half_pairs": dict(nx=18, ny=6, nz=10, potential="ll"),
    "ll_free_odd": dict(nx=13, ny=7, nz=5, potential="ll", xbound="free", ybound="free", zbound="free"),
    "ghrl_chiral": dict(nx=24, ny=10, nz=17, potential="ghrl", k11=1.48, k33=2.28, p0=40.0, zbound="free", elecA=0.4,
                        elecZ=1.0),
    "pear": dict(nx=20, ny=14, nz=18, potential="pear", B1=0.04, C=0.3),
    "slab_mixed": dict(nx=12, ny=14, nz=11, geometry="slab", potential="ghrl", k22=0.8, k33=1.2,
                       surfaces=[O.Surface("rp", 2.0, theta_s=30, phi_s=40), O.Surface("fg_ghrl", 1.5)]),
    "droplet_hom_odd": dict(nx=21, ny=21, nz=21, geometry="sphere", potential="ghrl", k11=1.48, k33=2.28,
                            xbound="free", ybound="free", zbound="free", surfaces=[HOM]),
    "droplet_fg_field": dict(nx=26, ny=26, nz=26, geometry="sphere", potential="ghrl", k22=0.6, k33=1.4, p0=20.0,
                             xbound="free", ybound="free", zbound="free", elecA=1.0, elecZ=1.0, elecE=0.7, radius=10.0,
                             surfaces=[FG]),
}


def _run(name, kind, shape=None, sweeps=(3, 40, 150), replicas=3):
    m = O.Model(**MODELS[name])
    descs = [desc_from_model(m, T=0.9, seed=70 + q, stream=q) for q in range(replicas)]
    with mcx.Engine(descs) as eng:
        eng.pass_kind = kind
        if shape:
            eng.set_march_shape(*shape)
        for q in range(replicas):
            eng.init_random(q, 5 + q)
        eng.sweep(sweeps[0])
        eng.sweep(sweeps[1], measure=True)
        eng.sweep(1, measure=True)
        eng.sweep(sweeps[2], measure=True)
        return [(eng.get_state(q), eng.stats(q)) for q in range(replicas)]


def _same(ref, out):
    for (s0, t0), (s1, t1) in zip(ref, out):
        assert np.array_equal(s0, s1)
        for k in (mcx.ST_N, mcx.ST_ACC, mcx.ST_SWEEPS, mcx.ST_ANG_VAR, mcx.ST_SWEEP_INDEX):
            assert t0[k] == t1[k]
        for k in (mcx.ST_E1, mcx.ST_EV1):
            assert abs(t0[k] - t1[k]) <= 3e-7 * abs(t0[k]) + 1e-9 * t0[mcx.ST_N]
        assert abs(t0[mcx.ST_S1] - t1[mcx.ST_S1]) <= 3e-8 * t0[mcx.ST_N]


@pytest.mark.parametrize("name", [n for n in MODELS if n.startswith(("slab", "droplet", "ll_free"))])
def test_masked_march_measures_as_the_direct_pass(name):
    ref = _run(name, "direct")
    _same(ref, _run(name, "march", (64, 0)))
    _same(ref, _run(name, "march", (128, 8)))

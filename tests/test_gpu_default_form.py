"""Calls that leave the form or the shape of the sweeps to the engine give back what
the engine chose.  Shapes are seen in the last digits of the measured sums."""
import numpy as np
import pytest

import mcx

pytestmark = pytest.mark.gpu


def _sums(eng):
    for q in range(eng.n):
        eng.init_random(q, 5 + q)
    eng.reset_stats()
    eng.sweep(20, measure=True)
    return np.stack([eng.stats(q) for q in range(eng.n)])[:, [mcx.ST_E1, mcx.ST_S1, mcx.ST_EV1]]


def _droplets():
    return [mcx.replica(nx=96, ny=96, nz=96, geometry="sphere", radius=40.0, potential="ghrl", k11=1.0, k33=1.4, T=0.8,
                        seed=3, stream=q, surfaces=[dict(anchoring="homeotropic", W=2.0)]) for q in range(2)]


def test_the_default_shape_comes_back_after_the_persistent_form():
    got = []
    for visit in (False, True):
        with mcx.Engine(_droplets()) as eng:
            if visit:
                try:
                    eng.pass_kind = "march_persistent"
                except mcx.McxError as e:
                    assert e.status == 4  # too many units to be resident at once: refused
                eng.pass_kind = "march"
            eng.set_adapt(False)
            got.append(_sums(eng))
    assert np.allclose(got[0], got[1], rtol=1e-12, atol=0.0)


def test_a_refused_form_leaves_the_one_before():
    # small lattices, a block of pairs each and more of them than the GPU holds CTAs at once
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16, seed=q + 1) for q in range(1200)]) as eng:
        before = eng.pass_kind
        assert before == "resident"
        with pytest.raises(mcx.McxError) as e:
            eng.pass_kind = "march_persistent"
        assert e.value.status == 4 and eng.pass_kind == before


def test_staging_off_is_the_default_form():
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as eng:
        assert eng.pass_kind == "resident"
        eng.staged = False
        assert eng.pass_kind == "resident"
        eng.staged = True
        assert eng.pass_kind == "staged"
        eng.staged = False
        assert eng.pass_kind == "resident"
        eng.pass_kind = "direct"
        eng.staged = False  # another pass was asked for
        assert eng.pass_kind == "march"
        eng.sweep(3)
        eng.sync()
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as eng:
        eng.set_march_shape(128, 8)
        eng.staged = False
        assert eng.pass_kind == "march"


@pytest.mark.parametrize("name,value", [("MCX_MARCH_NT", "64"), ("MCX_MARCH_K", "2")])
def test_a_shape_from_the_environment_runs_the_march(name, value, monkeypatch):
    monkeypatch.setenv(name, value)
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as eng:
        assert eng.pass_kind == "march"


@pytest.mark.parametrize("kind", ["march_persistent", "march_tma", "resident"])
def test_the_autotuner_leaves_a_form_it_timed(kind):
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as eng:
        eng.pass_kind = kind
        eng.autotune()
        assert eng.pass_kind in ("march", "march_async", "march_quad", "resident")
        eng.sweep(20)
        eng.sync()

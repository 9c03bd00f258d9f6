"""The resident sweeps (small lattices in the shared memory of a CTA cluster)
against the direct pass: the same chain bit for bit, and the same sums within
the bounds of test_gpu_measured_sums.py."""
import numpy as np
import pytest

import mcx
from test_gpu_measured_sums import MODELS, _run, _same

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("name", list(MODELS))
def test_resident_is_the_direct_chain(name):
    _same(_run(name, "direct"), _run(name, "resident"))


def test_small_lattices_run_resident_by_default_and_large_ones_do_not():
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as small:
        assert small.pass_kind == "resident"
        small.set_march_shape(128, 8)  # a z-march shape is asked for
        assert small.pass_kind == "march"
    with mcx.Engine([mcx.replica(nx=96, ny=96, nz=96)]) as large:
        assert large.pass_kind != "resident"
        with pytest.raises(mcx.McxError) as e:
            large.pass_kind = "resident"
        assert e.value.status == 4


def test_measured_sums_do_not_depend_on_the_batch():
    """A replica's resident sums are split so that they do not depend on how
    the batch cuts it: 1e-9 relative, alone and in batches of other sizes."""
    d = [mcx.replica(nx=n, ny=n, nz=n, T=0.9, seed=3, stream=n) for n in (16, 24, 8)]
    got = []
    for batch in ([0], [0, 1], [2, 0], [0] + [2] * 40):
        with mcx.Engine([d[q] for q in batch]) as eng:
            eng.pass_kind = "resident"
            r = batch.index(0)
            eng.init_random(r, 9)
            eng.sweep(25, measure=True)
            got.append((eng.get_state(r), eng.stats(r)))
    for s, t in got[1:]:
        assert np.array_equal(s, got[0][0])
        for k in (mcx.ST_E1, mcx.ST_S1, mcx.ST_S2):
            assert t[k] == pytest.approx(got[0][1][k], rel=1e-9)

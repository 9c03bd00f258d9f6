"""The resident sweeps' bounded waits: a run whose waits are for four bytes more than
anyone sends gives up after its limit with an error, and leaves the replicas' states
and the engine usable."""
import numpy as np
import pytest

import mcx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,reps", [(16, 1), (24, 5), (8, 40)])
def test_run_gives_up_and_the_engine_goes_on(n, reps):
    d = [mcx.replica(nx=n, ny=n, nz=n, T=1.0, seed=4, stream=q) for q in range(reps)]
    with mcx.Engine(d) as eng, mcx.Engine(d) as ref:
        for e in (eng, ref):
            e.pass_kind = "resident"
            for q in range(reps):
                e.init_random(q, 3 + q)
            e.sweep(10)
        assert mcx.lib().mcx_debug_barrier_timeout(eng._h) == 2  # MCX_ERR_CUDA
        assert "resident" in mcx.lib().mcx_last_error(eng._h).decode()
        for e in (eng, ref):
            e.sweep(20, measure=True)
            e.sync()
        for q in range(reps):
            assert np.array_equal(eng.get_state(q), ref.get_state(q))
            assert np.allclose(eng.stats(q), ref.stats(q), rtol=1e-12)


def test_other_forms_refuse_the_test():
    with mcx.Engine([mcx.replica(nx=16, ny=16, nz=16)]) as eng:
        eng.pass_kind = "march"
        assert mcx.lib().mcx_debug_barrier_timeout(eng._h) == 1  # MCX_ERR_INVALID

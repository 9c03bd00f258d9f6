"""An engine of custom geometry that is given a droplet's mask plans as the engine
that makes the droplet itself: the same form of the sweeps and, seen in the last
digits of the measured sums, the same shape and units; also for masks that come with
a checkpoint, and for the learned proposal."""
import numpy as np
import pytest

import mcx
from mcx.gain import init_weights

pytestmark = pytest.mark.gpu
FREE = dict(xbound="free", ybound="free", zbound="free")
KEY = dict(potential="ghrl", k11=1.0, k22=0.6, k33=1.4, T=0.8, surfaces=[dict(anchoring="homeotropic", W=2.0)], **FREE)


def _descs(geometry, n, radius, reps):
    return [mcx.replica(nx=n, ny=n, nz=n, geometry=geometry, radius=radius, seed=3, stream=q, **KEY)
            for q in range(reps)]


def _measured(eng, learned=False):
    for q in range(eng.n):
        eng.init_random(q, 5 + q)
    if learned:
        eng.set_proposal("vmf_mlp")
    eng.sweep(3)
    eng.sweep(20, measure=True)
    return eng.pass_kind, [eng.get_state(q) for q in range(eng.n)], [eng.stats(q) for q in range(eng.n)]


def _same(a, b):
    assert a[0] == b[0]
    assert all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))
    for x, y in zip(a[2], b[2]):  # FP64 sums in any order; another shape shows at 1e-9 to 1e-8
        assert np.allclose(x, y, rtol=1e-12, atol=0.0)


@pytest.mark.parametrize("n,radius,reps", [(16, 5.0, 1), (24, 0.0, 4), (40, 12.0, 2), (44, 14.0, 1), (48, 10.0, 3), (52, 12.0, 1),
                                           (61, 20.0, 1),
                                           (96, 40.0, 2)])
@pytest.mark.parametrize("how", ["set_mask", "load"])
def test_a_droplet_mask_is_planned_as_the_droplet(n, radius, reps, how, tmp_path):
    path = str(tmp_path / "c.mcx")
    with mcx.Engine(_descs("sphere", n, radius, reps)) as own:
        masks = [own.get_mask(q) for q in range(reps)]
        want = _measured(own)
    with mcx.Engine(_descs("custom", n, radius, reps)) as eng:
        for q in range(reps):
            eng.set_mask(q, *masks[q])
        if how == "load":
            eng.save(path)
        else:
            _same(want, _measured(eng))
    if how == "load":
        with mcx.Engine(_descs("custom", n, radius, reps)) as eng:
            eng.load(path)
            _same(want, _measured(eng))


@pytest.mark.parametrize("n,radius,reps", [(52, 18.0, 2), (64, 20.0, 6), (80, 34.0, 3)])
def test_learned_units_follow_the_mask(n, radius, reps):
    with mcx.Engine(_descs("sphere", n, radius, reps)) as own, mcx.Engine(_descs("custom", n, radius, reps)) as eng:
        masks = [own.get_mask(q) for q in range(reps)]
        own.set_mlp(init_weights(3))
        eng.set_mlp(init_weights(3))
        for q in range(reps):
            eng.set_mask(q, *masks[q])
        _same(_measured(own, True), _measured(eng, True))


def test_learned_units_follow_the_network_path(monkeypatch):
    d = [mcx.replica(nx=96, ny=96, nz=96, T=1.1, seed=3, stream=q) for q in range(2)]
    monkeypatch.setenv("MCX_MLP_PATH", "1")
    with mcx.Engine(d) as own:
        own.set_mlp(init_weights(3))
        monkeypatch.delenv("MCX_MLP_PATH")
        with mcx.Engine(d) as eng:
            eng.set_mlp(init_weights(3))
            eng.mlp_path = "tcgen05"
            assert own.mlp_path == eng.mlp_path == "tcgen05"
            _same(_measured(own, True), _measured(eng, True))


@pytest.mark.parametrize("learned", [False, True])
def test_a_captured_run_after_a_mask(learned):
    """A caller that captures the engine's stream right after setting a mask: nothing
    can be planned there, and the plans there are give the same chain."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs torch on the GPU")
    got = []
    for capture in (False, True):
        with mcx.Engine(_descs("sphere", 24, 8.0, 2)) as own, mcx.Engine(_descs("custom", 24, 8.0, 2)) as eng:
            eng.set_mlp(init_weights(3))
            if learned:
                eng.set_proposal("vmf_mlp")
            for q in range(2):
                eng.init_random(q, 5 + q)
            eng.sweep(2)
            for q in range(2):
                eng.set_mask(q, *own.get_mask(q))
            if capture:
                stream = torch.cuda.ExternalStream(mcx.lib().mcx_stream(eng._h))
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
                    eng.sweep(3)
                graph.replay()
                torch.cuda.synchronize()
            else:
                eng.sweep(3)
            got.append([eng.get_state(q) for q in range(2)])
    assert all(np.array_equal(x, y) for x, y in zip(*got))

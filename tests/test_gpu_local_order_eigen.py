"""Local order where the largest eigenvalue is easy, near a double one and
exactly double, against FP64 eigenvalues.  The kernel's Q is a FP32 sum of up
to seven terms below 3 less the identity, over 14: six roundings of at most
half a unit of 16 (4.8e-7), 2.1e-7 in an entry, 6.2e-7 in an eigenvalue, and
3e-8 from the result's own rounding: 7e-7."""
import numpy as np
import pytest

import mcx

pytestmark = pytest.mark.gpu


def _states(n):
    rng = np.random.default_rng(4)
    k, j, i = np.meshgrid(*(np.arange(n),) * 3, indexing="ij")
    unit = lambda v: (v / np.linalg.norm(v, axis=-1, keepdims=True)).astype(np.float32)
    rnd = rng.normal(size=(n, n, n, 3))
    plane = np.stack([np.cos(0.9 * i), np.sin(0.9 * i), 0 * i], -1)
    xy = np.where(((i + j + k) % 2 == 0)[..., None], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0])
    return {
        "random": unit(rnd),
        "ordered": unit(rnd * 0.05 + [0.0, 0.6, 0.8]),
        "aligned": unit(np.broadcast_to([0.0, 0.6, 0.8], rnd.shape)),
        "in_a_plane": unit(plane + 1e-3 * rnd),
        "two_axes": unit(xy),
        "two_axes_almost": unit(xy + 1e-4 * rnd),
        "three_axes": unit(np.eye(3)[(i + j + k) % 3]),
    }


@pytest.mark.parametrize("name", list(_states(2)))
@pytest.mark.parametrize("n", [6, 20])
def test_local_order_is_the_largest_eigenvalue(name, n):
    v = _states(n)[name]
    with mcx.Engine([mcx.replica(nx=n, ny=n, nz=n, zbound="free")]) as eng:
        eng.set_state(0, v.reshape(-1, 3))
        got = eng.local_order(0).reshape(n, n, n)
    q = 3 * np.einsum("...a,...b->...ab", v.astype(np.float64), v.astype(np.float64)) - np.eye(3)
    Q, cnt = q.copy(), np.full((n, n, n), 5.0)
    for ax in (1, 2):
        Q += np.roll(q, 1, ax) + np.roll(q, -1, ax)
    Q[1:] += q[:-1]
    Q[:-1] += q[1:]
    cnt[1:] += 1
    cnt[:-1] += 1
    want = np.linalg.eigvalsh(Q / (2 * cnt)[..., None, None])[..., -1]
    assert np.abs(got - want).max() <= 7e-7

"""Resident sweeps of masks whose planes have active sites of one colour only, so
that a CTA sends its neighbours rows of one colour or none: the direct pass's chain,
bit for bit, and the sums within the bounds of test_gpu_measured_sums.py."""
import numpy as np
import pytest

import mcx
from test_gpu_measured_sums import _same

pytestmark = pytest.mark.gpu


def _mask(kind, n):
    k, j, i = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    colour = (i + j + k) % 2
    if kind == "by_plane":  # colours 0 0 1 1 0 0 ... along z
        on = colour == (k // 2) % 2
    elif kind == "thirds":  # full planes between planes of one colour
        on = (k % 3 == 0) | (colour == (k // 3) % 2)
    else:  # one active site on the first and last plane, full between
        on = ((k > 1) & (k < n - 2)) | ((i == 3) & (j == 4))
    return on.astype(np.int32).reshape(-1)


@pytest.mark.parametrize("kind", ["by_plane", "thirds", "poles"])
@pytest.mark.parametrize("measured", [False, True])
def test_one_coloured_planes(kind, measured):
    n, got = 18, []
    for form in ("direct", "resident"):
        d = [mcx.replica(nx=n, ny=n, nz=n, geometry="custom", potential="ghrl", k11=1.0, k22=0.8, k33=1.3, T=0.7,
                         seed=11, stream=q) for q in range(3)]
        with mcx.Engine(d) as eng:
            for q in range(3):
                eng.set_mask(q, _mask(kind, n))
                eng.init_random(q, 7 + q)
            eng.pass_kind = form
            eng.sweep(300, measure=measured)
            eng.sync()
            got.append([(eng.get_state(q), eng.stats(q)) for q in range(3)])
    _same(*got)

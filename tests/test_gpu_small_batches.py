"""Batches of lattices of some hundred active sites, whose z-march passes add
inactive sites' field energy themselves: every form's chain and sums against
the direct pass (bounds of test_gpu_measured_sums.py), and the default form and
shape of such a batch."""
import pytest

import mcx
from oracle import oracle as O
from test_gpu_measured_sums import MODELS, _run, _same

pytestmark = pytest.mark.gpu

SPHERE = dict(geometry="sphere", potential="ghrl", k22=0.6, k33=1.4, p0=20.0, xbound="free", ybound="free",
              zbound="free", elecA=1.0, elecZ=1.0, elecE=0.7, surfaces=[O.Surface("fg", 1.0)])
SMALL = {
    "odd": dict(nx=9, ny=9, nz=9, **SPHERE),
    "mostly_inactive": dict(nx=30, ny=30, nz=30, radius=5.0, **SPHERE),
    "slab": dict(nx=8, ny=6, nz=7, geometry="slab", potential="ghrl", k22=0.8, elecA=1.0, elecZ=1.0, elecE=0.7,
                 surfaces=[O.Surface("homeotropic", 4.0), O.Surface("homeotropic", 4.0)]),
    "unmasked": dict(nx=8, ny=6, nz=10, potential="ghrl", k33=2.0, elecA=1.0, elecZ=1.0, elecE=0.7),
}


@pytest.mark.parametrize("name", list(SMALL))
def test_every_form_measures_the_same(name, monkeypatch):
    monkeypatch.setitem(MODELS, name, SMALL[name])
    ref = _run(name, "direct")
    for kind, shape in (("march", None), ("march", (64, 0)), ("resident", None), ("march_persistent", (128, 4))):
        _same(ref, _run(name, kind, shape))


def test_default_form_follows_the_smallest_replica():
    small, large = mcx.replica(nx=8, ny=8, nz=8), mcx.replica(nx=24, ny=24, nz=24)
    for descs, kind in (([small], "march"), ([large, small], "march"), ([large], "resident")):
        with mcx.Engine(descs) as eng:
            assert eng.pass_kind == kind

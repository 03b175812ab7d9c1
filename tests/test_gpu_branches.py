"""The equation of motion on three streams (td_device) against the same launches in
one row, which a profiled context takes: every kernel sums in a fixed order, so the
two agree bit for bit.  Repeated, on fresh states, so that a missing dependency
between the branches has chances to show; captured in the step's graph and not.
"""
import numpy as np
import pytest

from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu

SYSTEMS = {"helium": (100, (1, 1), (4, 4), True), "two types": (20, (2, 1), (4, 3), False),
           "one type": (60, (4,), (9,), False), "one orbital": (4, (1, 1), (1, 1), True)}


def _spec(name):
    n_el, bodies, orbs, restricted = SYSTEMS[name]
    sp = S.helium_fedvr(n_el, 6, 1, laser=S.sin2_pulse(0.05), restricted=restricted)
    sp.xmin, sp.xmax = -float(n_el), float(n_el)
    sp.n_bodies, sp.n_orbs = bodies, orbs
    sp.masses, sp.stats = (1.0,) * len(bodies), "f" * len(bodies)
    return sp


def _state(sp, x, w, seed):
    rng = np.random.default_rng(seed)
    c = rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs)
    return I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, x, w, seed))


@pytest.mark.parametrize("precision", ["fp64", "mixed_fx", "mixed_fx6"])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_branches_equal_the_row(name, precision):
    from codyfortran_gb300.engine import Engine
    sp = _spec(name)
    e, row = Engine(sp, precision=precision), Engine(sp, precision=precision)
    row.profile_begin("vector")
    for seed in range(8):
        st = _state(sp, e.x, e.w, seed)
        for which in ("full", "nonlin"):
            assert np.array_equal(e.time_derivative(st, 3.0, which), row.time_derivative(st, 3.0, which)), (seed, which)
    for x in (e, row):
        x.upload(st)
        x.propagate_resident(1.0, 0.02, 6, 6, use_graph=True)
    assert np.array_equal(e.download(), row.download())
    row.profile_end()
    e.close()
    row.close()

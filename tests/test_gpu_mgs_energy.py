"""Modified Gram-Schmidt by a cluster (k_mgs2_cluster) and by one block where the
columns do not fit its shared memory, and the energy over several blocks, against
the oracle.

Grids smaller than the cluster, with a remainder, and beyond the fit; one column
and more columns than grid points of a block.  Columns of random numbers: their
condition stays below a hundred, and two sweeps leave 2^-53 times it, 1e-13 with
room for the sums of 14001 points.  The energy's 18^4 terms of size up to one
in FP64: 1e-11 of its value.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu




@pytest.mark.parametrize("n_el,m", [(1, 1), (1, 4), (2, 3), (100, 4), (100, 16), (600, 9), (1400, 9), (1400, 16)])
def test_orthonormalize_matches_the_oracle(n_el, m):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(n_el, 6, m)
    sp.xmin, sp.xmax = -float(n_el), float(n_el)
    sp.has_interaction = n_el <= 600
    o, e = Oracle(sp), Engine(sp)
    rng = np.random.default_rng(m)
    f = np.asfortranarray(rng.normal(size=(o.nG, m)) + 1j * rng.normal(size=(o.nG, m)))
    got, want = e.orthonormalize(f), o.orthonormalize(f)
    e.close()
    s = (got.conj().T * o.w) @ got
    print(f"{o.nG} x {m}: {np.abs(got - want).max() / np.abs(want).max():.1e}, overlap {np.abs(s - np.eye(m)).max():.1e}")
    assert np.abs(got - want).max() < 1e-13 * np.abs(want).max()
    assert np.abs(s - np.eye(m)).max() < 1e-13


@pytest.mark.parametrize("bodies,orbs", [((1, 1), (2, 2)), ((1, 1), (3, 3)), ((2, 1), (6, 5)), ((3,), (18,))])
def test_energy_matches_the_oracle(bodies, orbs):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(10, 6, 1, restricted=False)
    sp.xmin, sp.xmax = -10.0, 10.0
    sp.n_bodies, sp.n_orbs = bodies, orbs
    sp.masses, sp.stats = (1.0,) * len(bodies), "f" * len(bodies)
    o, e = Oracle(sp), Engine(sp)
    rng = np.random.default_rng(sum(orbs))
    c = rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs)
    st = I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, o.x, o.w, 1))
    got, want = e.energy(st), o.energy(st)
    e.close()
    print(f"{bodies} in {orbs}: {abs(got - want) / abs(want):.1e}")
    assert abs(got - want) < 1e-11 * abs(want)

"""H.C with the singles of two body types on both sides of the 32 entries that the
lanes of a warp hold (k_ci_apply: the pairs over all lanes, else lane by lane),
against the oracle's traversal.

The sums have at most 34 x 34 products of entries below one in size with h2 scaled
to 1e-1: 1156 2^-53 < 2e-13 of the largest possible sum covers any order.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies,orbs", [((1, 1), (4, 4)), ((1, 2), (3, 17)), ((1, 2), (3, 18)), ((2, 1), (18, 2)),
                                         ((1, 1, 2), (2, 2, 18))])
def test_inter_type_pairs_match_the_oracle(bodies, orbs):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(4, 6, 1, restricted=False)
    sp.xmin, sp.xmax = -4.0, 4.0
    sp.n_bodies, sp.n_orbs = bodies, orbs
    sp.masses, sp.stats = (1.0,) * len(bodies), "f" * len(bodies)
    rng = np.random.default_rng(sum(orbs))
    c = rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs)
    c /= np.linalg.norm(c)
    n = sum(orbs)
    h = 0.1 * (rng.uniform(-1, 1, size=(n,) * 4) + 1j * rng.uniform(-1, 1, size=(n,) * 4))
    h2 = np.asfortranarray(h + h.conj().transpose(2, 3, 0, 1))
    o, e = Oracle(sp), Engine(sp)
    got, want = e.apply_h2(c, h2), o.apply_h2(c, h2)
    e.close()
    print(f"{bodies} in {orbs}: {np.abs(got - want).max():.1e} of {np.abs(want).max():.1e}")
    assert np.abs(got - want).max() < 2e-13

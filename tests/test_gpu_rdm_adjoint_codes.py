"""Density matrices summed over the orbital codes up to their adjoints
(k_ci_rdm_codes, k_ci_rdm_pairs and their double-float forms), against the
oracle's traversal over every code.

One to three body types of equal and unequal counts, one body, all orbitals but
one filled, a single orbital (no excitation but the diagonal), a CI vector
beyond the shared memory.  The sums of products of a normalised vector have at
most nC <= 8008 terms with absolute values summing to at most one: 8008 2^-53 <
1e-12 covers any order in FP64; the double-float sums hold 47 bits, 2^-43 after
the terms' roundings.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu

SYSTEMS = [((1, 1), (3, 3)), ((3, 2), (4, 4)), ((2, 1), (3, 5)), ((1, 1), (1, 1)), ((3,), (7,)), ((1,), (5,)),
           ((1, 2, 1), (2, 3, 3)), ((6,), (16,))]


@pytest.mark.parametrize("precision", ["fp64", "mixed_fx"])
@pytest.mark.parametrize("bodies,orbs", SYSTEMS)
def test_rdms_match_the_oracle(bodies, orbs, precision):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(4, 6, 1, restricted=False)
    sp.xmin, sp.xmax = -4.0, 4.0
    sp.n_bodies, sp.n_orbs = bodies, orbs
    sp.masses, sp.stats = (1.0,) * len(bodies), "f" * len(bodies)
    rng = np.random.default_rng(sum(orbs))
    c = rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs)
    c /= np.linalg.norm(c)
    o, e = Oracle(sp), Engine(sp, precision=precision)
    tol = 1e-12 if precision == "fp64" else 2.0 ** -43
    r1, r2 = e.rdm1(c), e.rdm2(c)
    e.close()
    d1, d2 = np.abs(r1 - o.rdm1(c)).max(), np.abs(r2 - o.rdm2(c)).max()
    print(f"{precision} {bodies} in {orbs}: rdm1 {d1:.1e} rdm2 {d2:.1e}")
    assert d1 < tol and d2 < tol

"""The coefficients' projector by one block and in two launches, against numpy: one
determinant, more than a block's threads, and both sides of the limit of 512.

dC - C <C, dC> with |C| = 1: sums of at most 2380 products, 2380 2^-53 < 3e-13 of |dC|.
"""
import numpy as np
import pytest

from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies,orbs", [(1, 1), (1, 16), (2, 24), (3, 24), (4, 16), (2, 32), (4, 17)])
def test_projector(bodies, orbs):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(8, 6, 1, restricted=False)
    sp.xmin, sp.xmax = -8.0, 8.0
    sp.n_bodies, sp.n_orbs, sp.masses, sp.stats = (bodies,), (orbs,), (1.0,), "f"
    rng = np.random.default_rng(orbs)
    c, d = (rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs) for _ in range(2))
    c, d = c / np.linalg.norm(c), d / np.linalg.norm(d)
    e = Engine(sp)
    got = e.project_coeffs(d, c)
    e.close()
    print(sp.n_coeffs, np.abs(got - (d - c * np.vdot(c, d))).max())
    assert np.abs(got - (d - c * np.vdot(c, d))).max() < 3e-13

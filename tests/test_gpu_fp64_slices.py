"""The FP64 form's contractions on digit slices against the oracle.

Grids around the edges of the kernels: below one 64-wide K block, at and past
one K = 256 accumulation chunk and at several, one orbital up to several
column tiles, two body types with their own orbitals, orbitals of very
different magnitude.  rho1 is the identity and rho2 random, so that rho^-1
adds no rounding of its own (a random CI vector's rho1 may be ill-conditioned,
and two eigensolvers then differ by more than the contractions).

Tolerance: the slices hold 55 bits of a row's maximum and a sum rounds once, so
the GPU result is within about 2^-53 of the exact product of the rounded
operands; the oracle's serial sums of up to 1281 terms carry sqrt(1281) 2^-53 =
4e-15 of their largest partial sum.  2e-14 leaves a factor five.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu
TOL = 2e-14


def _spec(n_el, m, spins=2):
    sp = S.helium_fedvr(n_el, 6, m, restricted=spins == 2)
    sp.xmin, sp.xmax = -0.5 * n_el, 0.5 * n_el
    if spins == 1:
        sp.n_bodies, sp.n_orbs, sp.masses, sp.stats = (2,), (m,), (1.0,), "f"
    return sp


def _check(sp, orbs, seed, tol=TOL):
    from codyfortran_gb300.engine import Engine
    o, e = Oracle(sp), Engine(sp)
    rng = np.random.default_rng(seed)
    r1 = np.eye(o.nO, dtype=complex)
    r2 = rng.normal(size=(o.nO,) * 4) + 1j * rng.normal(size=(o.nO,) * 4)
    d, h2 = e.apply_correlation_op(orbs, r1, r2, 0.0)
    dr, h2r = o.apply_correlation_op(orbs, r1, r2, 0.0)
    f2 = e.fill_h2(orbs, 0.0)
    e.close()
    assert np.linalg.norm(d - dr) <= tol * np.linalg.norm(dr)
    assert np.linalg.norm(h2 - h2r) <= tol * np.linalg.norm(h2r)
    assert np.linalg.norm(f2 - h2r) <= tol * np.linalg.norm(h2r)


@pytest.mark.parametrize("n_el,m,spins", [(1, 2, 2), (12, 1, 2), (13, 4, 2), (51, 5, 2), (52, 8, 2), (102, 9, 2),
                                          (103, 3, 1), (256, 12, 2), (41, 16, 1)])
def test_grid_and_column_edges(n_el, m, spins):
    sp = _spec(n_el, m, spins)
    o = Oracle(sp)
    _check(sp, I.seeded_gaussian_orbitals(sp, o.x, o.w, m), n_el)


def test_unrestricted_orbitals():
    sp = _spec(30, 4)
    sp.restricted = False
    o = Oracle(sp)
    _check(sp, I.seeded_gaussian_orbitals(sp, o.x, o.w, 5), 6)


@pytest.mark.parametrize("scale", [1e-60, 1e60])
def test_magnitudes(scale):
    """Each row has its own power of two: a common factor leaves the relative error unchanged."""
    sp = _spec(30, 4)
    o = Oracle(sp)
    _check(sp, scale * I.seeded_gaussian_orbitals(sp, o.x, o.w, 5), 7)


def test_zero_orbital_and_nan():
    from codyfortran_gb300.engine import Engine
    sp = _spec(30, 4)
    o = Oracle(sp)
    orbs = I.seeded_gaussian_orbitals(sp, o.x, o.w, 5)
    orbs[:, 2] = 0.0
    _check(sp, orbs, 8)
    # a NaN reaches every mean-field column, as it does in a sum
    e = Engine(sp)
    c = np.ones(e.nC, dtype=complex) / np.sqrt(e.nC)
    bad = orbs.copy()
    bad[10, 1] = np.nan
    d, h2 = e.apply_correlation_op(bad, e.rdm1(c), e.rdm2(c), 0.0)
    assert np.isnan(d).all() and np.isnan(h2).any()
    # and the context is usable afterwards
    d, _ = e.apply_correlation_op(orbs, e.rdm1(c), e.rdm2(c), 0.0)
    assert np.isfinite(d).all()
    e.close()

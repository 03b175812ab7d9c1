"""Output widths of the fixed-point contractions.

The MMA of a digit slice spans the tile columns of several slices and is cut
into one or two instructions of at most 256 columns; the columns of a system
are spread over equal tiles.  One to thirteen orbitals give 2 to 182 pair
columns and 2 to 338 mean-field columns: below one 16-column unit, exactly one
tile, just past it, several tiles.

Tolerance: 2^-30 / 2^-36 of the operands' row maxima (30 / 36 digit bits),
times the 60 by which a sum over the grid may exceed its terms' rounding, is
6e-8 / 9e-10 of the result.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu
TOL = {"mixed_fx": 6e-8, "mixed_fx6": 9e-10}


@pytest.mark.parametrize("precision", sorted(TOL))
@pytest.mark.parametrize("m", [1, 2, 3, 5, 6, 8, 9, 11, 13])
def test_mean_field_and_h2_widths(m, precision):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(27, 6, m)
    sp.xmin, sp.xmax = -27.0, 27.0
    o, e = Oracle(sp), Engine(sp, precision=precision)
    rng = np.random.default_rng(m)
    c = rng.normal(size=o.nC) + 1j * rng.normal(size=o.nC)
    c /= np.linalg.norm(c)
    orbs = I.seeded_gaussian_orbitals(sp, o.x, o.w, m)
    r1, r2 = o.rdm1(c), o.rdm2(c)
    d, h2 = e.apply_correlation_op(orbs, r1, r2, 0.0)
    dr, h2r = o.apply_correlation_op(orbs, r1, r2, 0.0)
    assert np.linalg.norm(d - dr) < TOL[precision] * np.linalg.norm(dr)
    assert np.linalg.norm(h2 - h2r) < TOL[precision] * np.linalg.norm(h2r)
    e.close()

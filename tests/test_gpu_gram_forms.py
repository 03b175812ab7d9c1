"""The weighted Gram matrix (k_gram_partial, k_gram_partial_df) where its forms
change: one block, blocks whose last sums, partials for k_gram_final; one lane to
32 lanes an entry.  FillH1 of random orbitals against the oracle.

A sum over nG <= 3001 points in FP64: 3001 2^-53 = 4e-13 of its largest possible
value, the norm of h phi, which the oracle's own h1 of these orbitals bounds from
below by less than ten; the double-float sums hold 2^-43.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed_fx"])
@pytest.mark.parametrize("n_el,m", [(1, 1), (2, 2), (20, 1), (100, 4), (100, 9), (600, 5), (120, 16), (40, 17)])
def test_h1_matches_the_oracle(n_el, m, precision):
    from codyfortran_gb300.engine import Engine
    sp = S.helium_fedvr(n_el, 6, m)
    sp.xmin, sp.xmax = -float(n_el), float(n_el)
    o, e = Oracle(sp), Engine(sp, precision=precision)
    orbs = I.seeded_gaussian_orbitals(sp, o.x, o.w, 3)
    got, want = e.fill_h1(orbs, 0.3), o.fill_h1(orbs, 0.3)
    e.close()
    err = np.abs(got - want).max() / np.abs(want).max()
    print(f"{precision} {o.nG} points, {m} orbitals: {err:.1e}")
    assert err < (4e-12 if precision == "fp64" else 10 * 2.0 ** -43)

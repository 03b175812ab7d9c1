"""CI kernels of a context after another context with a shorter CI vector has been set up.

Both vectors lie in shared memory and need more than the default limit, which is a
property of the kernel, not of the context.  Products and density matrices against the
oracle: at most 4356 x 144 terms of a normalised vector and h2 entries of size 0.1, 1e-11
absolute covers any order of the FP64 sums.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


def _spec(n, m):
    sp = S.helium_fedvr(4, 6, m)
    sp.xmin, sp.xmax, sp.n_bodies = -4.0, 4.0, (n, n)
    return sp


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed_fx", 2.0 ** -36)])
def test_a_smaller_context_beside(precision, tol):
    from codyfortran_gb300.engine import Engine
    sp = _spec(2, 12)
    e, o = Engine(sp, precision), Oracle(sp)
    small = Engine(_spec(3, 8), precision)
    assert (e.nC, small.nC) == (4356, 3136)
    rng = np.random.default_rng(0)
    c = rng.normal(size=e.nC) + 1j * rng.normal(size=e.nC)
    c /= np.linalg.norm(c)
    h = 0.05 * (rng.uniform(-1, 1, size=(24,) * 4) + 1j * rng.uniform(-1, 1, size=(24,) * 4))
    h2 = np.asfortranarray(h + h.conj().transpose(2, 3, 0, 1))
    got, r1 = e.apply_h2(c, h2), e.rdm1(c)
    e.close()
    small.close()
    assert np.abs(got - o.apply_h2(c, h2)).max() < tol
    assert np.abs(r1 - o.rdm1(c)).max() < tol

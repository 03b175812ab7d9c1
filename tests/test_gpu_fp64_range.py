"""The FP64 form's contractions over the range of a double.

* All orbitals times 2^k: every row has its own power of two, so the integrals are those of
  the unscaled orbitals times 2^4k and the mean field times 2^3k, bit for bit.
* Each orbital times a power of two of its own: the integrals scale bit for bit; the mean
  field, whose sums then run over pairs of very different size, is within 24 units of 2^-53
  of the sum of its terms' sizes (as in tests/test_gpu_fp64_precision.py).
* Results below the smallest normal number keep what a subnormal holds (operands there count
  as zero).

Entries below 2^-200 of the largest are left out: at k = -200 they underflow.
"""
import numpy as np
import pytest

from test_gpu_fp64_precision import UNIT, _exact, _orbitals, _spec

pytestmark = pytest.mark.gpu
SIZES = [(4, 4.0, 1.0, 2), (51, 100.0, 1.0, 4), (100, 100.0, 0.01, 3)]


def _run(e, F, r2):
    n = F.shape[1]
    d, h2 = e.apply_correlation_op(F, np.eye(2 * n, dtype=complex), r2, 0.0)
    assert np.array_equal(h2, e.fill_h2(F, 0.0))
    return d, h2[:n, :n, :n, :n]


def _engine(n_el, box, soft, n):
    from codyfortran_gb300.engine import Engine
    sp = _spec(n_el, box, soft, n)
    e = Engine(sp)
    assert e.contraction_slices() > 0
    rng = np.random.default_rng(n_el)
    r2 = np.asfortranarray(rng.normal(size=(2 * n,) * 4) + 1j * rng.normal(size=(2 * n,) * 4))
    return sp, e, _orbitals("compact", e.x, e.w, n, rng), r2


def _same(got, want):
    big = np.abs(want) > 2.0**-200 * np.max(np.abs(want))
    return big.any() and np.array_equal(got[big], want[big])


@pytest.mark.parametrize("k", [-200, -60, 60, 200])
@pytest.mark.parametrize("size", SIZES)
def test_a_common_factor(size, k):
    sp, e, F, r2 = _engine(*size)
    d, h = _run(e, F, r2)
    ds, hs = _run(e, F * 2.0**k, r2)
    e.close()
    assert _same(ds, d * 2.0 ** (3 * k)) and _same(hs, h * 2.0 ** (4 * k))


@pytest.mark.parametrize("size", SIZES)
def test_factors_of_their_own(size):
    sp, e, F, r2 = _engine(*size)
    n = F.shape[1]
    k = np.array([0, -90, 60, -30])[:n]
    d, h = _run(e, F, r2)
    ds, hs = _run(e, F * 2.0**k, r2)
    e.close()
    f = 2.0**k
    assert _same(hs, h * f[:, None, None, None] * f[:, None, None] * f[:, None] * f)
    P, W, A = _exact(sp, e.x, e.w, F * f)
    spins = (slice(0, n), slice(n, 2 * n))
    R = sum(r2[a, b, a, b].astype(np.clongdouble) for a in spins for b in spins)
    R = R * (np.longdouble(2) / (np.longdouble(4) + np.longdouble(1e-10)))

    def field(W, R, F):
        return np.einsum("xk,xkj->xj", F, (W @ R.transpose(3, 1, 0, 2).reshape(n * n, n * n)).reshape(-1, n, n))
    want, size = field(W, R, (F * f).astype(np.clongdouble)), field(A, np.abs(R).astype(float), np.abs(F * f))
    ok = size > 1e-200
    worst = float(np.max(np.abs(ds - want).astype(float)[ok] / size[ok])) / UNIT
    print(f"{worst:.1f} units")
    assert worst <= 24.0


@pytest.mark.parametrize("size", SIZES)
def test_subnormal_results(size):
    """Integrals times 2^-1040 (orbitals times 2^-260): the result's rounding and the scaled
    reference's, and two for the sum of K splits.  A mean field times 2^-1055 (rho2 times 2^-950,
    orbitals times 2^-35): one unit of Z, times an orbital below one, for each of four
    orbitals, a product and a sum each, the reference's: at most 16."""
    sp, e, F, r2 = _engine(*size)
    d, h = _run(e, F, r2)
    n = F.shape[1]
    _, hs = _run(e, F * 2.0**-260, r2)
    ds, _ = _run(e, F * 2.0**-35, r2 * 2.0**-950)
    e.close()
    least = 2.0**-1074
    assert np.max(np.abs(hs - h * 2.0**-1040)) <= 4 * least and np.any(hs != 0.0)
    assert np.max(np.abs(ds - d * 2.0**-1055)) <= 16 * least and np.any(ds != 0.0)

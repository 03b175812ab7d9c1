"""The FP64 form's contractions, entry by entry, against extended precision.

In each entry, (l1 l2 | k1 k2), the error is measured in units of 2^-53 of the sum of the
terms' sizes, over x and y |S_l1k1(x)| V(x, y) |S_l2k2(y)|, however small it is beside other
entries.  V's formula takes three roundings, S's two products three, W, the product and the
result one each; twelve units cover them and the losses of the digit slices, which are chosen
to stay below (orbitals far apart and a short softening are what they lose most on: 108 and
14000 units with seven slices).  The slices' sums do not round; on the FP64 pipe (a range of V
that slices do not suit) two sums of all points in order may lose a unit a term.
"""
import numpy as np
import pytest

from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu
UNIT = 2.0**-53


def _spec(n_el, box, soft, n):
    sp = S.helium_fedvr(n_el, 6, n)
    sp.xmin, sp.xmax, sp.int_s1 = -box, box, soft
    return sp


def _orbitals(kind, x, w, n, rng):
    far = 0.8 * x[-1] * np.where(np.arange(n) % 2, 1.0, -1.0)
    c = {"compact": rng.uniform(-2.5, 2.5, n), "apart": far, "spread": np.zeros(n)}[kind]
    s = np.full(n, x[-1] / 3) if kind == "spread" else rng.uniform(0.5, 2.5, n)
    f = np.exp(-((x[:, None] - c) ** 2) / (2 * s**2)) * np.exp(1j * rng.uniform(-1, 1, n) * x[:, None])
    r = np.sqrt(w)[:, None]
    return np.asfortranarray(np.linalg.qr((f * (rng.normal(size=n) + 1j * rng.normal(size=n))) * r)[0] / r)


def _exact(sp, x, w, F):
    """W and |S| V of every pair (x, l, k), and S, in extended precision."""
    n, nG = F.shape[1], len(x)
    V = (1.0 / np.sqrt(((x[:, None] - x[None, :]) ** 2).astype(np.longdouble) + np.longdouble(sp.int_s1) ** 2))
    Fq = F.astype(np.clongdouble)
    P = (Fq.conj()[:, :, None] * Fq[:, None, :] * w.astype(np.longdouble)[:, None, None]).reshape(nG, n * n)
    W = (V @ P.real) + 1j * (V @ P.imag)
    A = V.astype(float) @ np.abs(P).astype(float)
    return P, W, A


# range of V up to 2^10 (eight slices), up to 2^16 (nine), beyond (FP64 pipe); grids below one
# chunk of 128 points, at its edges and of several with splits; up to 45 pairs (column tiles of 48)
CASES = [(4, 4.0, 1.0, 2, 8), (25, 25.0, 1.0, 3, 8), (26, 26.0, 0.5, 3, 8), (51, 100.0, 1.0, 3, 8), (100, 100.0, 1.0, 4, 8),
         (100, 100.0, 0.1, 3, 9), (100, 100.0, 0.01, 3, 9), (25, 25.0, 0.002, 3, 9), (100, 100.0, 0.001, 3, 0),
         (30, 60.0, 0.05, 6, 9), (52, 60.0, 0.05, 9, 9), (512, 400.0, 0.1, 2, 9)]


@pytest.mark.parametrize("kind", ["compact", "apart", "spread"])
@pytest.mark.parametrize("n_el,box,soft,n,slices", CASES)
def test_integrals_entry_by_entry(n_el, box, soft, n, slices, kind):
    from codyfortran_gb300.engine import Engine
    sp = _spec(n_el, box, soft, n)
    e, m = Engine(sp), Engine(sp, "mixed_fx")
    assert e.contraction_slices() == slices
    F = _orbitals(kind, e.x, e.w, n, np.random.default_rng(n_el))
    P, W, A = _exact(sp, e.x, e.w, F)
    want = (P.T @ W / 2).reshape((n,) * 4).transpose(0, 2, 1, 3)
    size = (np.abs(P).astype(float).T @ A / 2).reshape((n,) * 4).transpose(0, 2, 1, 3)
    one = np.eye(2 * n, dtype=complex)
    got = {"fill_h2": e.fill_h2(F, 0.0), "correlation": e.apply_correlation_op(F, one, np.zeros((2 * n,) * 4, complex), 0.0)[1],
           "mixed_fx fill_h2": m.fill_h2(F, 0.0)}
    nG = e.nG
    e.close()
    m.close()
    for name, h2 in got.items():
        err = np.abs(h2[:n, :n, :n, :n] - want).astype(float)
        ok = size > 1e-250  # below, a term underflows
        worst = float(np.max(err[ok] / size[ok])) / UNIT
        print(f"{name} {nG} points, softening {soft}, {kind}: {worst:.1f} units")
        assert worst <= (12.0 if slices else 2.0 * nG), name
        assert np.all(err[~ok] <= 1e-250)


@pytest.mark.parametrize("kind", ["compact", "apart"])
@pytest.mark.parametrize("weight", [1.0, 1e-12, 1e-30])
@pytest.mark.parametrize("n_el,box,soft,n", [(4, 4.0, 1.0, 2), (51, 100.0, 1.0, 3), (100, 100.0, 1.0, 4), (100, 100.0, 0.01, 3),
                                             (30, 60.0, 0.05, 6), (30, 60.0, 1.0, 9)])
def test_mean_field_entry_by_entry(n_el, box, soft, n, weight, kind):
    """dphi_j(x) in units of the sum of the sizes of its terms.  The coefficients of the pairs
    of orbitals on one side are small, so that with the sides far apart the sum lies in pairs
    whose potentials are 1e-17 of the others'.  V and S six roundings, W one, rho2's spin blocks three, rho^-1 of a
    multiple of the identity four, R'' two, the product one, the sum over the orbitals n + 1: 24.
    """
    from codyfortran_gb300.engine import Engine
    sp = _spec(n_el, box, soft, n)
    e = Engine(sp)
    rng = np.random.default_rng(n_el)
    F = _orbitals(kind, e.x, e.w, n, rng)
    P, W, A = _exact(sp, e.x, e.w, F)
    r2 = rng.normal(size=(2 * n,) * 4) + 1j * rng.normal(size=(2 * n,) * 4)
    o = np.arange(2 * n) % n
    r2 = np.asfortranarray(r2 * np.where((o[None, :, None, None] - o[None, None, None, :]) % 2 == 0, weight, 1.0))
    d, _ = e.apply_correlation_op(F, np.eye(2 * n, dtype=complex), r2, 0.0)
    e.close()
    spins = (slice(0, n), slice(n, 2 * n))
    R = sum(r2[a, b, a, b].astype(np.clongdouble) for a in spins for b in spins)
    R = R * (np.longdouble(2) / (np.longdouble(4) + np.longdouble(1e-10)))  # rho1 = 2, regularised

    def field(W, R, F):
        Z = W @ R.transpose(3, 1, 0, 2).reshape(n * n, n * n)  # (l2 k2) -> (k1 j)
        return np.einsum("xk,xkj->xj", F, Z.reshape(-1, n, n))
    want, size = field(W, R, F.astype(np.clongdouble)), field(A, np.abs(R).astype(float), np.abs(F))
    ok = size > 1e-250
    worst = float(np.max(np.abs(d - want).astype(float)[ok] / size[ok])) / UNIT
    print(f"{n_el} elements, softening {soft}, weight {weight}, {kind}: {worst:.1f} units")
    assert worst <= 24.0

"""The regularised inverse of rho1 inside ApplyCorrelationOp.

R' = rho2 x rho^-1 is read off the mean field of a system whose interaction is
constant (one softening length far above the box), so that every pair potential
is V0 <phi_l|phi_k> = V0 delta_lk and dphi_j = V0 sum_k phi_k sum_l R(k, l, j, l).
rho1 has prescribed occupations from 1 down to 0 in a random basis, for 1 to 32
orbitals.

Tolerance: an occupation n carries an absolute rounding of a few 2^-53 ||rho||
in any algorithm, which f(n) = n / (n^2 + 1e-10) turns into |f'(n)| of it; the
check is 40 2^-53 max(|f'|, |f|) ||rho|| ||rho2|| n, against the mean field from
numpy's eigenvectors.
"""
import numpy as np
import pytest

from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 8, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("kind", ["spread", "small", "degenerate", "zero"])
def test_mean_field_of_a_constant_interaction(n, kind):
    from codyfortran_gb300.engine import Engine
    soft = 1e9
    sp = S.SystemSpec(grid_kind="fedvr", xmin=-8.0, xmax=8.0, n_elements=16, n_locals=6, n_bodies=(1,), n_orbs=(n,),
                      masses=(1.0,), stats="f", nuclei=[S.Nucleus(0.0, 1.0)], int_strength=soft, int_s1=soft,
                      int_kind="dense")
    e = Engine(sp)
    rng = np.random.default_rng(n)
    occ = {"spread": np.linspace(1.0, 0.1, n), "small": 10.0 ** -np.linspace(0.0, 6.0, n),
           "degenerate": np.repeat([1.0, 0.25], n)[:n] if n < 2 else np.r_[np.full(n // 2, 0.5), np.full(n - n // 2, 0.25)],
           "zero": np.r_[1.0, np.zeros(n - 1)]}[kind]
    U = np.linalg.qr(rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))[0]
    r1 = (U * occ) @ U.conj().T
    r1 = 0.5 * (r1 + r1.conj().T)
    r2 = rng.normal(size=(n,) * 4) + 1j * rng.normal(size=(n,) * 4)
    F = np.linalg.qr(rng.normal(size=(e.nG, n)) + 1j * rng.normal(size=(e.nG, n)))[0] / np.sqrt(e.w)[:, None]
    d, _ = e.apply_correlation_op(F, r1, r2, 0.0)
    e.close()
    w, V = np.linalg.eigh(r1)
    f = w / (w * w + 1e-10)
    M = (V * f) @ V.conj().T
    S_ = (F.conj() * e.w[:, None]).T @ F  # the identity to rounding
    R = np.einsum("abkd,kj->abjd", r2, M)
    ref = F @ np.einsum("kbjl,lb->kj", R, S_)
    slope = np.max(np.abs((1e-10 - w * w) / (w * w + 1e-10) ** 2))
    tol = 40 * 2.0**-53 * max(slope, np.max(np.abs(f))) * np.linalg.norm(r2) * n
    assert np.sqrt(np.sum(np.abs(d - ref) ** 2 * e.w[:, None])) <= tol

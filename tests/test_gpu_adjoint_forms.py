"""MCTDHF pulse gradient at the edges of its kernels, against the host restatement
of the adjoint (tests/adjoint_reference.py, FP64 numpy).

* Orbital counts from 1 to the largest, grids below and above the tiles of the
  pair potentials (16 points x 4 pairs) and of the pointwise kernels (4 points),
  segments of checkpoints that the backward sweep recomputes, and a second
  backward sweep after the first.  The CI matrix has singular values within a
  factor three, so rho^-1 amplifies rounding by less than ten: the bounds are
  those of the gradient's other checks, 1e-12 for the state and J and 1e-9 for
  the gradient.
* A Krylov space that holds the top of a fine grid's spectrum, where the
  exponential of the subspace is taken in several parts (|tau| R above 700).
  Phases of z = 2000 carry errors of z 2^-53 = 2e-13: ten times the bounds above.
  One step: a second one amplifies a change of the start by one unit in the last
  place to 2e-11 of the state in the host reference itself.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S
from adjoint_reference import Adjoint, Dense

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _system(n_el, m, half, field, dt):
    sp = S.helium_fedvr(n_el, 6, m, laser=S.Laser(kind="sampled", samples=field, sample_dt=dt, sample_t0=0.0))
    sp.xmin, sp.xmax = -half, half
    return sp


def _coeffs(m, rng):
    u, v = (np.linalg.qr(rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m)))[0] for _ in range(2))
    s = np.linspace(0.5, 1.5, m) if m > 1 else np.ones(1)
    return ((u * (s / np.linalg.norm(s))) @ v).T.reshape(-1)


def _reference(o, field, dt, K):
    X = o.x
    return Adjoint(Dense(o, 1.0 / np.sqrt((X[:, None] - X[None, :]) ** 2 + 1.0)), field, dt, K)


@pytest.mark.parametrize("n_el,m,K,chk", [(2, 1, 6, 1), (3, 2, 6, 2), (7, 5, 8, 64), (40, 8, 12, 2), (9, 16, 32, 3)])
def test_gradient_sizes(n_el, m, K, chk):
    from codyfortran_gb300.engine import Engine
    nT, dt = 3, 0.05
    rng = np.random.default_rng(n_el)
    field = rng.normal(0.0, 0.01, size=nT)
    sp = _system(n_el, m, float(n_el), field, dt)
    o, e = Oracle(sp), Engine(sp, max_krylov=K)
    st = I.pack_state(_coeffs(m, rng), I.seeded_gaussian_orbitals(sp, o.x, o.w, 5))
    Jr, Or, sNr, gr = _reference(o, field, dt, K).run(st, checkpoint=chk)
    J, ov, fin = e.mc_adjoint_forward(st, field, dt, krylov_dim=K, checkpoint=chk)
    g = e.mc_adjoint_backward()
    again = e.mc_adjoint_backward()
    e.close()
    print(f"state {rel(fin, sNr):.1e} J {abs(J - Jr):.1e} gradient {rel(g, gr):.1e}")
    assert abs(J - Jr) < 1e-12
    assert rel(fin, sNr) < 1e-12
    assert rel(g, gr) < 1e-9
    assert np.array_equal(g, again)


def test_gradient_exponential_in_parts():
    from codyfortran_gb300.engine import Engine
    nT, dt, K, n_el, m, half = 1, 0.25, 12, 60, 2, 3.0
    rng = np.random.default_rng(3)
    field = rng.normal(0.0, 0.01, size=nT)
    sp = _system(n_el, m, half, field, dt)
    o, e = Oracle(sp), Engine(sp, max_krylov=K)
    # two sines with a little of every frequency
    phi = np.stack([np.sin((i + 1) * np.pi * (o.x + half) / (2 * half)) for i in range(m)], axis=1).astype(complex)
    phi += 1e-3 * (rng.normal(size=phi.shape) + 1j * rng.normal(size=phi.shape))
    q = np.linalg.qr(np.sqrt(o.w)[:, None] * phi)[0]
    st = I.pack_state(_coeffs(m, rng), q / np.sqrt(o.w)[:, None])
    ref = _reference(o, field, dt, K)
    _, tape = ref.lanczos(st, ref.E(0.0)[0], 0.5 * dt)
    al, be = np.array(tape["al"]), np.abs(np.array(tape["be"][:K - 1]))
    r = np.concatenate([[0.0], be]) + np.concatenate([be, [0.0]])
    assert 0.5 * dt * 0.5 * ((al + r).max() - (al - r).min()) > 1400.0
    Jr, Or, sNr, gr = ref.run(st, checkpoint=2)
    J, ov, fin = e.mc_adjoint_forward(st, field, dt, krylov_dim=K, checkpoint=2)
    g = e.mc_adjoint_backward()
    e.close()
    print(f"state {rel(fin, sNr):.1e} J {abs(J - Jr):.1e} gradient {rel(g, gr):.1e}")
    assert abs(J - Jr) < 1e-11
    assert rel(fin, sNr) < 1e-11
    assert rel(g, gr) < 1e-8

"""The one-launch SIL against the oracle: piece sizes from below one block's
minimum to several per trajectory, every re-orthogonalisation window, uneven
batches (one block per trajectory and many), adaptive steps that converge at
once, halve the step and give up, a zero state, a Krylov space that breaks down.

Tolerance 1e-12 relative, the FP64 form's parity bound: both run the same
recurrence, whose rounding the unitary exponential does not amplify.
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


def _spec(n_el, n_locals, m, restricted=True):
    sp = S.helium_fedvr(n_el, n_locals, m, laser=S.sin2_pulse(0.05, omega=0.2, n_cycles=2.0), restricted=restricted)
    sp.xmin, sp.xmax = -0.5 * n_el, 0.5 * n_el
    return sp


def _state(sp, o, seed):
    rng = np.random.default_rng(seed)
    c = rng.normal(size=o.nC) + 1j * rng.normal(size=o.nC)
    return I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, o.x, o.w, seed))


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n_el,n_locals,m,restricted", [(1, 4, 1, True), (6, 6, 1, True), (13, 8, 2, True), (20, 6, 5, False),
                                                        (160, 6, 8, True), (300, 9, 12, True)])
@pytest.mark.parametrize("window", [0, 1, 3])
def test_fixed_order(n_el, n_locals, m, restricted, window):
    from codyfortran_gb300.engine import Engine
    sp = _spec(n_el, n_locals, m, restricted)
    o, e = Oracle(sp), Engine(sp, max_krylov=12, krylov_window=window)
    st = _state(sp, o, 3)
    mw = o.metric_weights()
    for k in (1, 2, 11):
        a = e.sil(st, 3.0, 3.01, k, metric=mw)
        b = o.sil(st, 3.0, 3.01, k, metric=mw)
        assert _rel(a, b) < 1e-12, k
    e.close()


@pytest.mark.parametrize("tol,restarts,dt", [(1e-4, 0, 0.01), (1e-11, 6, 0.05), (1e-13, 1, 0.2), (1e-11, 3, -0.05)])
def test_adaptive(tol, restarts, dt):
    from codyfortran_gb300.engine import Engine
    sp = _spec(30, 6, 3)
    o, e = Oracle(sp), Engine(sp, max_krylov=16)
    st = _state(sp, o, 4)
    a = e.sil(st, 2.0, 2.0 + dt, 14, tol=tol, max_restarts=restarts, metric=o.metric_weights())
    b = o.sil(st, 2.0, 2.0 + dt, 14, tol=tol, max_restarts=restarts, metric=o.metric_weights())
    assert _rel(a, b) < 1e-12
    e.close()


def test_zero_state_and_breakdown():
    from codyfortran_gb300.engine import Engine
    sp = _spec(6, 6, 2)
    o, e = Oracle(sp), Engine(sp, max_krylov=12)
    z = np.zeros(e.nS, dtype=complex)
    assert np.array_equal(e.sil(z, 0.0, 0.1, 8), z)
    c = z.copy()  # only coefficients: H v = 0, the Krylov space has one vector
    c[: e.nC] = 1.0
    assert _rel(e.sil(c, 0.0, 0.1, 8), o.sil(c, 0.0, 0.1, 8)) < 1e-12
    assert _rel(e.sil(c, 0.0, 0.1, 8, tol=1e-10, max_restarts=2), c) < 1e-12
    e.close()


@pytest.mark.parametrize("n,window,precision", [(3, 0, "fp64"), (40, 0, "fp64"), (40, 1, "mixed_fx6"), (151, 1, "fp64"),
                                                (153, 1, "fp64")])
def test_batches(n, window, precision):
    """Every trajectory of an uneven batch as it comes out of a context of its own."""
    from codyfortran_gb300.engine import Batch, Engine
    specs = []
    for k in range(n):
        sp = _spec(4 + 7 * (k % 9), 6, 1 + k % 4)
        specs.append(sp)
    b = Batch(specs, precision, max_krylov=8, krylov_window=window)
    states = [_state(sp, s, k) for k, (sp, s) in enumerate(zip(specs, b.systems))]
    b.upload(states)
    b.propagate(1.0, 0.02, 1, 8)
    got = b.download()
    for k in range(0, n, max(1, n // 5)):
        e = Engine(specs[k], precision, max_krylov=8, krylov_window=window)
        e.upload(states[k])
        e.propagate_resident(1.0, 0.02, 1, 8, use_graph=True)
        assert _rel(got[k], e.download()) < (1e-12 if precision == "fp64" else 1e-10)
        e.close()
    b.close()

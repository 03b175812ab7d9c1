"""The decisions of an adaptive SIL on the device: the count of sub-steps that did not
reach the tolerance, against the oracle's, and the bound on the work of one launch.

The tolerances (1e-9 at the smallest) lie far above the estimates' rounding, and an
estimate a tenth off decides at most one sub-step of a hundred otherwise.  States: 1e-12
relative, the FP64 form's parity bound, for each of the sub-steps.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import Oracle
from oracle import lib as oracle_lib
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


def _system(n_el=10, m=2):
    sp = S.helium_fedvr(n_el, 6, m, laser=S.sin2_pulse(0.05, omega=0.2, n_cycles=2.0))
    sp.xmin, sp.xmax = -0.5 * n_el, 0.5 * n_el
    o = Oracle(sp)
    rng = np.random.default_rng(n_el)
    c = rng.normal(size=o.nC) + 1j * rng.normal(size=o.nC)
    return sp, o, I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, o.x, o.w, 5))


def _engine_sil(e, state, dt, K, tol, restarts):
    s, w = state.copy(), C.c_int(-1)
    e._check(e.lib.cgpu_integrate_sil(e.h, 1, s.ctypes.data_as(C.c_void_p), C.c_double(2.0), C.c_double(2.0 + dt), K,
                                      C.c_double(tol), restarts, None, C.byref(w)))
    return s, w.value


def _oracle_sil(o, state, dt, K, tol, restarts):
    s = state.copy()
    return s, oracle_lib().orc_integrate_sil(o.h, 1, s.ctypes.data_as(C.c_void_p), C.c_double(2.0), C.c_double(2.0 + dt),
                                             K, C.c_double(tol), restarts, None)


def _sub_steps(dt, restarts):
    """Sub-steps of an integration that never converges."""
    n, rem = 0, dt
    while abs(rem) > 1e-14:
        d = rem
        for _ in range(restarts):
            if abs(d) <= 1e-14:
                break
            d *= 0.5
        rem -= d
        n += 1
    return n


def test_a_launch_is_bounded():
    """A tolerance that most sub-steps miss: hundreds of Krylov passes, of which a launch takes 64."""
    from codyfortran_gb300.engine import Engine
    sp, o, st = _system()
    e = Engine(sp, max_krylov=6)
    restarts = 3
    e.launch_count(reset=True)
    a, wa = _engine_sil(e, st, 0.2, 2, 1e-9, restarts)
    launches = e.launch_count()
    b, wb = _oracle_sil(o, st, 0.2, 2, 1e-9, restarts)
    e.close()
    print(wa, wb, "warnings,", launches, "launches", np.linalg.norm(a - b) / np.linalg.norm(b))
    assert wa == wb > 100
    assert launches >= wb * (restarts + 1) // 64
    assert np.linalg.norm(a - b) < _sub_steps(0.2, restarts) * 1e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("restarts", [0, 2])
def test_a_state_that_is_not_finite_does_not_converge(bad, restarts):
    from codyfortran_gb300.engine import Engine
    sp, o, st = _system()
    e = Engine(sp, max_krylov=6)
    st[o.nC + 7] = bad
    a, w = _engine_sil(e, st, 0.01, 6, 1e-7, restarts)
    assert w == _sub_steps(0.01, restarts)
    assert np.isnan(a).all()
    # and the context is usable afterwards
    sp, o, st = _system()
    a, w = _engine_sil(e, st, 0.01, 6, 1e-7, 4)
    b, wb = _oracle_sil(o, st, 0.01, 6, 1e-7, 4)
    e.close()
    assert w == wb
    assert np.linalg.norm(a - b) < 1e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("K,tol,restarts,dt", [(2, 1e-7, 0, 0.05), (3, 1e-7, 2, 0.2), (6, 1e-7, 6, 0.05), (6, 1e-3, 0, 0.001)])
def test_warnings_are_the_oracles(K, tol, restarts, dt):
    from codyfortran_gb300.engine import Engine
    sp, o, st = _system()
    e = Engine(sp, max_krylov=6)
    a, wa = _engine_sil(e, st, dt, K, tol, restarts)
    b, wb = _oracle_sil(o, st, dt, K, tol, restarts)
    e.close()
    print(wa, wb)
    assert wa == wb
    assert np.linalg.norm(a - b) < (1 + wb) * 1e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("dt", [0.1, 1.0, 2.0, -3.0])
@pytest.mark.parametrize("tol", [0.0, 1e-9])
def test_one_krylov_vector(dt, tol):
    """A spectrum of no width, whatever the step: the Krylov order 1, and a state of
    coefficients alone (H v = 0, a breakdown at once)."""
    from codyfortran_gb300.engine import Engine
    sp, o, st = _system()
    e = Engine(sp, max_krylov=6)
    a, _ = _engine_sil(e, st, dt, 1, tol, 0)
    b, _ = _oracle_sil(o, st, dt, 1, tol, 0)
    assert np.linalg.norm(a - b) < 1e-12 * np.linalg.norm(b)
    st[o.nC:] = 0.0
    a, w = _engine_sil(e, st, dt, 6, tol, 0)
    e.close()
    assert np.linalg.norm(a - st) < 1e-12 * np.linalg.norm(st) and (tol == 0.0 or w == 0)


def test_a_split_step_whose_sil_takes_several_launches():
    """The step is issued in one piece and taken again, part by part, where a SIL half did not end
    within a launch: hundreds of sub-steps against the oracle, then a step that ends at once."""
    from codyfortran_gb300.engine import Engine
    sp, o, st = _system()
    e = Engine(sp, max_krylov=6)
    for dt, K, tol, restarts in [(0.2, 2, 1e-9, 3), (0.01, 6, 1e-7, 4)]:
        a = e.propagate_split2(st, 2.0, 2.0 + dt, K, tol, restarts)
        b = o.propagate_split2(st, 2.0, 2.0 + dt, K, tol, restarts)
        print(dt, np.linalg.norm(a - b) / np.linalg.norm(b))
        assert np.linalg.norm(a - b) < _sub_steps(dt, restarts) * 1e-12 * np.linalg.norm(b)
    e.close()

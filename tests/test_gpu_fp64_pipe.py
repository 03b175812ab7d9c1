"""The contractions on the FP64 pipe (precision fp64_pipe), which also serve FP64 contexts
that digit slices do not suit, against the oracle: ApplyCorrelationOp, FillH2, the energy,
a derivative, a split step, a batch.

Tolerance: the FP64 form's parity bound, 1e-12 relative, and 2e-14 for the contractions
with rho1 = 1 (no amplification by rho^-1).
"""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu

SYSTEMS = {"helium": (40, (1, 1), (5, 5), True), "one orbital": (3, (1, 1), (1, 1), True),
           "two types": (21, (2, 1), (4, 3), False), "one type": (70, (3,), (9,), False)}


def _spec(name):
    n_el, bodies, orbs, restricted = SYSTEMS[name]
    sp = S.helium_fedvr(n_el, 6, 1, laser=S.sin2_pulse(0.05), restricted=restricted)
    sp.xmin, sp.xmax = -0.5 * n_el, 0.5 * n_el
    sp.n_bodies, sp.n_orbs = bodies, orbs
    sp.masses, sp.stats = (1.0,) * len(bodies), "f" * len(bodies)
    return sp


def _state(sp, x, w, seed):
    rng = np.random.default_rng(seed)
    c = rng.normal(size=sp.n_coeffs) + 1j * rng.normal(size=sp.n_coeffs)
    return I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, x, w, seed))


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_entry_points_match_the_oracle(name):
    from codyfortran_gb300.engine import Engine
    sp = _spec(name)
    o, e = Oracle(sp), Engine(sp, "fp64_pipe")
    assert e.contraction_slices() == 0
    st = _state(sp, o.x, o.w, 3)
    orbs = st[o.nC:].reshape(-1, o.nG).T
    rng = np.random.default_rng(1)
    r2 = rng.normal(size=(o.nO,) * 4) + 1j * rng.normal(size=(o.nO,) * 4)
    d, h2 = e.apply_correlation_op(orbs, np.eye(o.nO, dtype=complex), r2, 0.0)
    dr, h2r = o.apply_correlation_op(orbs, np.eye(o.nO, dtype=complex), r2, 0.0)
    assert _rel(d, dr) < 2e-14 and _rel(h2, h2r) < 2e-14 and _rel(e.fill_h2(orbs, 0.0), h2r) < 2e-14
    assert abs(e.energy(st, 1.0) - o.energy(st, 1.0)) < 1e-12 * abs(o.energy(st, 1.0))
    for which in ("full", "nonlin"):
        assert _rel(e.time_derivative(st, 1.0, which), o.time_derivative(st, 1.0, which)) < 1e-12
    a = e.propagate_split2(st, 1.0, 1.01, 8, use_metric=True)
    assert _rel(a, o.propagate_split2(st, 1.0, 1.01, 8, metric=o.metric_weights())) < 1e-12
    e.close()


def test_the_choice_is_the_callers():
    from codyfortran_gb300.engine import Batch, Engine
    sp = _spec("helium")
    slices = {}
    for p in ("fp64", "fp64_pipe", "mixed", "mixed_fx", "mixed_fx6"):
        e = Engine(sp, p)
        slices[p] = e.contraction_slices()
        e.close()
    assert slices["fp64_pipe"] == slices["mixed"] == 0
    assert slices["fp64"] > slices["mixed_fx6"] >= slices["mixed_fx"] > 0
    specs = []
    for n in (20, 40, 30):
        q = _spec("helium")
        q.n_elements, q.xmin, q.xmax = n, -0.5 * n, 0.5 * n
        specs.append(q)
    out = []
    for p in ("fp64", "fp64_pipe"):
        b = Batch(specs, p, max_krylov=8)
        assert (b.contraction_slices() > 0) == (p == "fp64")
        states = [_state(q, s.x, s.w, k) for k, (q, s) in enumerate(zip(specs, b.systems))]
        b.upload(states)
        b.propagate(1.0, 0.01, 2, 8)
        out.append(b.download())
        b.close()
    for x, y in zip(*out):
        assert _rel(x, y) < 1e-11


@pytest.mark.parametrize("precision,shared", [("fp64", True), ("mixed_fx", True), ("fp64_pipe", False)])
def test_shared_interactions_are_reported(precision, shared):
    """FEDVR grids of one element size and count parity: pieces of the longest one."""
    from codyfortran_gb300.engine import Batch
    specs = []
    for n in (12, 20, 16):
        q = _spec("helium")
        q.n_elements, q.xmin, q.xmax = n, -1.0 * n, 1.0 * n
        specs.append(q)
    b = Batch(specs, precision, max_krylov=4)
    n = b.shared_interactions()
    b.close()
    assert n == (1 if shared else 0)

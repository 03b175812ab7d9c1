"""A batch in the FP64 form with the three-term Lanczos recurrence: every
trajectory as the oracle's, at Krylov orders too low to hide a wrong recurrence
coefficient behind convergence.  1e-12: the FP64 form's parity bound."""
import numpy as np
import pytest

from oracle import Oracle
from codyfortran_gb300 import init as I
from codyfortran_gb300 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,krylov", [(3, 1), (3, 2), (3, 5), (153, 2)])
def test_low_order_steps(n, krylov):
    from codyfortran_gb300.engine import Batch
    specs = []
    for k in range(n):
        sp = S.helium_fedvr(6 + 5 * (k % 3), 6, 2 + k % 2)
        sp.xmin, sp.xmax = -0.5 * sp.n_elements, 0.5 * sp.n_elements
        specs.append(sp)
    b = Batch(specs, "fp64", max_krylov=8, krylov_window=1)
    states = []
    for k, (sp, s) in enumerate(zip(specs, b.systems)):
        rng = np.random.default_rng(k)
        c = rng.normal(size=s.nC) + 1j * rng.normal(size=s.nC)
        states.append(I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, s.x, s.w, k)))
    b.upload(states)
    b.propagate(0.0, 0.02, 1, krylov)
    got = b.download()
    for k in range(0, n, max(1, n // 5)):
        o = Oracle(specs[k])
        ref = o.propagate_split2(states[k], 0.0, 0.02, krylov_dim=krylov, metric=o.metric_weights())
        assert np.linalg.norm(got[k] - ref) < 1e-12 * np.linalg.norm(ref), k
    b.close()

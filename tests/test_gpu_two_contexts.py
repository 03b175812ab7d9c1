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


def test_two_threads():
    """Two contexts driven by two threads at once, captured steps (whose one-launch SIL wants
    every SM) and adaptive ones: the results of the same calls one after the other, bit for bit."""
    import threading
    from codyfortran_gb300 import init as I
    from codyfortran_gb300.engine import Engine

    def state(e, sp, seed):
        rng = np.random.default_rng(seed)
        c = rng.normal(size=e.nC) + 1j * rng.normal(size=e.nC)
        return I.pack_state(c / np.linalg.norm(c), I.seeded_gaussian_orbitals(sp, e.x, e.w, seed))

    def work(e, st):
        e.upload(st)
        e.propagate_resident(0.0, 0.01, 20, 8, use_metric=True, use_graph=True)
        out = [e.download()]
        for k in range(5):
            out.append(e.propagate_split2(out[-1], 0.01 * k, 0.01 * (k + 1), 8, 1e-9, 3))
        return out

    jobs = []
    for n_el, m, precision in [(100, 4, "fp64"), (160, 6, "mixed_fx6")]:
        sp = S.helium_fedvr(n_el, 6, m, laser=S.sin2_pulse(0.05))
        sp.xmin, sp.xmax = -float(n_el), float(n_el)
        e = Engine(sp, precision, max_krylov=8)
        jobs.append((e, state(e, sp, m)))
    want = [work(*j) for j in jobs]
    got = [None, None]

    def run(i):
        for _ in range(3):
            got[i] = work(*jobs[i])
    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e, _ in jobs:
        e.close()
    for a, b in zip(got, want):
        assert a is not None and all(np.array_equal(x, y) for x, y in zip(a, b))

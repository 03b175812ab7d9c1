"""Performance cases: the calls that a user of the MCTDHF engine makes, over the sizes it is used at.

Every case is one 1D system (or a scan of them) and one public call sequence.

kind        what a user does
----------  -----------------------------------------------------------------
call        the Fortran host's propagator call: host state in, one Strang step
            with the adaptive Lanczos integrator, host state out
steps       real-time run on the resident state between two read-outs: upload,
            some fixed-order Strang steps, observables, download
relax       imaginary-time relaxation rounds from a correlated guess
derivative  Method_TimeDerivative of a host state (the non-linear part)
meanfield   ApplyCorrelationOp: mean-field term and two-body integrals
coeffs      Coeffs entry points: rho2 of a CI vector and H2 on it
lanczos     one adaptive short-iterative-Lanczos step of the one-body part
scan        a batch of independent trajectories (pulse-intensity and phase
            scan): upload, one Strang step of all, download
gradient    pulse gradient: forward sweep and the adjoint sweep back

Systems: `spins` = 2 is a restricted pair of spin body types with electrons / 2
bodies each in `orbitals` spatial orbitals; `spins` = 1 is one body type of
spin-polarised electrons; `grid` "uniform" is the 8th-order finite-difference
grid with unrestricted spin orbitals, otherwise FEDVR with `elements` elements
of `locals` Gauss-Lobatto points on [-box, box].
"""
import functools
import itertools
import math

import numpy as np
import torch

OMEGA, CYCLES = 0.057, 4.0
PULSE = 2.0 * math.pi * CYCLES / OMEGA


# --------------------------------------------------------------------------- cases
def _system(**kw):
    c = dict(spins=2, electrons=2, orbitals=4, elements=100, locals=6, box=100.0, grid="fedvr", precision="fp64",
             krylov=12)
    c.update(kw)
    return c


def listed():
    return [
        # the reference's He1d chain: 21 points, 4 + 4 spin orbitals, SIL 24 at 1e-12 (the smallest call)
        _system(name="call_he1d", kind="call", grid="uniform", elements=20, locals=2, box=20.0, krylov=24, dt=1e-3,
                tol=1e-12, restarts=8),
        # 1D helium, 501 points, FP64: a short real-time run between two read-outs
        _system(name="steps_helium", kind="steps", dt=0.01, steps=10),
        # the same system's imaginary-time relaxation
        _system(name="relax_helium", kind="relax", dt=0.005, inner=10, rounds=2),
        # an odd mid-size system of the scan, as a program with its own integrator calls it
        _system(name="derivative_fx6", kind="derivative", electrons=4, orbitals=9, elements=217, box=217.0,
                precision="mixed_fx6"),
        # the mean-field operator alone, FP64, odd grid
        _system(name="meanfield", kind="meanfield", orbitals=10, elements=161, box=161.0),
        # 8008 determinants: the CI entry points alone
        _system(name="coeffs_8008", kind="coeffs", spins=1, electrons=6, orbitals=16, elements=10, locals=8, box=20.0),
        # one-body propagation on the largest grid
        _system(name="lanczos_2801", kind="lanczos", spins=1, electrons=6, orbitals=16, elements=400, locals=8,
                box=400.0, krylov=16, dt=0.01, tol=1e-10, restarts=4),
        # three wells, 2801 points, 16 spin orbitals, 8008 determinants: plain and split-precision form
        _system(name="steps_trimer", kind="steps", spins=1, electrons=6, orbitals=16, elements=400, locals=8,
                box=400.0, krylov=16, dt=0.02, steps=1),
        _system(name="steps_trimer_fx6", kind="steps", spins=1, electrons=6, orbitals=16, elements=400, locals=8,
                box=400.0, krylov=16, dt=0.02, steps=2, precision="mixed_fx6"),
        # intensity / phase scans with uneven sizes: a small one in FP64, the full one in the split-precision form
        dict(name="scan_24", kind="scan", trajectories=24, scan=77, precision="fp64", krylov=12, dt=0.02),
        dict(name="scan_512_fx6", kind="scan", trajectories=512, scan=1234, precision="mixed_fx6", krylov=12, dt=0.02),
        # pulse optimisation: 1D helium, 8 orbitals, gradient with respect to every field sample
        _system(name="gradient_helium", kind="gradient", orbitals=8, dt=0.05, samples=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "steps", "steps", "relax", "derivative", "derivative", "meanfield", "coeffs", "lanczos",
                       "scan", "scan", "gradient"])
    if kind == "scan":
        prec = rng.choice(["fp64", "mixed_fx", "mixed_fx6", "mixed_fx6"])
        return dict(kind=kind, trajectories=_log(rng, 2, 32 if prec == "fp64" else 384), scan=rng.randrange(1, 10**6),
                    precision=prec, krylov=rng.choice([8, 12, 12, 16]), dt=0.02)
    ne = _log(rng, 20, 400)
    c = _system(kind=kind, elements=ne, box=float(ne), locals=rng.choice([5, 6, 6, 8]),
                krylov=rng.choice([8, 12, 12, 16]))
    prec = rng.choice(["fp64", "fp64", "mixed_fx", "mixed_fx6", "mixed_fx6"])
    if kind == "gradient":
        c.update(orbitals=rng.randrange(2, 10), elements=_log(rng, 20, 100), locals=6, dt=0.05,
                 samples=rng.randrange(1, 13), krylov=12)
        c["box"] = float(c["elements"])
        return c
    if kind == "call":
        c.update(dt=0.01, tol=1e-11, restarts=4, krylov=24, orbitals=rng.randrange(2, 9), elements=_log(rng, 4, 200))
        c["box"] = float(c["elements"])
        return c
    if kind == "lanczos":
        c.update(dt=0.01, tol=1e-10, restarts=4, orbitals=rng.randrange(2, 17), krylov=16)
        return c
    if rng.random() < 0.3:
        n = rng.randrange(2, 7)
        c.update(spins=1, electrons=n, orbitals=rng.randrange(max(4, n + 1), 17))
    else:
        n = rng.choice([2, 2, 4, 4, 6])
        c.update(electrons=n, orbitals=rng.randrange(max(3, n // 2 + 1), 13 if n < 6 else 9))
    if kind in ("steps", "derivative"):
        c["precision"] = prec
    if kind == "steps":
        c.update(dt=0.02, steps=rng.randrange(1, 4))
    if kind == "relax":
        c.update(dt=0.002, inner=rng.randrange(2, 7), rounds=rng.randrange(1, 3))
    if kind == "coeffs":
        c.update(elements=10, box=10.0)
    return c


def _members(case):
    """The systems of a case: one, or the trajectories of a scan (electrons, orbitals, box length and pulse differ)."""
    if case["kind"] != "scan":
        return [dict(case, E0=0.0755 if case["spins"] == 1 else 0.0534, cep=0.0)]
    rng, out = np.random.default_rng(case["scan"]), []
    for _ in range(case["trajectories"]):
        ne = int(rng.integers(100, 401))
        out.append(_system(electrons=int(rng.choice([2, 4])), orbitals=int(rng.integers(4, 13)), elements=ne,
                           box=float(ne), E0=math.sqrt(10.0 ** rng.uniform(13.0, 15.0) / 3.509e16),
                           cep=float(rng.uniform(0.0, 2.0 * math.pi))))
    return out


def _bodies(m):
    """(bodies, orbitals) per body type, and whether the types share their orbitals."""
    if m["grid"] == "uniform":
        return (1, 1), (m["orbitals"], m["orbitals"]), False
    if m["spins"] == 1:
        return (m["electrons"],), (m["orbitals"],), False
    return (m["electrons"] // 2,) * 2, (m["orbitals"],) * 2, True


def _wells(m):  # position, charge, softening inside and outside the root
    if m["grid"] == "uniform":
        return [(0.0, 2.0, 0.0, 1.0)]
    return [(-4.0, 2.0, 1.0, 0.0), (0.0, 2.0, 1.0, 0.0), (4.0, 2.0, 1.0, 0.0)] if m["spins"] == 1 else [(0.0, 2.0, 1.0, 0.0)]


def _pulsed(m):
    return m["grid"] != "uniform" and m.get("kind") not in ("relax", "coeffs", "meanfield")


# --------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=64)
def _lobatto(n):
    """Gauss-Lobatto points and weights on [-1, 1]."""
    p = np.polynomial.legendre.Legendre.basis(n - 1)
    d1, d2 = p.deriv(), p.deriv(2)
    x = np.sort(d1.roots().real) if n > 2 else np.zeros(0)
    for _ in range(3):
        x = x - d1(x) / d2(x)
    x = np.concatenate([[-1.0], x, [1.0]])
    return x, 2.0 / (n * (n - 1) * p(x) ** 2)


@functools.lru_cache(maxsize=1024)
def _grid(kind, elements, locals_, box):
    if kind == "uniform":
        n = elements + 1
        return np.linspace(-box, box, n), np.full(n, 2.0 * box / (n - 1))
    t, wt = _lobatto(locals_)
    es = 2.0 * box / elements
    n = elements * (locals_ - 1) + 1
    x, w = np.zeros(n), np.zeros(n)
    for e in range(elements):
        s = slice(e * (locals_ - 1), e * (locals_ - 1) + locals_)
        x[s] = -box + (e + 0.5) * es + 0.5 * es * t
        w[s] += 0.5 * es * wt
    return x, w


def _points(m):
    return _grid(m["grid"], m["elements"], m["locals"], m["box"])


def _n_coeffs(m):
    b, o, _ = _bodies(m)
    return math.prod(math.comb(k, n) for n, k in zip(b, o))


def _groups(m):
    """Column ranges of the stored orbitals that are orthonormal among themselves."""
    _, o, shared = _bodies(m)
    return [(0, o[0])] if shared or len(o) == 1 else [(0, o[0]), (o[0], o[0] + o[1])]


def _state(m, rng):
    """A correlated wave packet: random normalised CI vector, Gaussian-envelope orbitals made orthonormal."""
    x, w = _points(m)
    n = _groups(m)[-1][1]
    x0, sigma = rng.uniform(-2.5, 2.5, n), rng.uniform(0.5, 2.5, n)
    f = np.exp(-((x[:, None] - x0) ** 2) / (2.0 * sigma**2)) * (rng.normal(size=n) + 1j * rng.normal(size=n))
    f = f * np.exp(1j * rng.uniform(-1.0, 1.0, n) * x[:, None])
    r = np.sqrt(w)[:, None]
    for a, b in _groups(m):
        q = np.linalg.qr(f[:, a:b] * r)[0]
        f[:, a:b] = np.linalg.qr(q)[0] / r
    c = rng.normal(size=_n_coeffs(m)) + 1j * rng.normal(size=_n_coeffs(m))
    return np.concatenate([c / np.linalg.norm(c), f.T.ravel()])


def _inputs(case, seed):
    """Everything that the seed decides."""
    rng = np.random.default_rng(seed)
    ms = _members(case)
    d = {"states": [_state(m, rng) for m in ms], "t0": PULSE * rng.uniform(0.3, 0.6)}
    if case["kind"] == "gradient":
        d["field"] = rng.normal(0.0, 0.01, size=case["samples"])
    if case["kind"] == "coeffs":
        n = sum(_bodies(ms[0])[1])
        h = rng.normal(size=(n,) * 4) + 1j * rng.normal(size=(n,) * 4)
        d["h2"] = np.asfortranarray(0.05 * (h + h.conj().transpose(2, 3, 0, 1)))
    if case["kind"] == "meanfield":
        s = _Exact(ms[0])
        C, F = s.split(torch.from_numpy(d["states"][0]))
        one, two = s.rdms(C)
        d["rdm1"] = np.asfortranarray(one.numpy())
        d["rdm2"] = np.asfortranarray(two.numpy())
        d["orbs"] = np.asfortranarray(F.numpy())
    return d


def _spec(m, field=None):
    from codyfortran_gb300 import spec as S
    b, o, shared = _bodies(m)
    laser = S.Laser()
    if field is not None:
        laser = S.Laser(kind="sampled", samples=field, sample_dt=m["dt"], sample_t0=0.0)
    elif _pulsed(m):
        laser = S.sin2_pulse(m["E0"], OMEGA, CYCLES, m["cep"])
    uniform = m["grid"] == "uniform"
    return S.SystemSpec(
        grid_kind="const" if uniform else "fedvr", xmin=-m["box"], xmax=m["box"], n_points=m["elements"] + 1,
        n_elements=m["elements"], n_locals=m["locals"], n_bodies=b, n_orbs=o, masses=(1.0,) * len(b),
        stats="f" * len(b), restricted=shared, nuclei=[S.Nucleus(p, q, s1, s2, 0.0) for p, q, s1, s2 in _wells(m)],
        int_s1=0.0 if uniform else 1.0, int_s2=1.0 if uniform else 0.0, int_kind="toeplitz" if uniform else "dense",
        laser=laser)


def prepare(case, seed):
    from codyfortran_gb300 import engine as E
    d = dict(_inputs(case, seed), case=case)
    fp64 = case.get("precision", "fp64") == "fp64"
    more = dict(max_krylov=case["krylov"], krylov_window=0 if fp64 else 1)
    ms = _members(case)
    if case["kind"] == "scan":
        d["h"] = E.Batch([_spec(m) for m in ms], case["precision"], **more)
        flat = np.concatenate(d.pop("states"))
        d["state"], d["out"] = E.pinned_empty(flat.size), E.pinned_empty(flat.size)
        d["state"][:] = flat
        return d
    d["h"] = E.Engine(_spec(ms[0], d.get("field")), case["precision"], **more)
    d["state"] = d.pop("states")[0]
    d["metric"] = d["h"].metric_weights()
    return d


def run(s):
    c, e, kind = s["case"], s["h"], s["case"]["kind"]
    if kind == "call":
        return e.propagate_split2(s["state"], s["t0"], s["t0"] + c["dt"], c["krylov"], c["tol"], c["restarts"])
    if kind == "steps":
        e.upload(s["state"])
        e.propagate_resident(s["t0"], c["dt"], c["steps"], c["krylov"], use_metric=True, use_graph=True)
        o = e.observables(s["t0"] + c["steps"] * c["dt"])
        return {"state": e.download(), "values": np.array([o["energy"], o["norm"], o["dipole"]]),
                "occupations": o["occupations"]}
    if kind == "relax":
        energy, state, rounds = e.relax(s["state"], c["dt"], c["inner"], 0.0, c["rounds"])
        return {"energy": energy, "state": state, "rounds": rounds}
    if kind == "derivative":
        return e.time_derivative(s["state"], s["t0"], "nonlin")
    if kind == "meanfield":
        return e.apply_correlation_op(s["orbs"], s["rdm1"], s["rdm2"], 0.0)
    if kind == "coeffs":
        C = s["state"][: e.nC]
        return {"rdm2": e.rdm2(C), "product": e.apply_h2(C, s["h2"])}
    if kind == "lanczos":
        return e.sil(s["state"], s["t0"], s["t0"] + c["dt"], c["krylov"], c["tol"], c["restarts"], s["metric"])
    if kind == "scan":
        e.upload(s["state"])
        e.propagate(s["t0"], c["dt"], 1, c["krylov"])
        return e.download_packed(s["out"])
    objective, overlap, final = e.mc_adjoint_forward(s["state"], s["field"], c["dt"], c["krylov"])
    return {"objective": objective, "overlap": np.array([overlap]), "final": final, "gradient": e.mc_adjoint_backward()}


# --------------------------------------------------------------------------- work
def _nonlin_flops(m):
    """One non-linear derivative: pair potentials, mean field and h2, CI products and density matrices."""
    b, o, shared = _bodies(m)
    n, nG, nC = _groups(m)[-1][1], len(_points(m)[0]), _n_coeffs(m)
    pairs = sum((h - l) * (h - l + 1) // 2 for l, h in _groups(m))
    singles = [k * (q - k + 1) for k, q in zip(b, o)]
    doubles = sum(math.comb(k, 2) * math.comb(q - k + 2, 2) for k, q in zip(b, o))
    cross = singles[0] * singles[1] if len(b) == 2 else 0
    terms = nC * (sum(singles) + doubles + cross)
    return 4.0 * nG * nG * pairs + 2 * 8.0 * nG * n**4 + 2 * 8.0 * terms, 8.0 * terms


def _step_flops(m, krylov):
    n, nG = _groups(m)[-1][1], len(_points(m)[0])
    lanczos = krylov * nG * n * (4.0 * (2 * m["locals"] - 1) + 40.0)
    return 4 * _nonlin_flops(m)[0] + 2 * lanczos


def work(case):
    flops, nbytes, kind = 0.0, 0.0, case["kind"]
    for m in _members(case):
        n, nG, nC = _groups(m)[-1][1], len(_points(m)[0]), _n_coeffs(m)
        nO = sum(_bodies(m)[1])
        state = 16.0 * (nC + nG * n)
        k = case["krylov"]
        if kind in ("steps", "scan", "call"):
            flops += case.get("steps", 1) * _step_flops(m, 6 if kind == "call" else k)
            nbytes += 2 * state
        elif kind == "relax":
            flops += case["inner"] * case["rounds"] * _nonlin_flops(m)[0]
            nbytes += 2 * state
        elif kind == "derivative":
            flops += _nonlin_flops(m)[0]
            nbytes += 2 * state
        elif kind == "meanfield":
            flops += _nonlin_flops(m)[0] - 2 * _nonlin_flops(m)[1]
            nbytes += 2 * 16.0 * nG * n + 16.0 * (nO**2 + 2 * nO**4)
        elif kind == "coeffs":
            flops += 2 * _nonlin_flops(m)[1]
            nbytes += 2 * 16.0 * nC + 2 * 16.0 * nO**4
        elif kind == "lanczos":
            flops += 8 * nG * n * (4.0 * (2 * m["locals"] - 1) + 40.0)
            nbytes += 2 * state
        else:  # forward, recomputation and about two products for each of the forward's in the adjoint
            flops += 4.0 * case["samples"] * _step_flops(m, k)
            nbytes += 2 * state + 16.0 * case["samples"]
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------------------------- the same in 64 bits
class _RegularisedInverse(torch.autograd.Function):
    """Hermitian r -> r (r^2 + eps)^-1 through its eigenvectors."""

    @staticmethod
    def forward(ctx, r, eps):
        n, U = torch.linalg.eigh(r)
        ctx.save_for_backward(n, U)
        ctx.eps = eps
        return (U * (n / (n * n + eps))) @ U.mH

    @staticmethod
    def backward(ctx, g):
        n, U = ctx.saved_tensors
        a, b = n[:, None], n[None, :]
        # (f(a) - f(b)) / (a - b) of f(n) = n / (n^2 + eps), without the difference
        D = (ctx.eps - a * b) / ((a * a + ctx.eps) * (b * b + ctx.eps))
        return U @ (D * (U.mH @ g @ U)) @ U.mH, None


@functools.lru_cache(maxsize=64)
def _strings(M, N):
    s = list(itertools.combinations(range(M), N))
    return s, {t: i for i, t in enumerate(s)}


@functools.lru_cache(maxsize=64)
def _removed(M, N, k):
    """a_jk .. a_j1 on the N-body strings: for each k-subset and (N - k)-string the source string and sign (0: none)."""
    if N < k:
        return None
    full, small = _strings(M, N)[1], _strings(M, N - k)[0]
    subs = list(itertools.combinations(range(M), k))
    idx, sgn = np.zeros((len(subs), len(small)), np.int64), np.zeros((len(subs), len(small)))
    for p, js in enumerate(subs):
        for q, rest in enumerate(small):
            if set(js) & set(rest):
                continue
            src, f = tuple(sorted(rest + js)), 0
            left = list(src)
            for j in js:
                f += left.index(j)
                left.remove(j)
            idx[p, q], sgn[p, q] = full[src], -1.0 if f % 2 else 1.0
    return idx, sgn


@functools.lru_cache(maxsize=64)
def _sectors(bodies, orbs):
    """(one, two): index and sign arrays of the annihilated CI vectors, with the spin orbitals that each row removes."""
    nO, sizes = sum(orbs), [math.comb(q, k) for k, q in zip(bodies, orbs)]
    cols = [np.arange(s) for s in sizes]
    start = [0, orbs[0]]

    def spread(per_type):  # per body type: (rows or None, index, sign) -> rows x everything else
        idx, sgn = None, None
        stride = 1
        for b, (i, s) in enumerate(per_type):
            i = i * stride
            stride *= sizes[b]
            if idx is None:
                idx, sgn = i[:, None, :], s[:, None, :]
            else:  # rows of both types, columns of both types
                idx = (idx[:, None, :, :] + i[None, :, None, :].transpose(0, 1, 3, 2)).reshape(
                    idx.shape[0] * i.shape[0], i.shape[1], -1)
                sgn = (sgn[:, None, :, :] * s[None, :, None, :].transpose(0, 1, 3, 2)).reshape(idx.shape)
        return torch.from_numpy(idx.reshape(idx.shape[0], -1)), torch.from_numpy(sgn.reshape(idx.shape[0], -1)) + 0j

    def whole(b):
        return cols[b][None, :], np.ones((1, sizes[b]))

    one, two = [], []
    for b in range(len(bodies)):
        if (r := _removed(orbs[b], bodies[b], 1)) is not None:
            i, s = spread([r if q == b else whole(q) for q in range(len(bodies))])
            one.append((list(range(start[b], start[b] + orbs[b])), i, s))
        if (r := _removed(orbs[b], bodies[b], 2)) is not None and orbs[b] > 1:
            i, s = spread([r if q == b else whole(q) for q in range(len(bodies))])
            pairs = [(start[b] + p, start[b] + q) for p, q in itertools.combinations(range(orbs[b]), 2)]
            two.append((_antisymmetric(pairs, nO), i, s))
    if len(bodies) == 2 and min(bodies) > 0:
        i, s = spread([_removed(orbs[0], bodies[0], 1), _removed(orbs[1], bodies[1], 1)])
        two.append((_antisymmetric([(p, orbs[0] + q) for p in range(orbs[0]) for q in range(orbs[1])], nO), i, s))
    return one, two


def _antisymmetric(pairs, nO):
    T = np.zeros((nO * nO, len(pairs)))
    for k, (p, q) in enumerate(pairs):
        T[p * nO + q, k], T[q * nO + p, k] = 1.0, -1.0
    return torch.from_numpy(T) + 0j


class _Exact:
    """The equations of one system in plain 64-bit torch."""

    def __init__(self, m, field=None):
        self.m, self.field = m, field
        self.bodies, self.orbs, self.shared = _bodies(m)
        self.nC, self.n, self.nO = _n_coeffs(m), _groups(m)[-1][1], sum(self.orbs)
        x, w = _points(m)
        self.x, self.w, self.nG = torch.from_numpy(x), torch.from_numpy(w), len(x)
        self.one, self.two = _sectors(self.bodies, self.orbs)
        V = np.zeros_like(x)
        for p, q, s1, s2 in _wells(m):
            V -= q / (np.sqrt((x - p) ** 2 + s1 * s1) + s2)
        self.V = torch.from_numpy(V)
        d = np.abs(x[:, None] - x[None, :])
        self.K = torch.from_numpy(1.0 / (d + 1.0) if m["grid"] == "uniform" else 1.0 / np.sqrt(d * d + 1.0))
        if m["grid"] != "uniform":
            L = m["locals"]
            t, wt = _lobatto(L)
            D = np.array([[sum(1.0 / (t[i] - t[k]) for k in range(L) if k != i) if i == j else
                           math.prod((t[i] - t[k]) / (t[j] - t[k]) for k in range(L) if k not in (i, j)) / (t[j] - t[i])
                           for j in range(L)] for i in range(L)])
            half = m["box"] / m["elements"]
            self.Kin = torch.from_numpy(0.5 * (D.T * wt) @ D / half) + 0j
            self.idx = torch.from_numpy(np.arange(m["elements"])[:, None] * (L - 1) + np.arange(L)[None, :])

    def split(self, s):
        return s[: self.nC], s[self.nC:].reshape(self.n, self.nG).T

    def join(self, C, F):
        return torch.cat([C, F.T.reshape(-1)])

    def E(self, t):
        if self.field is not None:
            k = int(math.floor(t / self.m["dt"] + 1e-9))
            return self.field[k] if 0 <= k < len(self.field) else 0.0
        if not _pulsed(self.m) or not 0.0 <= t <= PULSE:
            return 0.0
        return self.m["E0"] * math.sin(math.pi * t / PULSE) ** 2 * math.cos(OMEGA * (t - 0.5 * PULSE) + self.m["cep"])

    def h(self, F, t):
        if self.m["grid"] == "uniform":
            dx = float(self.w[0])
            c = [-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0]
            P = torch.cat([torch.zeros(4, self.n) + 0j, F, torch.zeros(4, self.n) + 0j])
            out = sum(c[abs(k)] * P[4 + k: 4 + k + self.nG] for k in range(-4, 5)) * (-0.5 / (dx * dx))
        else:
            local = torch.einsum("ab,ebn->ean", self.Kin, F[self.idx])
            out = torch.zeros(self.nG, self.n, dtype=F.dtype).index_add(0, self.idx.reshape(-1),
                                                                        local.reshape(-1, self.n)) / self.w[:, None]
        return out + (self.V + self.E(t) * self.x)[:, None] * F

    def inner(self, A, B):
        return (A.conj() * self.w[:, None]).T @ B

    def same_type(self, A):
        """Zero between orbitals of different body types."""
        if len(_groups(self.m)) == 1:
            return A
        keep = torch.zeros(self.n, self.n)
        for a, b in _groups(self.m):
            keep[a:b, a:b] = 1.0
        return A * keep

    def spin(self, h):
        return torch.block_diag(h, h) if self.shared else h

    def rdms(self, C):
        one = torch.zeros(self.nO, self.nO, dtype=C.dtype)
        for rows, i, s in self.one:
            A = C[i] * s
            one = one + torch.nn.functional.pad(A.conj() @ A.T, (rows[0], self.nO - rows[-1] - 1) * 2)
        two = torch.zeros(self.nO**2, self.nO**2, dtype=C.dtype)
        for T, i, s in self.two:
            A = C[i] * s
            two = two + T @ (A.conj() @ A.T) @ T.T
        return one, two.reshape((self.nO,) * 4)

    def h1_on(self, C, h1):
        out = torch.zeros_like(C)
        for rows, i, s in self.one:
            sub = h1[rows[0]:rows[-1] + 1, rows[0]:rows[-1] + 1]
            out = out.index_add(0, i.reshape(-1), (s * (sub.T @ (C[i] * s))).reshape(-1))
        return out

    def h2_on(self, C, H):
        out, H = torch.zeros_like(C), H.reshape(self.nO**2, self.nO**2)
        for T, i, s in self.two:
            out = out.index_add(0, i.reshape(-1), (s * ((T.T @ H @ T).T @ (C[i] * s))).reshape(-1))
        return out

    def potentials(self, F):
        S = (F.conj() * self.w[:, None])[:, :, None] * F[:, None, :]  # (x, l, k)
        S = S.reshape(self.nG, -1)
        W = torch.complex(self.K @ S.real, self.K @ S.imag).reshape(self.nG, self.n, self.n)
        return self.same_type(W)

    def h2(self, F, W):
        S = self.same_type((F.conj() * self.w[:, None])[:, :, None] * F[:, None, :]).reshape(self.nG, -1)
        g = 0.5 * (S.T @ W.reshape(self.nG, -1)).reshape((self.n,) * 4).permute(0, 2, 1, 3)  # (i1, i2, j1, j2)
        if not self.shared:
            return g
        one = torch.eye(2) + 0j
        return torch.einsum("ac,bd,ijkl->aibjckdl", one, one, g).reshape((self.nO,) * 4)

    def mean_field(self, F, W, one, two):
        n = self.n
        if self.shared:
            r1 = one[:n, :n] + one[n:, n:]
            r2 = torch.einsum("aibjakbl->ijkl", two.reshape(2, n, 2, n, 2, n, 2, n))
        else:
            r1, r2 = one, two
        R = torch.einsum("abkd,kj->abjd", r2, _RegularisedInverse.apply(r1, 1e-10))
        Z = W.reshape(self.nG, -1) @ R.permute(3, 1, 0, 2).reshape(n * n, n * n)  # (l2 k2) -> (k1 j1)
        Z = self.same_type(Z.reshape(self.nG, n, n))
        return torch.einsum("xk,xkj->xj", F, Z)

    def project(self, dF, F):
        parts = [dF[:, a:b] - F[:, a:b] @ self.inner(F[:, a:b], dF[:, a:b]) for a, b in _groups(self.m)]
        return torch.cat(parts, 1)

    def derivative(self, s, t, full=False):
        C, F = self.split(s)
        one, two = self.rdms(C)
        hF, W = self.h(F, t), self.potentials(F)
        dF = self.mean_field(F, W, one, two) + (hF if full else 0.0)
        dC = self.h1_on(C, self.spin(self.same_type(self.inner(F, hF)))) + self.h2_on(C, self.h2(F, W))
        dC = dC - C * torch.sum(C.conj() * dC)
        return -1j * self.join(dC, self.project(dF, F))

    def rk4(self, s, t, dt):
        k1 = self.derivative(s, t)
        k2 = self.derivative(s + 0.5 * dt * k1, t + 0.5 * dt)
        k3 = self.derivative(s + 0.5 * dt * k2, t + 0.5 * dt)
        k4 = self.derivative(s + dt * k3, t + dt)
        return s + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)

    def lanczos(self, s, t, dt, krylov, tol, metric):
        m = torch.cat([torch.ones(self.nC), self.w.repeat(self.n) if metric else torch.ones(self.nG * self.n)]).double()
        dot = lambda a, b: torch.sum(a.conj() * m * b)  # noqa: E731
        norm = torch.sqrt(dot(s, s).real)
        V, alpha, beta = [s / norm], [], []
        for j in range(krylov):
            u = self.join(torch.zeros(self.nC) + 0j, self.h(self.split(V[j])[1], t + 0.5 * dt))
            if j:
                u = u - beta[-1] * V[j - 1]
            alpha.append(dot(V[j], u).real)
            u = u - alpha[-1] * V[j]
            for v in V:
                u = u - dot(v, u) * v
            beta.append(torch.sqrt(dot(u, u).real))
            T = torch.diag(torch.stack(alpha))
            if j:
                off = torch.stack(beta[:-1])
                T = T + torch.diag(off, 1) + torch.diag(off, -1)
            if tol > 0.0 or j == krylov - 1:
                phi = torch.linalg.matrix_exp(-1j * dt * T)[:, 0]
                err = float(beta[-1].detach()) * abs(complex(phi[-1].detach()))
                if err <= tol or float(beta[-1].detach()) <= 1e-14:
                    err = 0.0
                    break
            V.append(u / beta[-1])
        return norm * sum(p * v for p, v in zip(phi, V)), err <= tol

    def sil(self, s, t, dt, krylov, tol=0.0, restarts=0, metric=True):
        left = dt
        while abs(left) > 1e-14:
            part = left
            for k in range(restarts + 1):
                new, ok = self.lanczos(s, t, part, krylov, tol, metric)
                if ok or k == restarts:
                    break
                part *= 0.5
            s, t, left = new, t + part, left - part
        return s

    def strang(self, s, t, dt, krylov, **more):
        s = self.sil(s, t, 0.5 * dt, krylov, **more)
        s = self.rk4(s, t, dt)
        return self.sil(s, t + 0.5 * dt, 0.5 * dt, krylov, **more)

    def values(self, s, t):
        """Energy, norm, dipole; natural occupations."""
        C, F = self.split(s)
        one, two = self.rdms(C)
        h1 = self.spin(self.same_type(self.inner(F, self.h(F, t))))
        xm = self.spin(self.same_type(self.inner(F, self.x[:, None] * F)))
        H = self.h2(F, self.potentials(F)).reshape(self.nO**2, self.nO**2)
        energy = torch.trace(h1 @ one) + torch.trace(H @ two.reshape(self.nO**2, self.nO**2))
        r1 = one[: self.n, : self.n] + one[self.n:, self.n:] if self.shared else one
        occ = torch.linalg.eigvalsh(r1).flip(0)
        return torch.stack([energy.real, torch.linalg.norm(C), torch.trace(xm @ one).real]), occ

    def orthonormal(self, F):
        cols = []
        for a, b in _groups(self.m):
            group = []
            for k in range(a, b):
                f = F[:, k]
                for _ in range(2):
                    for g in group:
                        f = f - g * torch.sum(g.conj() * f * self.w)
                group.append(f / torch.sqrt(torch.sum(f.abs() ** 2 * self.w)))
            cols += group
        return torch.stack(cols, 1)


def exact(case, seed):
    if case["kind"] == "scan" and case["trajectories"] > 40:
        return None  # hundreds of systems: minutes on the host
    d, ms = _inputs(case, seed), _members(case)
    t, dt, k = d["t0"], case.get("dt"), case["krylov"]
    if case["kind"] == "scan":
        return torch.cat([_Exact(m).strang(torch.from_numpy(s), t, dt, k) for m, s in zip(ms, d["states"])]).numpy()
    field = torch.tensor(d["field"], requires_grad=True) if "field" in d else None
    x, s = _Exact(ms[0], field), torch.from_numpy(d["states"][0])
    if case["kind"] == "call":
        return x.strang(s, t, dt, k, tol=case["tol"], restarts=case["restarts"], metric=False).numpy()
    if case["kind"] == "steps":
        for j in range(case["steps"]):
            s = x.strang(s, t + j * dt, dt, k)
        values, occ = x.values(s, t + case["steps"] * dt)
        return {"state": s.numpy(), "values": values.numpy(), "occupations": occ.numpy()}
    if case["kind"] == "relax":
        for _ in range(case["inner"] * case["rounds"]):
            C, F = x.split(s - 1j * dt * x.derivative(s, 0.0, full=True))
            s = x.join(C / torch.linalg.norm(C), x.orthonormal(F))
        return {"energy": float(x.values(s, 0.0)[0][0]), "state": s.numpy(), "rounds": None}
    if case["kind"] == "derivative":
        return x.derivative(s, t).numpy()
    if case["kind"] == "meanfield":
        F = torch.from_numpy(d["orbs"])
        W = x.potentials(F)
        dF = x.mean_field(F, W, torch.from_numpy(d["rdm1"]), torch.from_numpy(d["rdm2"]))
        return np.asfortranarray(dF.numpy()), np.asfortranarray(x.h2(F, W).numpy())
    if case["kind"] == "coeffs":
        C = s[: x.nC]
        return {"rdm2": x.rdms(C)[1].numpy(), "product": x.h2_on(C, torch.from_numpy(d["h2"])).numpy()}
    if case["kind"] == "lanczos":
        return x.sil(s, t, dt, k, case["tol"], case["restarts"]).numpy()
    C0, F0 = x.split(s)
    for j in range(case["samples"]):
        s = x.strang(s, j * dt, dt, k)
    C, F = x.split(s)
    n = x.n
    S = x.inner(F0, F)
    overlap = torch.sum(C0.reshape(n, n).conj() * (S @ C.reshape(n, n) @ S.T))
    objective = 1.0 - overlap.abs() ** 2
    gradient, = torch.autograd.grad(objective, field)
    return {"objective": float(objective.detach()), "overlap": np.array([complex(overlap.detach())]),
            "final": s.detach().numpy(), "gradient": gradient.numpy()}

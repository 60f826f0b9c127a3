"""The work that programs have this package do, as timed cases.

Every case goes through the public Python entry points: the Hamiltonian
action (``matvec``, ``apply``), the plain FP64 propagator, the batched
mixed-precision propagator (equal and unequal recombination rates), the
adjoint gradients and the factorized ensemble yields.  Sizes are those of the
repository's workloads: the 96-dimension smoke system, nuclear subsets of the
221,184-dimension FAD-TrpH pair (864 and 13,824 dimensions) and the full pair,
on the benchmark's 0.00125-us observation grid with lifetime 1 us.  Horizons
are cut from the workloads' 5 us where a pass would otherwise take seconds;
the cost per simulated microsecond is stationary.

A case names its nuclei per radical: ``l1`` spin-1 and ``lh`` spin-1/2 nuclei
on the left (FAD) radical, ``r1`` and ``rh`` on the right (TrpH) one.
"""

from __future__ import annotations

import math

import numpy as np
import torch

GRID_US = 0.00125     # observation grid of the benchmark workloads
HORIZON_US = 5.0      # their full horizon: budgets are scaled by a case's share of it
LIFETIME_US = 1.0
BATCH_BUDGET = 5e-7   # state-error budget of the batched workload over 5 us
PLAIN_BUDGET = 1e-10  # Lanczos tolerance of the plain full-size workload


def listed():
    small = dict(l1=1, lh=1, r1=0, rh=2)     # 96 dimensions: the smoke system
    six = dict(l1=2, lh=1, r1=1, rh=2)       # 864: three nuclei per radical
    ten = dict(l1=2, lh=3, r1=1, rh=4)       # 13,824: five nuclei per radical
    full = dict(l1=2, lh=5, r1=1, rh=6)      # 221,184: the production pair
    return [
        # One H psi of a small subset: the call SciPy solvers and tests repeat; launch latency.
        dict(name="matvec_864", kind="matvec", **six),
        # One FP64 H psi of the full state: the reference's own hot call.
        dict(name="matvec_221184", kind="matvec", **full),
        # Complex64 H psi of a benchmark-sized batch (12 orientations x 4 vectors of one system).
        dict(name="apply_c64_221184_x48", kind="apply", count=48, precision=64, **full),
        # The plain FP64 method on the smoke system (Krylov <= 30): one vector to 1 us.
        dict(name="plain_96", kind="plain", horizon=1.0, kmin=8, kmax=30, **small),
        # The plain FP64 production call (adaptive Krylov 8-40, tolerance 1e-10), a 0.05-us stretch.
        dict(name="plain_221184", kind="plain", horizon=0.05, kmin=8, kmax=40, **full),
        # The smoke system's 64 random-phase vectors as one batch, the whole 5 us.
        dict(name="batched_96_x64", kind="batched", orientations=1, vectors=64, krylov=30, horizon=5.0,
             final=False, **small),
        # An orientation sweep of a ten-nucleus subset; final states wanted (segments, checkpoints).
        dict(name="batched_13824_x30", kind="batched", orientations=10, vectors=3, krylov=32, horizon=1.0,
             final=True, **ten),
        # The benchmark's batch: 12 Fibonacci orientations x 4 vectors, Krylov cap 40.
        dict(name="batched_221184_x48", kind="batched", orientations=12, vectors=4, krylov=40, horizon=0.5,
             final=False, **full),
        # Uneven sizes in one call with kS = 1e6, kT = 2e6 1/s (Arnoldi), the directional sweep at 1/32 scale.
        dict(name="uneven_rates_x32", kind="uneven", n864=16, n13824=10, n221184=6, krylov=40, horizon=0.25),
        # Yield gradients with the FP64 Taylor passes on a subset, forward and backward.
        dict(name="gradient_c128_864_x16", kind="gradient", vectors=16, precision="c128", horizon=0.5, **six),
        # The same at full size (the differentiation workload, few vectors, short horizon).
        dict(name="gradient_c128_221184_x4", kind="gradient", vectors=4, precision="c128", horizon=0.1, **full),
        # The factorized exact ensemble yields of an uncoupled subset over field orientations.
        dict(name="factorized_3456_x6", kind="factorized", orientations=6, lifetimes=3, l1=2, lh=2, r1=1, rh=3),
    ]


# Nuclear subsets of the full pair, smallest to largest (dimensions 96 .. 110,592).
_SUBSETS = [(1, 1, 0, 2), (1, 1, 1, 1), (2, 1, 1, 2), (1, 3, 0, 3), (2, 2, 1, 3), (2, 3, 1, 4), (1, 4, 1, 5),
            (2, 4, 1, 5), (2, 5, 1, 5)]


def _horizon(rng, low, high):
    """A horizon between low and high (logarithmic), on the observation grid."""
    us = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(8, round(us / GRID_US)) * GRID_US


def draw(rng):
    """One more case of the listed ones' ranges: any kind, odd sizes among them."""
    kind = rng.choice(["matvec", "apply", "plain", "plain", "batched", "batched", "batched", "uneven", "gradient",
                       "factorized"])
    l1, lh, r1, rh = rng.choice(_SUBSETS)
    shape = dict(l1=l1, lh=lh, r1=r1, rh=rh)
    n = 4 * 3 ** (l1 + r1) * 2 ** (lh + rh)
    if kind == "matvec":
        return dict(kind=kind, **shape)
    if kind == "apply":
        count = int(round(math.exp(rng.uniform(0.0, math.log(64.0)))))
        return dict(kind=kind, count=count, precision=rng.choice([64, 64, 128]), **shape)
    if kind == "plain":
        top = 0.5 if n <= 4000 else 0.05
        return dict(kind=kind, horizon=_horizon(rng, 0.02, top), kmin=8, kmax=rng.choice([24, 30, 40]), **shape)
    if kind == "batched":
        orientations, vectors = rng.randint(1, 9), rng.randint(1, 5)
        top = 2.0 if n <= 4000 else 0.4
        return dict(kind=kind, orientations=orientations, vectors=vectors, krylov=rng.choice([16, 24, 32, 40]),
                    horizon=_horizon(rng, 0.1, top), final=rng.random() < 0.5, **shape)
    if kind == "uneven":
        return dict(kind=kind, n864=rng.randint(1, 24), n13824=rng.randint(1, 12), n221184=rng.randint(0, 4),
                    krylov=rng.choice([24, 32, 40]), horizon=_horizon(rng, 0.05, 0.25))
    if kind == "gradient":
        top = 0.5 if n <= 4000 else 0.1
        return dict(kind=kind, vectors=rng.randint(1, 12), precision=rng.choice(["c128", "c128", "c64"]),
                    horizon=_horizon(rng, 0.05, top), **shape)
    l1, lh, r1, rh = rng.choice(_SUBSETS[1:5])
    return dict(kind=kind, orientations=rng.randint(1, 6), lifetimes=rng.randint(1, 4), l1=l1, lh=lh, r1=r1, rh=rh)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _system(case, seed, **knobs):
    from rpm_b200 import synthetic

    return synthetic.make_system(seed % (1 << 31), (case["l1"], case["lh"]), (case["r1"], case["rh"]), **knobs)


def _subset(seed, per_radical):
    from rpm_b200 import synthetic

    full = synthetic.make_system(seed % (1 << 31), (2, 5), (1, 6))
    return full if per_radical == 7 else synthetic.prefix_system(full, per_radical)


def _hamiltonian(system, terms):
    import rpm_b200 as rb

    return rb.CompiledFullPairHamiltonian(system.dimensions, terms, left_axes=system.left_axes,
                                          right_axes=system.right_axes)


def _directions(count):
    from rpm_b200 import synthetic

    return synthetic.fibonacci_sphere(count)


def _grid(horizon):
    return np.arange(int(round(horizon / GRID_US)) + 1) * GRID_US


def _states(n, count, seed):
    """``count`` electron-singlet states with random nuclear phases, (count, n) complex128 on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = n // 4
    phase = 2.0 * math.pi * torch.rand((count, m), generator=g, device="cuda", dtype=torch.float64)
    nuclei = torch.polar(torch.full_like(phase, 1.0 / math.sqrt(2.0 * m)), phase)
    psi = torch.zeros((count, n), dtype=torch.complex128, device="cuda")
    psi[:, m:2 * m] = nuclei
    psi[:, 2 * m:3 * m] = -nuclei
    return psi


def _vectors(n, count, seed, precision):
    """``count`` normalised complex Gaussian vectors, as a Krylov basis holds them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((count, n), generator=g, device="cuda", dtype=torch.complex128)
    x /= torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return x.to(torch.complex64) if precision == 64 else x


def _sweep(case, seed):
    """The systems' terms of an orientation sweep and the system of each trajectory."""
    s = _system(case, seed)
    terms = [s.terms(th, ph) for th, ph in _directions(case["orientations"])]
    return s, terms, np.repeat(np.arange(case["orientations"], dtype=np.int32), case["vectors"])


def _uneven(case, seed):
    """(system, terms) and the states of each trajectory of an uneven batch, sizes interleaved."""
    rng = np.random.default_rng(seed)
    members = [(3, k) for k in range(case["n864"])] + [(5, k) for k in range(case["n13824"])]
    members += [(7, k) for k in range(case["n221184"])]
    subsets = {per: _subset(seed, per) for per in {p for p, _ in members}}
    systems, states = [], {}
    counts = {3: case["n864"], 5: case["n13824"], 7: case["n221184"]}
    for per, s in sorted(subsets.items()):
        states[per] = _states(s.dimension, counts[per], seed + per)
    order = rng.permutation(len(members))
    rows = []
    for at in order:
        per, k = members[at]
        th, ph = math.acos(rng.uniform(-1.0, 1.0)), rng.uniform(0.0, 2.0 * math.pi)
        systems.append((subsets[per], subsets[per].terms(th, ph)))
        rows.append(states[per][k])
    return systems, rows


def _gradient_inputs(case, seed):
    rng = np.random.default_rng(seed)
    s = _system(case, seed)
    params = np.array([50.0, math.acos(rng.uniform(-1.0, 1.0)), rng.uniform(0.0, 2.0 * math.pi),
                       rng.uniform(50.0, 500.0), 1.0])
    # the transverse pulse covers the middle of the horizon
    points = int(round(case["horizon"] / GRID_US))
    start, length = points // 4, max(1, points // 2)
    return s, params, start * GRID_US, length * GRID_US, _states(s.dimension, case["vectors"], seed)


def prepare(case, seed):
    import rpm_b200 as rb
    from rpm_b200.batched import BatchedPropagator

    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("matvec", "apply"):
        s = _system(case, seed)
        st["h"] = _hamiltonian(s, s.terms(math.pi / 4, 0.0))
        count, precision = case.get("count", 1), case.get("precision", 128)
        x = _vectors(s.dimension, count, seed, precision)
        if kind == "matvec":
            st["x"] = x[0]
        else:
            st.update(x=x, out=torch.empty_like(x), count=count, precision=precision)
    elif kind == "plain":
        s = _system(case, seed)
        h = _hamiltonian(s, s.terms(math.pi / 4, 0.0))
        st["propagator"] = rb.AdaptiveLanczosPropagator(
            h, minimum_dimension=case["kmin"], maximum_dimension=case["kmax"],
            state_error_budget=PLAIN_BUDGET * case["horizon"] / HORIZON_US)
        st["observable"] = rb.SingletPopulationObservable(s.dimensions)
        st["psi"] = _states(s.dimension, 1, seed)[0]
        st["times"] = _grid(case["horizon"])
    elif kind == "batched":
        s, terms, index = _sweep(case, seed)
        st["propagator"] = BatchedPropagator([_hamiltonian(s, t) for t in terms], krylov_dimension=case["krylov"],
                                             state_error_budget=BATCH_BUDGET * case["horizon"] / HORIZON_US)
        st.update(psi=_states(s.dimension, index.size, seed), index=index, times=_grid(case["horizon"]),
                  final=case["final"])
    elif kind == "uneven":
        systems, rows = _uneven(case, seed)
        hams = [_hamiltonian(s, t) for s, t in systems]
        for h in hams:
            h.set_recombination_rates(1.0, 2.0)
        st["propagator"] = BatchedPropagator(hams, krylov_dimension=case["krylov"],
                                             state_error_budget=BATCH_BUDGET * case["horizon"] / HORIZON_US)
        st.update(psi=rows, index=np.arange(len(rows), dtype=np.int32), times=_grid(case["horizon"]))
    elif kind == "gradient":
        from rpm_b200.adjoint import AdjointYieldGradient, ParametricRadicalPair

        s, params, start, length, psi = _gradient_inputs(case, seed)
        model = ParametricRadicalPair(s, pulse_start_us=start, pulse_duration_us=length)
        st["engine"] = AdjointYieldGradient(model, precision=case["precision"])
        st.update(params=params, psi=psi, times=_grid(case["horizon"]))
    elif kind == "factorized":
        s, terms = _factorized_terms(case, seed)
        st["hamiltonians"] = [_hamiltonian(s, t) for t in terms]
        st["lifetimes"] = _lifetimes(case)
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return st


def _factorized_terms(case, seed):
    """An uncoupled pair (no exchange, no dipolar term) over field orientations."""
    s = _system(case, seed, exchange_J_mT=0.0, dipolar_D_mT=0.0)
    return s, [s.terms(th, ph) for th, ph in _directions(case["orientations"])]


def _lifetimes(case):
    return [1.0, 0.2, 5.0, 2.0][:case["lifetimes"]]


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(st):
    kind = st["kind"]
    if kind == "matvec":
        return st["h"].matvec(st["x"])
    if kind == "apply":
        st["h"].apply(st["x"], st["out"], batch=st["count"], precision=st["precision"])
        return st["out"]
    if kind == "plain":
        r = st["propagator"].propagate(st["psi"], st["times"], st["observable"])
        return r.observable_values, r.final_state
    if kind == "batched":
        r = st["propagator"].propagate(st["psi"], st["times"], system_index=st["index"], lifetime_us=LIFETIME_US,
                                       return_final_states=st["final"])
        return [r.observable_values, r.yields] + ([r.final_states] if st["final"] else [])
    if kind == "uneven":
        r = st["propagator"].propagate(st["psi"], st["times"], system_index=st["index"])
        return r.observable_values, r.yields
    if kind == "gradient":
        r = st["engine"](st["params"], st["psi"], st["times"], LIFETIME_US)
        return r.yields, r.gradients, r.populations
    from rpm_b200.factorized import factorized_singlet_yields

    return factorized_singlet_yields(st["hamiltonians"], st["lifetimes"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

def _macs(l1, lh, r1, rh):
    """Complex multiply-adds of H psi per component: per nucleus the transitions
    to its other levels from both electron values, the merged diagonal (half a
    multiply-add) and electron flip of each radical, and the pair operator."""
    return 2.0 * (lh + rh) + 4.0 * (l1 + r1) + 3.0 + 2.0


def _half_width(system, terms):
    """Half the spectrum's width: H psi applications per microsecond that a
    propagation needs at least (a polynomial of degree rho t resolves exp(-i H t))."""
    lo, hi = _bounds(_pair(system, terms, "cpu"))
    return 0.5 * (hi - lo)


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        total = {"bytes": 0.0, "flops": 0.0}
        for per, shape, count in ((3, (2, 1, 1, 2), case["n864"]), (5, (2, 3, 1, 4), case["n13824"]),
                                  (7, (2, 5, 1, 6), case["n221184"])):
            if count:
                s = _subset(1, per)
                steps = _half_width(s, s.terms(math.pi / 4, 0.0)) * case["horizon"]
                total["bytes"] += 2.0 * 8.0 * s.dimension * count * steps
                total["flops"] += 8.0 * _macs(*shape) * s.dimension * count * steps
        return total
    shape = (case["l1"], case["lh"], case["r1"], case["rh"])
    n = 4 * 3 ** (shape[0] + shape[2]) * 2 ** (shape[1] + shape[3])
    flops = 8.0 * _macs(*shape) * n
    if kind in ("matvec", "apply"):
        count = case.get("count", 1)
        return {"bytes": 2.0 * (8 if case.get("precision", 128) == 64 else 16) * n * count, "flops": flops * count}
    if kind == "factorized":
        # Hermitian eigen-decompositions with vectors (about 9 n^3 complex multiply-adds)
        dl, dr = 2 * 3 ** shape[0] * 2 ** shape[1], 2 * 3 ** shape[2] * 2 ** shape[3]
        per = 9.0 * (dl ** 3 + dr ** 3)
        return {"bytes": 16.0 * 2 * (dl * dl + dr * dr) * case["orientations"], "flops": 8.0 * per * case["orientations"]}
    s = _system(case, 1)
    steps = _half_width(s, s.terms(math.pi / 4, 0.0)) * case["horizon"]
    size, vectors = 16, 1
    if kind == "batched":
        size, vectors = 8, case["orientations"] * case["vectors"]
    elif kind == "gradient":
        # forward, and backward for the state and the adjoint
        size, vectors = (8 if case["precision"] == "c64" else 16), 3 * case["vectors"]
    return {"bytes": 2.0 * size * n * vectors * steps, "flops": flops * vectors * steps}


# ---------------------------------------------------------------------------
# The same in 64 bits with plain torch
# ---------------------------------------------------------------------------
# The state is held as Y[b, (eA, l), (eB, r)]: H Y = L Y + Y R^T + P Y with
# dense radical blocks L, R and the 4 x 4 electron-pair operator P.

def _embed(op, axes, group, dims):
    """An operator on some axes of a group as a dense matrix of the whole group."""
    rest = [a for a in group if a not in axes]
    d = math.prod(dims[a] for a in rest)
    full = torch.kron(op, torch.eye(d, dtype=op.dtype, device=op.device))
    order = list(axes) + rest
    k = len(order)
    full = full.reshape([dims[a] for a in order] * 2)
    at = [order.index(a) for a in group]
    size = math.prod(dims[a] for a in group)
    return full.permute(at + [k + v for v in at]).reshape(size, size)


def _pair(system, terms, device="cuda"):
    dims = system.dimensions
    groups = (list(system.left_axes), list(system.right_axes))
    blocks = [torch.zeros([math.prod(dims[a] for a in g)] * 2, dtype=torch.complex128, device=device) for g in groups]
    pair = torch.zeros((4, 4), dtype=torch.complex128, device=device)
    for t in terms:
        op = torch.as_tensor(np.asarray(t.operator, dtype=complex), device=device)
        axes = list(t.axes)
        if axes == [0, 1]:
            pair += op
        else:
            side = 0 if set(axes) <= set(groups[0]) else 1
            blocks[side] += _embed(op, axes, groups[side], dims)
    return blocks[0], blocks[1], pair


def _bounds(h):
    """An interval that holds the spectrum."""
    lo = hi = 0.0
    for block in h:
        w = torch.linalg.eigvalsh(0.5 * (block + block.conj().T))
        lo, hi = lo + float(w[0]), hi + float(w[-1])
    return lo, hi


def _to_blocks(psi, dl, dr):
    return psi.reshape(-1, 2, 2, dl // 2, dr // 2).transpose(2, 3).reshape(-1, dl, dr)


def _from_blocks(y):
    b, dl, dr = y.shape
    return y.reshape(b, 2, dl // 2, 2, dr // 2).transpose(2, 3).reshape(b, -1)


def _act(h, y):
    left, right, pair = h
    b, dl, dr = y.shape
    out = torch.matmul(left, y)
    out += torch.matmul(y.reshape(b * dl, dr), right.T).reshape(b, dl, dr)
    if bool((pair != 0).any()):
        v = y.reshape(b, 2, dl // 2, 2, dr // 2)
        out += torch.einsum("acef,belfr->balcr", pair.reshape(2, 2, 2, 2), v).reshape(b, dl, dr)
    return out


def _chebyshev(times, centre, width, terms):
    """Coefficients of exp(-i H t) = sum_k c_k(t) T_k((H - centre) / width), (times, terms)."""
    nodes = 4 * terms
    theta = math.pi * (np.arange(nodes) + 0.5) / nodes
    f = np.exp(-1j * width * np.outer(times, np.cos(theta)))
    c = (2.0 / nodes) * f @ np.cos(np.outer(theta, np.arange(terms)))
    c[:, 0] *= 0.5
    return np.exp(-1j * centre * np.asarray(times))[:, None] * c


def _exact_populations(h, psi, times):
    """Singlet populations (states, times) and the final states of exp(-i H t)
    psi: Chebyshev steps of about 20 / width, every observation time of a step
    from the Gram of the step's singlet-projected vectors."""
    lo, hi = _bounds(h)
    centre, width = 0.5 * (lo + hi), max(0.5 * (hi - lo) * 1.01 + 1.0, 1e-3)
    dl, dr = h[0].shape[0], h[1].shape[0]
    y = _to_blocks(psi, dl, dr)
    dt = float(times[1] - times[0])
    per = max(1, min(len(times) - 1, int(20.0 / (width * dt))))
    terms = int(width * per * dt) + 50
    values = torch.empty((psi.shape[0], len(times)), dtype=torch.float64, device=psi.device)

    def singlet(v):
        w = v.reshape(-1, 2, dl // 2, 2, dr // 2)
        return ((w[:, 0, :, 1] - w[:, 1, :, 0]) / math.sqrt(2.0)).reshape(v.shape[0], -1)

    values[:, 0] = torch.linalg.vector_norm(singlet(y), dim=1) ** 2
    k0 = 0
    while k0 < len(times) - 1:
        k1 = min(k0 + per, len(times) - 1)
        c = torch.as_tensor(_chebyshev(times[k0 + 1:k1 + 1] - times[k0], centre, width, terms), device=psi.device)
        before, now = None, y
        end = c[-1, 0] * now
        amplitudes = [singlet(now)]
        for k in range(1, terms):
            hv = (_act(h, now) - centre * now) / width
            before, now = now, (hv if before is None else 2.0 * hv - before)
            end += c[-1, k] * now
            amplitudes.append(singlet(now))
        a = torch.stack(amplitudes, dim=1)                      # (states, terms, N/4)
        gram = torch.matmul(a.conj(), a.transpose(1, 2))        # <a_k, a_l>
        values[:, k0 + 1:k1 + 1] = torch.einsum("tk,bkl,tl->bt", c.conj(), gram, c).real
        y, k0 = end, k1
        del a, amplitudes
    return values, _from_blocks(y)


def _simpson(times, values, lifetime):
    """Composite Simpson (scipy's odd and even rules) of exp(-t / tau) P / tau over a uniform grid."""
    f = values * np.exp(-times / lifetime) / lifetime
    n, h = times.size, times[1] - times[0]
    stop = n if n % 2 else n - 1
    total = h / 3.0 * (f[:, 0:stop - 2:2] + 4.0 * f[:, 1:stop - 1:2] + f[:, 2:stop:2]).sum(axis=1)
    if n % 2 == 0:
        total = total + h * (5.0 / 12.0 * f[:, -1] + 2.0 / 3.0 * f[:, -2] - 1.0 / 12.0 * f[:, -3])
    return total


def _exact_gradient(case, seed):
    """Yields, gradients and populations of the gradient case: interval
    propagators and their derivatives (the exponential of a 2 x 2 block matrix),
    states and tangents marched over the grid."""
    s, params, start, length, psi = _gradient_inputs(case, seed)
    times = _grid(case["horizon"])
    n = s.dimension

    def dense(terms):
        left, right, pair = _pair(s, terms)
        dl, dr = left.shape[0], right.shape[0]
        eye = torch.eye(dl * dr, dtype=torch.complex128, device="cuda")
        # rows of eye as states Y: columns of the operator; back to the state order
        cols = _act((left, right, pair), eye.reshape(-1, dl, dr))
        order = _from_blocks(torch.arange(dl * dr, device="cuda").reshape(1, dl, dr))[0]
        return cols.reshape(dl * dr, dl * dr).T[order][:, order]

    zero = dense(s.terms(0.0, 0.0, field_microT=0.0, hyperfine_scale=0.0))
    hyper = dense(s.terms(0.0, 0.0, field_microT=0.0)) - zero
    axis = [dense(s.terms(0.0, 0.0, field_microT=0.0, hyperfine_scale=0.0, extra_field_mT=e)) - zero for e in np.eye(3)]
    b, th, ph, amp, scale = params
    st_, ct, sp, cp = math.sin(th), math.cos(th), math.sin(ph), math.cos(ph)
    unit = np.array([st_ * cp, st_ * sp, ct])
    e_th = np.array([ct * cp, ct * sp, -st_])
    e_ph = np.array([-sp, cp, 0.0])
    dt = GRID_US
    us = []
    for pulsed in (0, 1):
        a = 1e-6 * amp * pulsed
        field = 1e-3 * b * unit + a * e_th
        slopes = [1e-3 * unit, 1e-3 * b * e_th - a * unit, 1e-3 * b * st_ * e_ph + a * ct * e_ph, 1e-6 * pulsed * e_th]
        combine = lambda v: sum(float(x) * m for x, m in zip(v, axis))  # noqa: E731
        h = zero + scale * hyper + combine(field)
        ds = [combine(v) for v in slopes] + [hyper]
        rows = []
        for d in ds:
            blk = torch.zeros((2 * n, 2 * n), dtype=torch.complex128, device="cuda")
            blk[:n, :n] = blk[n:, n:] = -1j * dt * h
            blk[:n, n:] = -1j * dt * d
            e = torch.linalg.matrix_exp(blk)
            rows.append(e[:n, n:])
        us.append((e[:n, :n], torch.cat(rows)))
    mid = 0.5 * (times[:-1] + times[1:])
    inside = (mid > start) & (mid < start + length)
    m = n // 4
    y = psi.T.contiguous()
    tangent = torch.zeros((5, n, y.shape[1]), dtype=torch.complex128, device="cuda")
    pops, slopes = [], []

    def observe():
        a = (y[m:2 * m] - y[2 * m:3 * m]) / math.sqrt(2.0)
        d = (tangent[:, m:2 * m] - tangent[:, 2 * m:3 * m]) / math.sqrt(2.0)
        pops.append((a.abs() ** 2).sum(0))
        slopes.append(2.0 * (a.conj() * d).sum(1).real)

    observe()
    for k in range(times.size - 1):
        u, du = us[int(inside[k])]
        tangent = torch.matmul(u, tangent) + torch.matmul(du, y).reshape(5, n, -1)
        y = u @ y
        observe()
    values = torch.stack(pops, 1).cpu().numpy()
    slopes = torch.stack(slopes, 2).cpu().numpy()  # (5, vectors, times)
    yields = _simpson(times, values, LIFETIME_US)
    grads = np.stack([_simpson(times, v, LIFETIME_US) for v in slopes], axis=1)
    return yields, grads, values


def _exact_factorized(case, seed):
    """The binned convolution of the two radicals' transition lines, in plain NumPy."""
    s, terms = _factorized_terms(case, seed)
    lifetimes = _lifetimes(case)
    delta = (1.0 / max(lifetimes)) / 8.0
    spin = (np.array([[0.0, 0.5], [0.5, 0.0]], dtype=complex), np.array([[0.0, -0.5j], [0.5j, 0.0]]),
            np.array([[0.5, 0.0], [0.0, -0.5]], dtype=complex))
    yields, initial = np.empty((len(terms), len(lifetimes))), np.empty(len(terms))
    for row, t in enumerate(terms):
        spectra = []
        for block in [v.cpu().numpy() for v in _pair(s, t)[:2]]:
            lam, vec = np.linalg.eigh(block)
            d = lam.size
            half = int(math.ceil((lam[-1] - lam[0]) / delta)) + 3
            ops = [vec.conj().T @ np.kron(p, np.eye(d // 2)) @ vec for p in spin]
            at = (lam[:, None] - lam[None, :]).reshape(-1) / delta + half
            low = np.floor(at).astype(np.int64)
            part = at - low
            grids = []
            for p in ops:
                for q in ops:
                    w = (p * q.T).reshape(-1) / (d // 2)
                    g = np.zeros(2 * half + 1, dtype=complex)
                    for re, unit in ((w.real, 1.0), (w.imag, 1j)):
                        g += unit * np.bincount(low, re * (1.0 - part), g.size)
                        g += unit * np.bincount(low + 1, re * part, g.size)
                    grids.append(g)
            spectra.append((half, grids))
        (ha, ga), (hb, gb) = spectra
        size = 2 * (ha + hb) + 1
        conv = sum(np.fft.ifft(np.fft.fft(a, size) * np.fft.fft(b, size)) for a, b in zip(ga, gb))
        omega = (np.arange(size) - (ha + hb)) * delta
        initial[row] = (0.25 + conv.sum()).real
        for col, tau in enumerate(lifetimes):
            yields[row, col] = (0.25 + (conv * (1.0 / tau) / (1.0 / tau - 1j * omega)).sum()).real
    return yields, initial


def exact(case, seed):
    kind = case["kind"]
    if kind in ("matvec", "apply"):
        s = _system(case, seed)
        h = _pair(s, s.terms(math.pi / 4, 0.0))
        x = _vectors(s.dimension, case.get("count", 1), seed, case.get("precision", 128)).to(torch.complex128)
        out = _from_blocks(_act(h, _to_blocks(x, h[0].shape[0], h[1].shape[0])))
        return out[0] if kind == "matvec" else out
    if kind == "plain":
        s = _system(case, seed)
        v, psi = _exact_populations(_pair(s, s.terms(math.pi / 4, 0.0)), _states(s.dimension, 1, seed),
                                    _grid(case["horizon"]))
        return v[0], psi[0]
    if kind == "batched":
        s, terms, index = _sweep(case, seed)
        times, psi = _grid(case["horizon"]), _states(s.dimension, index.size, seed)
        parts = [_exact_populations(_pair(s, t), psi[torch.from_numpy(index == k).cuda()], times)
                 for k, t in enumerate(terms)]
        values = torch.cat([p[0] for p in parts]).cpu().numpy()
        # (the state buffer's rows are padded: the final states have no plain counterpart of its layout)
        return [values, _simpson(times, values, LIFETIME_US)] + ([None] if case["final"] else [])
    if kind == "uneven":
        systems, rows = _uneven(case, seed)
        times = _grid(case["horizon"])
        values = []
        # kS = 1, kT = 2: exp(-t / 2) is factored out, -(i/2) P_T is left of the decay
        triplet = np.eye(4, dtype=complex)
        triplet[1:3, 1:3] = 0.5
        for (s, t), row in zip(systems, rows):
            left, right, pair = _pair(s, t)
            pair = pair - 0.5j * torch.as_tensor(triplet, device="cuda")
            values.append(_exact_populations((left, right, pair), row[None], times)[0][0])
        values = torch.stack(values).cpu().numpy()
        return values, _simpson(times, values, 1.0)
    if kind == "gradient":
        n = 4 * 3 ** (case["l1"] + case["r1"]) * 2 ** (case["lh"] + case["rh"])
        return _exact_gradient(case, seed) if n <= 1200 else None
    return _exact_factorized(case, seed)

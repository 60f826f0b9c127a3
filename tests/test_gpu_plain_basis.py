"""One-launch Lanczos basis of the plain path and coefficients straight from the tridiagonal (GPU)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hermitian(rng, d):
    a = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
    return a + a.conj().T


def _system(rng, left, right, interleaved=False):
    """Random pair on the dimensions ``left`` and ``right``; interleaved: nuclei of both radicals alternate."""
    import rpm_b200 as rb

    order = sorted(range(len(left) + len(right)), key=lambda k: (k if k < len(left) else k - len(left), k)) \
        if interleaved else list(range(len(left) + len(right)))
    sizes = left + right
    dims = (2, 2) + tuple(sizes[k] for k in order)
    axis = {k: pos + 2 for pos, k in enumerate(order)}
    terms = [rb.LocalTerm((0,), _hermitian(rng, 2)), rb.LocalTerm((1,), _hermitian(rng, 2)),
             rb.LocalTerm((0, 1), _hermitian(rng, 4))]
    for k in axis:
        terms.append(rb.LocalTerm((0 if k < len(left) else 1, axis[k]), _hermitian(rng, 2 * sizes[k])))
    return rb.CompiledFullPairHamiltonian(dims, terms, left_axes=(0,) + tuple(axis[k] for k in range(len(left))),
                                          right_axes=(1,) + tuple(axis[k] for k in range(len(left), len(sizes))))


def _basis(h, state, m, tol=1e-14):
    import torch

    from rpm_b200 import _lib

    basis = torch.empty((m, h.dimension), dtype=torch.complex128, device="cuda")
    alpha = torch.zeros(m, dtype=torch.float64, device="cuda")
    beta = torch.zeros(max(m, 1), dtype=torch.float64, device="cuda")
    actual, norm = ctypes.c_int(), ctypes.c_double()
    _lib.call("rpm_lanczos_basis", h._system.handle, _lib.ptr(state), m, tol, _lib.ptr(basis), _lib.ptr(alpha),
              _lib.ptr(beta), ctypes.byref(actual), ctypes.byref(norm), _lib.stream_handle())
    k = actual.value
    return basis[:k], alpha[:k].cpu().numpy(), beta[:max(k - 1, 0)].cpu().numpy(), norm.value


# nuclear index counts: a few; below, at and above the two-block size (256); a
# last block that is not full (576 / 4 blocks is, 864 / 6 is, 1,440 / 11 is not);
# a basis that outgrows the blocks' shared memory (27,648 indices x 40 vectors);
# the cap of 128 vectors; nuclei of both radicals mixed (the general sequence)
@pytest.mark.parametrize("left,right,m,mixed", [
    ((2,), (2,), 5, False), ((15,), (16,), 20, False), ((16,), (16,), 20, False), ((3, 3), (2, 2, 2, 2, 2), 33, False),
    ((5, 3, 2), (3, 2, 2, 2, 2), 24, False), ((3, 2, 2, 2), (3, 2, 2, 2), 128, False),
    ((3, 3, 3, 2, 2), (2, 2, 2, 2, 2, 2, 2, 2), 40, False), ((3, 2), (2, 2), 20, True)])
def test_basis_is_orthonormal_and_satisfies_the_recurrence(left, right, m, mixed):
    """Bars: 1e-12, two Gram-Schmidt passes and H psi at FP64 rounding (1e-13 of the norm)."""
    import torch

    rng = np.random.default_rng(len(left) * 31 + m)
    h = _system(rng, left, right, mixed)
    n = h.dimension
    v = 3.0 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    state = torch.from_numpy(v).to("cuda")
    basis, alpha, beta, norm = _basis(h, state, m)
    k = basis.shape[0]
    assert k == min(m, n)
    assert abs(norm - np.linalg.norm(v)) <= 1e-13 * norm
    assert float(torch.linalg.vector_norm(basis[0] * norm - state)) <= 1e-13 * norm
    gram = (basis.conj() @ basis.T).cpu().numpy()
    assert np.max(np.abs(gram - np.eye(k))) <= 1e-12
    t = np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1)
    hv = torch.empty_like(basis)
    h.apply(basis, hv, batch=k)
    got = (basis.conj() @ hv.T).cpu().numpy()
    scale = np.max(np.abs(np.linalg.eigvalsh(t)))
    assert np.max(np.abs(got - t)) <= 1e-12 * scale
    resid = hv[:k - 1] - torch.from_numpy(t[:k - 1].astype(complex)).to("cuda") @ basis
    assert float(resid.abs().max()) <= 1e-12 * scale


def test_basis_breakdown_and_zero_state():
    """A state in a four-dimensional invariant subspace stops at its size; a zero state has norm 0."""
    import rpm_b200 as rb
    import torch

    # no transitions between the nuclear levels: each nuclear index is invariant
    rng = np.random.default_rng(2)
    dims, diag = (2, 2, 16, 16), lambda d: np.diag(rng.normal(size=d)).astype(complex)
    terms = [rb.LocalTerm((0,), _hermitian(rng, 2)), rb.LocalTerm((1,), _hermitian(rng, 2)),
             rb.LocalTerm((2,), diag(16)), rb.LocalTerm((3,), diag(16))]
    h = rb.CompiledFullPairHamiltonian(dims, terms, left_axes=(0, 2), right_axes=(1, 3))
    v = np.zeros((4, 256), complex)
    v[:, 37] = rng.standard_normal(4) + 1j * rng.standard_normal(4)
    basis, _, _, _ = _basis(h, torch.from_numpy(v.reshape(-1)).to("cuda"), 20, tol=1e-10)
    assert basis.shape[0] == 4
    with pytest.raises(ValueError):
        _basis(h, torch.zeros(1024, dtype=torch.complex128, device="cuda"), 20)


# one and two values per lane, four above 64; times whose series is split (radius
# x time above 256), zero time, a zero matrix (radius 0)
@pytest.mark.parametrize("size", [1, 2, 32, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("spread,times", [(1.0, (0.0, 1e-3, 0.7, 3.0)), (60.0, (0.02, 1.0, 9.0)), (0.0, (1.0,))])
def test_coefficients_match_dense_exponential(size, spread, times):
    """Bar 1e-13 + 1e-15 radius x time: FP64 rounding of as many series terms, and of the dense phases."""
    import torch

    from rpm_b200 import _lib

    rng = np.random.default_rng(size)
    alpha = spread * rng.uniform(-1, 1, size)
    beta = spread * rng.uniform(0.2, 1, size)
    t = np.diag(alpha) + np.diag(beta[:size - 1], 1) + np.diag(beta[:size - 1], -1)

    def exp_e1(d, time):
        w, u = np.linalg.eigh(t[:d, :d])
        out = np.zeros(size, complex)
        out[:d] = u @ (np.exp(-1j * w * time) * u[0])
        return out

    pairs = [(size, max(1, size - 4)), (max(1, size // 2), -1), (size, -1)]
    reqs = (_lib.rpm_krylov_req * (len(pairs) * len(times)))()
    cases = [(hi, lo, time) for hi, lo in pairs for time in times]
    for r, (hi, lo, time) in zip(reqs, cases):
        r.hi, r.lo, r.time = hi, lo, time
    coef = torch.full((len(cases), size), 9.0, dtype=torch.complex128, device="cuda")
    err = np.full(len(cases), -1.0)
    val = np.zeros(len(cases))
    dev = [torch.from_numpy(x).to("cuda") for x in (alpha, beta)]
    _lib.call("rpm_krylov_coefficients", _lib.ptr(dev[0]), _lib.ptr(dev[1]), size, len(cases), reqs, 2.0, 0.5, None, 0,
              _lib.ptr(coef), size, _lib.dptr(err), _lib.dptr(val), _lib.stream_handle())
    got = coef.cpu().numpy()
    for k, (hi, lo, time) in enumerate(cases):
        bar = 1e-13 + 1e-15 * 3.0 * spread * time
        want = exp_e1(hi, time)
        assert np.linalg.norm(got[k, :hi] - want[:hi]) <= bar
        assert np.all(got[k, hi:] == 9.0)
        gap = np.linalg.norm(want - exp_e1(lo, time)) if 0 < lo < hi else 0.0
        assert abs(err[k] - 2.0 * 0.5 * gap) <= 2.0 * bar

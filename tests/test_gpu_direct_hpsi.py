"""Direct complex128 H psi (one launch, any spins, standard layout) against the dense operator (GPU).

Bar: 1e-13 relative, the other FP64 H psi tests' bar -- a component sums fewer
than 200 products, so its rounding is below 200 x 1.1e-16 of the terms' sizes.
"""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-13

# nuclear dimensions per radical: single nuclei, spins above 1, index counts
# around the kernel's 128-thread blocks (4 .. 2,304 nuclear indices)
SHAPES = [((2,), (2,)), ((3,), (2, 2)), ((5,), (7,)), ((6, 2), (4, 3)), ((2, 2, 2, 2), (2, 2, 2)),
          ((3, 3, 2), (3, 2, 2)), ((16,), (8,)), ((2, 3, 4), (4, 3, 2, 2)), ((3, 2, 2, 2), (3, 2, 2, 2, 2, 2))]


def _terms(rb, rng, left, right, pair):
    def hermitian(d):
        a = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
        return a + a.conj().T

    out = [rb.LocalTerm((0,), hermitian(2)), rb.LocalTerm((1,), hermitian(2))]
    for k, d in enumerate(left + right):
        e = 0 if k < len(left) else 1
        out.append(rb.LocalTerm((e, k + 2), hermitian(2 * d)))
        if k % 2:
            out.append(rb.LocalTerm((k + 2,), hermitian(d)))
    if pair:
        out.append(rb.LocalTerm((0, 1), hermitian(4)))
    return out


def _dense_apply(dims, terms, x):
    """sum of local terms on each column of x by plain NumPy tensor products."""
    t = x.reshape(dims + (-1,))
    out = np.zeros_like(t)
    for term in terms:
        d = [dims[a] for a in term.axes]
        op = np.asarray(term.operator).reshape(d + d)
        y = np.tensordot(op, t, axes=(range(len(d), 2 * len(d)), term.axes))
        out += np.moveaxis(y, range(len(d)), term.axes)
    return out.reshape(x.shape)


@pytest.mark.parametrize("case", range(len(SHAPES)))
@pytest.mark.parametrize("batch,rates", [(1, None), (3, (1.0, 2.5))])
def test_direct_action_matches_dense(case, batch, rates):
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib

    left, right = SHAPES[case]
    dims = (2, 2) + left + right
    rng = np.random.default_rng(100 + case)
    terms = _terms(rb, rng, left, right, pair=case % 2 == 0)
    h = rb.CompiledFullPairHamiltonian(dims, terms, left_axes=(0,) + tuple(range(2, 2 + len(left))),
                                       right_axes=(1,) + tuple(range(2 + len(left), len(dims))))
    n = h.dimension
    x = rng.normal(size=(n, batch)) + 1j * rng.normal(size=(n, batch))
    ref = _dense_apply(dims, terms, x)
    if rates is not None:
        h.set_recombination_rates(*rates)
        # kT > kS: -(i/2) (kT - kS) P_T is added
        ps = np.zeros((4, 4))
        ps[1:3, 1:3] = [[0.5, -0.5], [-0.5, 0.5]]
        extra = rb.LocalTerm((0, 1), -0.5j * (rates[1] - rates[0]) * (np.eye(4) - ps))
        ref = ref + _dense_apply(dims, [extra], x)
    ld = n + 5  # a leading dimension without any alignment but the element's
    xs = torch.full((batch, ld), float("nan"), dtype=torch.complex128, device="cuda")
    xs[:, :n] = torch.from_numpy(np.ascontiguousarray(x.T))
    out = torch.full_like(xs, 7.0)
    _lib.call("rpm_hpsi", h._system.handle, _lib.PREC_C128, _lib.ptr(xs), _lib.ptr(out), batch, ld,
              _lib.stream_handle())
    got = out.cpu().numpy()
    assert np.linalg.norm(got[:, :n].T - ref) <= REL * np.linalg.norm(ref)
    assert np.all(got[:, n:] == 7.0)  # nothing beyond a vector's end is touched


def test_full_size_action_matches_general_kernels():
    """The full system, a batch, against the general cube kernels (forced through the tuning hook)."""
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib, synthetic

    full = synthetic.full_system()
    h = rb.CompiledFullPairHamiltonian(full.dimensions, full.terms(math.pi / 4, 0.3), left_axes=full.left_axes,
                                       right_axes=full.right_axes)
    x = torch.from_numpy(synthetic.random_phase_vectors(full.dimensions, 3, 9)).to("cuda")
    a, b = torch.empty_like(x), torch.empty_like(x)
    h.apply(x, a, batch=3)
    try:
        _lib.call("rpm_set_cube_tuning", 2, 2, 0, 0)
        h.apply(x, b, batch=3)
    finally:
        _lib.call("rpm_set_cube_tuning", 0, 0, 0, 0)
    assert float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b)) < REL


@pytest.mark.parametrize("case", [0, 1, 4, 6])
@pytest.mark.parametrize("batch", [592, 3001])
def test_two_vectors_per_thread_match_dense(case, batch):
    """Batches from which vectors go in pairs (two blocks per SM), even and with one left over."""
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib

    left, right = SHAPES[case]
    dims = (2, 2) + left + right
    rng = np.random.default_rng(300 + case)
    terms = _terms(rb, rng, left, right, pair=case % 4 == 0)
    h = rb.CompiledFullPairHamiltonian(dims, terms, left_axes=(0,) + tuple(range(2, 2 + len(left))),
                                       right_axes=(1,) + tuple(range(2 + len(left), len(dims))))
    n = h.dimension
    x = rng.normal(size=(n, batch)) + 1j * rng.normal(size=(n, batch))
    ref = _dense_apply(dims, terms, x)
    ld = n + 3
    xs = torch.full((batch, ld), float("nan"), dtype=torch.complex128, device="cuda")
    xs[:, :n] = torch.from_numpy(np.ascontiguousarray(x.T))
    out = torch.full_like(xs, 7.0)
    _lib.call("rpm_hpsi", h._system.handle, _lib.PREC_C128, _lib.ptr(xs), _lib.ptr(out), batch, ld,
              _lib.stream_handle())
    got = out.cpu().numpy()
    assert np.linalg.norm(got[:, :n].T - ref) <= REL * np.linalg.norm(ref)
    assert np.all(got[:, n:] == 7.0)


# fastest right nucleus a spin-1/2 (the complex64 form's condition): a lone
# right nucleus, index-pair counts below, at and around one 128-thread block,
# spins above 1/2 before it
SHAPES32 = [((2,), (2,)), ((3,), (2, 2)), ((5, 3), (7, 2)), ((16,), (8, 2)), ((2, 3, 4), (4, 3, 2, 2)),
            ((3, 2, 2, 2), (3, 2, 2, 2, 2, 2))]


@pytest.mark.parametrize("case", range(len(SHAPES32)))
@pytest.mark.parametrize("batch,rates", [(1, None), (3, (1.0, 2.5)), (741, None)])
@pytest.mark.parametrize("offset,pad", [(0, 6), (1, 6), (0, 5)])
def test_complex64_action_matches_dense(case, batch, rates, offset, pad):
    """offset 1 (8-byte aligned) and the odd stride take the general passes; 741 vectors go in pairs, one is left over.

    Bar 2e-6 of the norm: fewer than 200 products of rounding 6e-8, as a random sum 200^0.5 x 6e-8 = 0.9e-6.
    """
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib

    left, right = SHAPES32[case]
    dims = (2, 2) + left + right
    rng = np.random.default_rng(200 + case)
    terms = _terms(rb, rng, left, right, pair=case % 2 == 0)
    h = rb.CompiledFullPairHamiltonian(dims, terms, left_axes=(0,) + tuple(range(2, 2 + len(left))),
                                       right_axes=(1,) + tuple(range(2 + len(left), len(dims))))
    n = h.dimension
    x = (rng.normal(size=(n, batch)) + 1j * rng.normal(size=(n, batch))).astype(np.complex64)
    ref = _dense_apply(dims, terms, x.astype(np.complex128))
    if rates is not None:
        h.set_recombination_rates(*rates)
        ps = np.zeros((4, 4))
        ps[1:3, 1:3] = [[0.5, -0.5], [-0.5, 0.5]]
        extra = rb.LocalTerm((0, 1), -0.5j * (rates[1] - rates[0]) * (np.eye(4) - ps))
        ref = ref + _dense_apply(dims, [extra], x)
    ld = n + pad
    store = torch.full((2, offset + batch * ld), 7.0, dtype=torch.complex64, device="cuda")
    xs, out = (store[k, offset:].view(batch, ld) for k in range(2))
    xs.fill_(float("nan"))
    xs[:, :n] = torch.from_numpy(np.ascontiguousarray(x.T))
    _lib.call("rpm_hpsi", h._system.handle, _lib.PREC_C64, _lib.ptr(xs), _lib.ptr(out), batch, ld,
              _lib.stream_handle())
    got = out.cpu().numpy()
    assert np.linalg.norm(got[:, :n].T - ref) <= 2e-6 * np.linalg.norm(ref)
    assert np.all(got[:, n:] == 7.0)

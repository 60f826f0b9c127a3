"""Factorized exact ensemble singlet yields on the GPU (rpm_quantum_needle_reproduction.py:93-240).

For an uncoupled radical pair (no exchange or dipolar term, D = J = 0) the
Hamiltonian is H_A (x) 1 + 1 (x) H_B and the random-phase ensemble singlet
yield with Haberkorn rate k = 1/tau factorizes:

    Phi_S(tau) = 1/4 + sum_{p,q in x,y,z} sum_{lines a of A, b of B}
                 c^A_pq(a) c^B_pq(b) k / (k - i (w_a + w_b)),

a line of a radical being a pair of its eigenstates (i, j) with frequency
w = lambda_i - lambda_j and weight <i|S_p|j><j|S_q|i> / (nuclear dimension).
As in the reference, the lines of each radical are binned with linear
interpolation onto a frequency grid of spacing (1 / tau_max) / bins, the
two spectra are convolved by FFT, and the kernel k / (k - i w) is summed over
the convolved grid.

GPU work, all in the library's own FP64 kernels: the radical blocks come
from the library's split tables; both radicals' eigen-decompositions run
batched over the field orientations (``rpm_he_eigh_pair``: Householder
tridiagonalisation, implicit tridiagonal QR, back-transformation); the spin
operators in the eigenbases, the binned lines of all nine (p, q), their FFT
convolution (zero-padded to a power of two no shorter than the linear
convolution, which leaves the convolution itself unchanged) and the lifetime
sums are ``rpm_factorized_yields``, all orientations in the same launches.
"""

from __future__ import annotations

import ctypes
import math
from typing import Iterable, Sequence

import numpy as np

from . import _lib
from .engine import _torch

# bytes of workspace per call; more orientations go in several calls
_WORKSPACE_BYTES = 2_000_000_000


def radical_blocks(hamiltonian) -> tuple[np.ndarray, np.ndarray]:
    """Dense radical operators (electron digit slowest) of an uncoupled pair."""
    pair = np.asarray(hamiltonian.electron_pair_operator).reshape(4, 4)
    if np.max(np.abs(pair)) != 0.0:
        raise ValueError("The factorized yield needs an uncoupled radical pair (no electron-pair term).")
    return hamiltonian.left_operator.toarray(), hamiltonian.right_operator.toarray()


def hermitian_eigh(blocks):
    """Eigenvalues (ascending) and eigenvectors (columns) of a batch of
    Hermitian matrices (device tensor, batch x n x n complex128), by the
    library's FP64 solver; the input is Hermitian-symmetrised first."""
    torch = _torch()
    a = (0.5 * (blocks + blocks.conj().transpose(-1, -2))).contiguous()
    batch, n = a.shape[0], a.shape[-1]
    lam = torch.empty((batch, n), dtype=torch.float64, device="cuda")
    vec = torch.empty((batch, n, n), dtype=torch.complex128, device="cuda")
    if n == 1:
        lam.copy_(a[:, 0, 0].real)
        vec.fill_(1.0)
        return lam, vec
    # chunks: at most 65535 matrices (grid limit) and about 2 GB of workspace
    chunk = int(max(1, min(65535, _WORKSPACE_BYTES // (48 * n * n + 64 * n))))
    for b0 in range(0, batch, chunk):
        nb = min(chunk, batch - b0)
        size = ctypes.c_longlong()
        _lib.call("rpm_he_eigh_workspace", n, nb, ctypes.byref(size))
        work = torch.empty(size.value, dtype=torch.uint8, device="cuda")
        _lib.call("rpm_he_eigh", n, nb, _lib.ptr(a[b0:b0 + nb]), _lib.ptr(lam[b0:b0 + nb]), _lib.ptr(vec[b0:b0 + nb]),
                  _lib.ptr(work), _lib.stream_handle())
    return lam, vec


def _eigh_pair(blocks_a, blocks_b):
    """Eigensystems of both radicals (device tensors) of equally many
    orientations, in the same launches; inputs Hermitian-symmetrised."""
    torch = _torch()
    out = []
    for blocks in (blocks_a, blocks_b):
        out.append(torch.empty(blocks.shape[:2], dtype=torch.float64, device="cuda"))
        out.append(torch.empty_like(blocks))
    (lam_a, vec_a, lam_b, vec_b), (na, nb) = out, (blocks_a.shape[-1], blocks_b.shape[-1])
    batch = blocks_a.shape[0]
    chunk = int(max(1, min(32767, _WORKSPACE_BYTES // (48 * (na * na + nb * nb) + 64 * (na + nb)))))
    for k in range(0, batch, chunk):
        s = slice(k, min(k + chunk, batch))
        count = s.stop - k
        size, total = ctypes.c_longlong(), 0
        for n in (na, nb):
            _lib.call("rpm_he_eigh_workspace", n, count, ctypes.byref(size))
            total += size.value
        work = torch.empty(total, dtype=torch.uint8, device="cuda")
        _lib.call("rpm_he_eigh_pair", na, nb, count, _lib.ptr(blocks_a[s]), _lib.ptr(blocks_b[s]), _lib.ptr(lam_a[s]),
                  _lib.ptr(lam_b[s]), _lib.ptr(vec_a[s]), _lib.ptr(vec_b[s]), _lib.ptr(work), _lib.stream_handle())
    return lam_a, vec_a, lam_b, vec_b


def _half_widths(lam: np.ndarray, delta: float) -> np.ndarray:
    """Bins either side of zero that hold every line of each orientation."""
    margin = 3
    return np.array([int(math.ceil(float(gap) / delta)) + margin for gap in lam.max(axis=1) - lam.min(axis=1)],
                    dtype=np.int64)


def factorized_singlet_yields(hamiltonians: Sequence, lifetimes_us: Iterable[float], *,
                              bins_per_linewidth: float = 8.0) -> tuple[np.ndarray, np.ndarray]:
    """Ensemble singlet yields (n_hamiltonians, n_lifetimes) and initial singlet populations.

    ``hamiltonians``: uncoupled :class:`CompiledFullPairHamiltonian` objects
    (e.g. one per field orientation).  Mirrors ``solve_orientation`` and
    ``convolved_correlation_spectrum`` of the reference
    (rpm_quantum_needle_reproduction.py:172-240).
    """
    torch = _torch()
    lifetimes = tuple(float(t) for t in lifetimes_us)
    if not lifetimes or min(lifetimes) <= 0.0:
        raise ValueError("Lifetimes must be positive.")
    if bins_per_linewidth < 2.0:
        raise ValueError("bins_per_linewidth must be at least 2.")
    delta = (1.0 / max(lifetimes)) / float(bins_per_linewidth)
    blocks = [radical_blocks(h) for h in hamiltonians]
    # one batched eigen-decomposition of both radicals over all orientations
    lam_a, vec_a, lam_b, vec_b = _eigh_pair(*(torch.from_numpy(np.stack([b[k] for b in blocks])).to("cuda")
                                              for k in (0, 1)))
    da, db, count = lam_a.shape[1], lam_b.shape[1], len(blocks)
    half_a, half_b = (_half_widths(lam.cpu().numpy(), delta) for lam in (lam_a, lam_b))
    times = np.array(lifetimes)
    out = torch.empty((count, 1 + len(lifetimes)), dtype=torch.float64, device="cuda")
    bad = torch.zeros(1, dtype=torch.int32, device="cuda")

    def size(k, n):
        need = ctypes.c_longlong()
        _lib.call("rpm_factorized_workspace", da, db, n, half_a[k:].ctypes.data, half_b[k:].ctypes.data,
                  len(lifetimes), ctypes.byref(need))
        return need.value

    k = 0
    while k < count:
        n = min(count - k, 32767)
        while n > 1 and size(k, n) > _WORKSPACE_BYTES:
            n = (n + 1) // 2
        work = torch.empty(size(k, n), dtype=torch.uint8, device="cuda")
        _lib.call("rpm_factorized_yields", da, db, n, _lib.ptr(lam_a[k:]), _lib.ptr(vec_a[k:]), _lib.ptr(lam_b[k:]),
                  _lib.ptr(vec_b[k:]), delta, half_a[k:].ctypes.data, half_b[k:].ctypes.data, times.ctypes.data,
                  len(lifetimes), _lib.ptr(out[k:]), _lib.ptr(bad), _lib.ptr(work), _lib.stream_handle())
        k += n
    if int(bad.item()):
        raise ValueError("Frequency grid is too small for transition spectrum.")
    values = out.cpu().numpy()
    return np.ascontiguousarray(values[:, 1:]), np.ascontiguousarray(values[:, 0])

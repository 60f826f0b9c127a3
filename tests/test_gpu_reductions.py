"""Norms and singlet populations (rpm_norm, rpm_singlet_population) against NumPy, around block edges (GPU).

Bar: 1e-14 relative -- sums of n nonnegative FP64 squares added in blocks of
at most a few thousand, each rounding below 1.1e-16 of a partial sum.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(4, 1), (36, 70000), (1020, 3), (1024, 2), (4100, 5), (65536 + 4, 2), (221184, 1)])
def test_singlet_population_matches_numpy(n, batch):
    import torch

    from rpm_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(n)
    ld = n + 3
    x = torch.randn((batch, ld), dtype=torch.complex128, device="cuda", generator=g)
    out = np.full(batch, -1.0)
    _lib.call("rpm_singlet_population", _lib.ptr(x), n, batch, ld, _lib.dptr(out), _lib.stream_handle())
    v = x[:, :n].cpu().numpy().reshape(batch, 4, n // 4)
    ref = 0.5 * (np.abs(v[:, 1] - v[:, 2]) ** 2).sum(axis=1)
    np.testing.assert_allclose(out, ref, rtol=1e-14)


@pytest.mark.parametrize("dims", [(2, 2, 2), (2, 2, 3, 2), (2, 2, 16, 16), (2, 2, 3, 3, 2, 2, 2, 2, 2, 3, 2, 2)])
def test_norm_matches_numpy(dims):
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib

    h = rb.MatrixFreeHamiltonian(dims, [rb.LocalTerm((0,), np.diag([1.0, -1.0]))])
    x = torch.randn(h.dimension, dtype=torch.complex128, device="cuda")
    out = ctypes.c_double()
    _lib.call("rpm_norm", h._system.handle, _lib.ptr(x), ctypes.byref(out), _lib.stream_handle())
    assert out.value == pytest.approx(float(np.linalg.norm(x.cpu().numpy())), rel=1e-14)

"""rpm_tridiag_spectra and rpm_krylov_eval: spectra of the leading blocks of a
tridiagonal, exponentials evaluated against them (GPU)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("size", [1, 2, 33, 64, 128])
def test_spectra_and_evaluation_match_numpy(size):
    """Bars: 20 eps of the norm for eigenvalues and residuals (backward stable QR),
    1e-13 + 20 eps radius x time for the exponentials."""
    import torch

    from rpm_b200 import _lib

    rng = np.random.default_rng(size)
    alpha, beta = rng.uniform(-1, 1, size), rng.uniform(0.2, 1, size)
    t = np.diag(alpha) + np.diag(beta[:size - 1], 1) + np.diag(beta[:size - 1], -1)
    dims = sorted({1, max(1, size // 2), max(1, size - 4), size})
    dev = [torch.from_numpy(x).to("cuda") for x in (alpha, beta)]
    spectra = torch.zeros((len(dims), _lib.RPM_SPECTRUM_DOUBLES), dtype=torch.float64, device="cuda")
    _lib.call("rpm_tridiag_spectra", _lib.ptr(dev[0]), _lib.ptr(dev[1]), len(dims),
              _lib.iptr(np.array(dims, dtype=np.int32)), _lib.ptr(spectra), _lib.stream_handle())
    bar = 20.0 * EPS * 3.0 * np.sqrt(size)
    for d, rec in zip(dims, spectra.cpu().numpy()):
        k = _lib.RPM_MAX_KRYLOV
        assert (rec[0], rec[1]) == (d, 0.0)
        lam, z = rec[2:2 + d], rec[2 + k:].reshape(k, k)[:d, :d]
        np.testing.assert_allclose(np.sort(lam), np.linalg.eigvalsh(t[:d, :d]), rtol=0.0, atol=bar)
        assert np.linalg.norm(t[:d, :d] @ z - z * lam, 2) <= bar
        assert np.linalg.norm(z.T @ z - np.eye(d), 2) <= bar

    def exp_e1(d, time):
        w, u = np.linalg.eigh(t[:d, :d])
        out = np.zeros(size, complex)
        out[:d] = u @ (np.exp(-1j * w * time) * u[0])
        return out

    a = rng.normal(size=(size, size)) + 1j * rng.normal(size=(size, size))
    gram = a @ a.conj().T / size
    cases = [(hi, lo, time) for hi, lo in ((len(dims) - 1, 0), (0, -1)) for time in (0.0, 0.3, 50.0, 1e6)]
    reqs = (_lib.rpm_krylov_req * len(cases))()
    for r, (hi, lo, time) in zip(reqs, cases):
        r.hi, r.lo, r.time = hi, lo, time
    coef = torch.full((len(cases), size), 9.0, dtype=torch.complex128, device="cuda")
    g = torch.from_numpy(gram).to("cuda")
    err, val = np.full(len(cases), -1.0), np.zeros(len(cases))
    _lib.call("rpm_krylov_eval", _lib.ptr(spectra), len(cases), reqs, 2.0, 0.5, _lib.ptr(g), size, _lib.ptr(coef), size,
              _lib.dptr(err), _lib.dptr(val), _lib.stream_handle())
    got = coef.cpu().numpy()
    for k, (hi, lo, time) in enumerate(cases):
        bar = 1e-13 + 20.0 * EPS * 3.0 * time
        d, want = dims[hi], exp_e1(dims[hi], time)
        assert np.linalg.norm(got[k, :d] - want[:d]) <= bar
        assert np.all(got[k, d:] == 9.0)
        gap = np.linalg.norm(want - exp_e1(dims[lo], time)) if lo >= 0 else 0.0
        assert abs(err[k] - gap) <= 2.0 * bar
        assert abs(val[k] - 0.25 * np.vdot(want, gram @ want).real) <= 0.5 * np.linalg.norm(gram, 2) * bar

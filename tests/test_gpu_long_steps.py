"""Krylov exponentials over long times: beyond the reach of the tridiagonal's
Chebyshev series (radius x time 2,048) they come from its spectra, at a cost
that does not depend on the time; what is not finite is refused (GPU).

Bar: 1e-13 + 20 eps radius x time.  Both sides take phases from eigenvalues that
a backward stable solver gives to a few eps of the norm; twenty leaves ten to
each at up to 128 dimensions.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _bar(radius, time):
    return 1e-13 + 20.0 * EPS * radius * time


def _coefficients(alpha, beta, cases, gram=None):
    """(rows, errors, values) of the requests (hi, lo, time); safety 2, norm 0.5."""
    import torch

    from rpm_b200 import _lib

    size = alpha.size
    reqs = (_lib.rpm_krylov_req * len(cases))()
    for r, (hi, lo, time) in zip(reqs, cases):
        r.hi, r.lo, r.time = hi, lo, time
    coef = torch.full((len(cases), size), 9.0, dtype=torch.complex128, device="cuda")
    err, val = np.full(len(cases), -1.0), np.zeros(len(cases))
    dev = [torch.from_numpy(x).to("cuda") for x in (alpha, beta)]
    g = None if gram is None else torch.from_numpy(gram).to("cuda")
    _lib.call("rpm_krylov_coefficients", _lib.ptr(dev[0]), _lib.ptr(dev[1]), size, len(cases), reqs, 2.0, 0.5,
              None if g is None else _lib.ptr(g), 0 if g is None else size, _lib.ptr(coef), size, _lib.dptr(err),
              _lib.dptr(val), _lib.stream_handle())
    return coef.cpu().numpy(), err, val


# one and two values per lane, four above 64; below, just above and far above the
# reach, a short request among long ones
@pytest.mark.parametrize("size", [2, 33, 64, 65, 128])
def test_coefficients_beyond_the_series(size):
    rng = np.random.default_rng(size)
    alpha, beta = rng.uniform(-1, 1, size), rng.uniform(0.2, 1, size)
    t = np.diag(alpha) + np.diag(beta[:size - 1], 1) + np.diag(beta[:size - 1], -1)
    off = np.concatenate([[0.0], beta[:size - 1], [0.0]])
    spread = off[:-1] + off[1:]
    radius = 0.5 * (np.max(alpha + spread) - np.min(alpha - spread))
    a = rng.normal(size=(size, size)) + 1j * rng.normal(size=(size, size))
    gram = a @ a.conj().T / size

    def exp_e1(d, time):
        w, u = np.linalg.eigh(t[:d, :d])
        out = np.zeros(size, complex)
        out[:d] = u @ (np.exp(-1j * w * time) * u[0])
        return out

    times = (1900.0 / radius, 2100.0 / radius, 0.5, 1e5 / radius, 1e9 / radius)
    cases = [(hi, lo, time) for hi, lo in ((size, max(1, size - 4)), (max(1, size // 2), -1)) for time in times]
    got, err, val = _coefficients(alpha, beta, cases, gram)
    for k, (hi, lo, time) in enumerate(cases):
        bar = _bar(3.0, time)
        want = exp_e1(hi, time)
        assert np.linalg.norm(got[k, :hi] - want[:hi]) <= bar
        assert np.all(got[k, hi:] == 9.0)
        gap = np.linalg.norm(want - exp_e1(lo, time)) if 0 < lo < hi else 0.0
        assert abs(err[k] - 2.0 * 0.5 * gap) <= 2.0 * bar
        value = 0.25 * np.vdot(want, gram @ want).real
        assert abs(val[k] - value) <= 0.5 * np.linalg.norm(gram, 2) * bar


@pytest.mark.parametrize("bad", ["time", "alpha", "beta", "nan", "interval"])
def test_coefficients_that_are_not_finite(bad):
    """Infinite times are refused; infinite and NaN entries, and an interval that overflows, are reported."""
    from rpm_b200 import _lib

    alpha, beta = np.linspace(-1, 1, 20), np.ones(20)
    time = np.inf if bad == "time" else 1.0
    if bad == "alpha":
        alpha[3] = np.inf
    elif bad == "beta":
        beta[7] = -np.inf
    elif bad == "nan":
        alpha[0] = np.nan
    elif bad == "interval":
        alpha[:2] = 1.7e308, -1.7e308
    with pytest.raises((ValueError, _lib.RpmError)) as e:
        _coefficients(alpha, beta, [(20, 16, time)])
    assert isinstance(e.value, ValueError) if bad == "time" else e.value.code == _lib.RPM_E_NUMERIC


def _small_system():
    """16 components, a basis of 16 vectors is exact; and its dense Hamiltonian."""
    import torch

    import rpm_b200 as rb

    rng = np.random.default_rng(4)
    a = [rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4)) for _ in range(3)]
    h = rb.CompiledFullPairHamiltonian((2, 2, 2, 2), [rb.LocalTerm(ax, m + m.conj().T) for ax, m in
                                                      zip(((0, 2), (1, 3), (0, 1)), a)], left_axes=(0, 2), right_axes=(1, 3))
    eye = torch.eye(16, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(eye)
    h.apply(eye, out, batch=16)
    psi = rng.normal(size=16) + 1j * rng.normal(size=16)
    return h, out.cpu().numpy().T, psi / np.linalg.norm(psi)


# 2,050 points: more than one chunk of observation points in a step
@pytest.mark.parametrize("points,horizon", [(5, 3e3), (2050, 2e5)])
def test_an_exact_basis_takes_one_long_step(points, horizon):
    import rpm_b200 as rb

    h, dense, psi = _small_system()
    times = np.linspace(0.0, horizon, points)
    w, u = np.linalg.eigh(dense)
    states = (u * (u.conj().T @ psi)) @ np.exp(-1j * np.outer(w, times))
    singlet = (states[4:8] - states[8:12]) / np.sqrt(2.0)
    want = np.sum(np.abs(singlet) ** 2, axis=0)
    bar = 2.0 * _bar(np.max(np.abs(w)), horizon)
    for device in (True, False):
        prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=24, maximum_dimension=32, initial_step_us=1e6,
                                            maximum_step_us=1e6, device_steps=device)
        r = prop.propagate(psi, times, rb.SingletPopulationObservable((2, 2, 2, 2)))
        assert r.stats.accepted_steps == 1
        np.testing.assert_allclose(r.observable_values, want, atol=bar)
        np.testing.assert_allclose(r.final_state, states[:, -1], atol=bar)


def test_long_first_steps_are_rejected():
    """A first step far too long is halved until the budget holds; both loops take the same decisions."""
    import rpm_b200 as rb
    from rpm_b200 import synthetic

    s = synthetic.make_system(3, (2, 1), (1, 2))
    h = rb.CompiledFullPairHamiltonian(s.dimensions, s.terms(0.7, 0.3), left_axes=s.left_axes, right_axes=s.right_axes)
    m = s.dimension // 4
    psi = np.zeros((4, m), dtype=complex)
    psi[1], psi[2] = 1.0 / np.sqrt(2 * m), -1.0 / np.sqrt(2 * m)
    times = np.array([0.0, 0.05, 300.0])
    out = []
    for device in (True, False):
        prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=8, maximum_dimension=24, state_error_budget=1e-8,
                                            initial_step_us=300.0, maximum_step_us=300.0, minimum_step_us=200.0,
                                            device_steps=device)
        with pytest.raises(RuntimeError, match="below the configured minimum"):
            prop.propagate(psi.reshape(-1), times, rb.SingletPopulationObservable(s.dimensions))
        prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=8, maximum_dimension=24, state_error_budget=1e-8,
                                            initial_step_us=300.0, device_steps=device)
        out.append(prop.propagate(psi.reshape(-1), times[:2] * 20.0, rb.SingletPopulationObservable(s.dimensions)))
    assert (out[0].stats.accepted_steps, out[0].stats.rejected_steps, out[0].stats.matvecs) == \
        (out[1].stats.accepted_steps, out[1].stats.rejected_steps, out[1].stats.matvecs)
    np.testing.assert_allclose(out[0].observable_values, out[1].observable_values, atol=1e-12)


@pytest.mark.parametrize("scale,time", [(1.0, 1e-90), (1.0, 1e-110), (1.0, 1e-150), (1.0, 1e-300), (1e-200, 1.0),
                                        (1e-310, 1.0), (5e-324, 1e10)])
def test_coefficients_of_vanishing_times(scale, time):
    """Arguments down to the smallest numbers: e1 with the first-order entry -i beta_0 t (1e-13 of it; subnormal
    couplings count as zero).  The error's sum of squares underflows below 1e-162, so it is only bounded above."""
    alpha, beta = scale * np.array([0.5, -0.5, 0.25]), scale * np.array([1.0, 0.75, 0.0])
    got, err, _ = _coefficients(alpha, beta, [(3, 1, time), (2, -1, time)])
    first = -1j * beta[0] * time if scale > 1e-300 else 0.0
    for k in range(2):
        assert abs(got[k, 0] - 1.0) <= 1e-15
        assert abs(got[k, 1] - first) <= 1e-13 * abs(first)
    assert 0.0 <= err[0] <= (1.0 + 1e-13) * abs(first) and err[1] == 0.0

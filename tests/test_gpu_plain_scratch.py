"""Scratch and workspace of the plain propagation (GPU)."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(left, right, seed=3):
    """A fresh system and a singlet start state."""
    import rpm_b200 as rb
    from rpm_b200 import synthetic

    s = synthetic.make_system(seed, left, right)
    h = rb.CompiledFullPairHamiltonian(s.dimensions, s.terms(math.pi / 4, 0.3), left_axes=s.left_axes,
                                       right_axes=s.right_axes)
    m = s.dimension // 4
    rng = np.random.default_rng(seed)
    psi = np.zeros((4, m), dtype=complex)
    psi[1] = np.exp(2j * np.pi * rng.uniform(size=m)) / math.sqrt(2 * m)
    psi[2] = -psi[1]
    return s, h, psi.reshape(-1)


def _propagate(s, h, psi, times, device_steps=True, **knobs):
    import rpm_b200 as rb

    prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=8, maximum_dimension=24, state_error_budget=1e-10,
                                        device_steps=device_steps, **knobs)
    return prop.propagate(psi, times, rb.SingletPopulationObservable(s.dimensions))


# the basis build asks the reduction slot for more than the step's own sums from
# about 8,700 components on: below, just above, above, the full size
@pytest.mark.parametrize("left,right", [((2, 3), (1, 3)), ((1, 4), (1, 4)), ((2, 3), (1, 4)), ((2, 5), (1, 6))])
def test_first_propagation_of_a_fresh_system(left, right):
    """The first call, in which scratch grows, gives the bits of the second, in
    which none does, and the host loop's populations (1e-12) and state (1e-11)."""
    s, h, psi = _case(left, right)
    times = np.arange(9) * 0.00125
    first = _propagate(s, h, psi, times)
    again = _propagate(s, h, psi, times)
    np.testing.assert_array_equal(first.observable_values, again.observable_values)
    np.testing.assert_array_equal(first.final_state, again.final_state)
    assert first.stats == again.stats
    host = _propagate(s, h, psi, times, device_steps=False)
    np.testing.assert_allclose(first.observable_values, host.observable_values, atol=1e-12)
    np.testing.assert_allclose(first.final_state, host.final_state, atol=1e-11)


def _behind_a_busy_default_stream(run):
    """``run()`` on a stream of its own while the default stream still works for about 3 ms."""
    import torch

    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    torch.cuda._sleep(5_000_000)
    with torch.cuda.stream(stream):
        out = run()
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("left,right", [((2, 3), (1, 4)), ((2, 5), (1, 6))])
def test_propagation_on_a_stream_of_its_own(left, right):
    """A fresh system propagated on a non-blocking stream, with the default stream
    busy when its scratch is made, and again with more scratch, gives the bits
    that the default stream gives."""
    times = np.arange(41) * 0.00125
    want = _propagate(*_case(left, right), times)
    s, h, psi = _case(left, right)
    few = _behind_a_busy_default_stream(lambda: _propagate(s, h, psi, times[:9]))
    np.testing.assert_array_equal(few.observable_values, _propagate(s, h, psi, times[:9]).observable_values)
    got = _behind_a_busy_default_stream(lambda: _propagate(s, h, psi, times))
    np.testing.assert_array_equal(got.observable_values, want.observable_values)
    np.testing.assert_array_equal(got.final_state, want.final_state)


def test_gradient_on_a_stream_of_its_own():
    """The adjoint's workspace, made on a non-blocking stream while the default
    stream is busy, gives the default stream's gradients (1e-12: its sums are
    FP64 atomics)."""
    import torch

    from rpm_b200 import synthetic
    from rpm_b200.adjoint import AdjointYieldGradient, ParametricRadicalPair

    def gradient():
        s = synthetic.make_system(5, (2, 3), (1, 4))
        model = ParametricRadicalPair(s, pulse_start_us=0.005, pulse_duration_us=0.02)
        psi = torch.from_numpy(np.stack([_case((2, 3), (1, 4), seed)[2] for seed in (3, 4)])).to("cuda")
        r = AdjointYieldGradient(model, precision="c128")(np.array([50.0, 0.7, 0.3, 200.0, 1.0]), psi,
                                                          np.arange(33) * 0.00125, 1.0)
        return r.yields, r.gradients, r.populations

    want = gradient()
    for a, b in zip(_behind_a_busy_default_stream(gradient), want):
        np.testing.assert_allclose(a, b, rtol=1e-12, atol=1e-12 * np.max(np.abs(b)))


def test_a_basis_that_is_not_finite_is_reported():
    """Couplings of 1e160 overflow the norms of the basis: the step control's block
    ends with an error on every call, and the system stays usable."""
    import rpm_b200 as rb
    from rpm_b200 import _lib

    rng = np.random.default_rng(1)
    a = rng.normal(size=(4, 4)) + 1j * rng.normal(size=(4, 4))
    h = rb.CompiledFullPairHamiltonian((2, 2, 2, 2), [rb.LocalTerm((0, 2), 1e160 * (a + a.conj().T)),
                                                      rb.LocalTerm((1, 3), a + a.conj().T)],
                                       left_axes=(0, 2), right_axes=(1, 3))
    psi = rng.normal(size=16) + 1j * rng.normal(size=16)
    prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=6, maximum_dimension=12)
    for _ in range(20):
        with pytest.raises(_lib.RpmError) as e:
            prop.propagate(psi / np.linalg.norm(psi), [0.0, 0.01], rb.SingletPopulationObservable((2, 2, 2, 2)))
        assert e.value.code == _lib.RPM_E_NUMERIC


def test_propagations_leave_little_memory_with_each_system():
    """Four more systems kept alive after their propagation hold well below a basis each (85 MB at 24 vectors)."""
    import torch

    kept, free = [], []
    for seed in range(6):
        s, h, psi = _case((2, 5), (1, 6), seed)
        _propagate(s, h, psi, np.arange(5) * 0.00125)
        kept.append(h)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[5] <= 4 * 24 * 221184 * 16 // 4


def test_propagations_on_several_streams_at_once():
    """Threads with a stream and systems of their own give the bits of one after the other."""
    import threading

    import torch

    times = np.arange(17) * 0.00125
    cases = [_case((2, 3), (1, 4), seed) for seed in range(4)]
    want = [_propagate(*c, times) for c in cases]
    got = [None] * len(cases)

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                got[k] = _propagate(*cases[k], times)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a.observable_values, b.observable_values)
        np.testing.assert_array_equal(a.final_state, b.final_state)

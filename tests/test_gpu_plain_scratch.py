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

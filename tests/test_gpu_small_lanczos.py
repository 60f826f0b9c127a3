"""One-block Lanczos steps of small states against the launch sequence they replace: the same bits (GPU).

The general cube launches are forced through the tuning hook with the tile
sizes they would choose by themselves, so every sum runs in the same order
and populations, error estimates, final states and step counts have to be
equal, not close.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (spin-1, spin-1/2) per radical: 16 to 4,096 components; tiles of fewer than
# 32, of 32 and of more tasks, one and two inner digits, one and two 2,048-component chunks
SHAPES = [((0, 1), (0, 1)), ((1, 1), (0, 2)), ((1, 1), (1, 1)), ((0, 4), (0, 2)), ((2, 1), (1, 2)), ((0, 2), (1, 4)),
          ((2, 2), (1, 3)), ((0, 5), (0, 5)), ((0, 3), (0, 7))]


def _natural(dims_left, dims_right, batch, sms):
    """(ni_l, ni_r, tl) of the general cube launches for a batch."""
    def inner(dims):
        k = 0
        while k < len(dims) and dims[-1 - k] == 2:
            k += 1
        return min(k, 2)

    nl = 2 * int(np.prod(dims_left))
    tl = next((t for t in (16, 8, 4) if -(-nl // t) * batch >= 2 * sms), 2)
    return inner(dims_left), inner(dims_right), tl


@pytest.mark.parametrize("fad,trp", SHAPES)
@pytest.mark.parametrize("count,krylov,caps", [(1, 7, None), (5, 12, (5, 12)), (120, 16, None)])
def test_small_steps_have_the_launches_bits(fad, trp, count, krylov, caps):
    import torch

    import rpm_b200 as rb
    from rpm_b200 import _lib, synthetic
    from rpm_b200.batched import BatchedPropagator

    system = synthetic.make_system(11, fad, trp)
    hams = [rb.CompiledFullPairHamiltonian(system.dimensions, system.terms(th, 0.4), left_axes=system.left_axes,
                                           right_axes=system.right_axes) for th in (0.3, 1.2)]
    if hams[0]._system.fast_hpsi:
        pytest.skip("shape-specialised passes")
    psi = synthetic.random_phase_vectors(system.dimensions, count, 8)
    index = np.arange(count) % 2
    times = np.arange(25 if krylov != 12 else 5) * 0.00125
    dims = system.dimensions
    nleft = len(system.left_axes) - 1
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ni_l, ni_r, tl = _natural(dims[2:2 + nleft], dims[2 + nleft:], count, sms)

    def run():
        bp = BatchedPropagator(hams, krylov_dimension=krylov, state_error_budget=1e-8, krylov_caps=caps,
                               embedded_offset=2)
        return bp.propagate(psi, times, system_index=index, return_final_states=True)

    small = run()
    _lib.call("rpm_set_cube_tuning", ni_l, ni_r, 0, tl)
    try:
        launches = run()
    finally:
        _lib.call("rpm_set_cube_tuning", 0, 0, 0, 0)
    np.testing.assert_array_equal(small.observable_values, launches.observable_values)
    np.testing.assert_array_equal(small.state_error_estimates, launches.state_error_estimates)
    assert torch.equal(small.final_states, launches.final_states)
    assert [s.matvecs for s in small.stats] == [s.matvecs for s in launches.stats]

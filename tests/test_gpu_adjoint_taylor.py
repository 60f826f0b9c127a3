"""Taylor terms of the complex128 adjoint passes in one launch per interval (states that fit in shared memory) and
one launch per term (larger states): forward populations against the plain FP64 propagator (GPU).

Bar: 1e-9 absolute.  The Taylor remainder per interval is below 1e-10 of the state's norm (the engine's tolerance),
its effect on a population twice that, over 20 intervals at most 4e-9 if all added in phase; the plain run's budget
is 1e-12.  Remainders alternate in sign of (-i)^d with the intervals' phases, and the degree is rounded up, so a
quarter of the bound is asked for.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (spin-1, spin-1/2) per radical: 16 to 13,824 dimensions, around 384 threads and the shared-memory limit
SHAPES = [((0, 1), (0, 1)), ((1, 1), (0, 2)), ((2, 1), (1, 2)), ((2, 2), (1, 3)), ((1, 4), (1, 4)), ((2, 3), (1, 4))]


@pytest.mark.parametrize("fad,trp", SHAPES)
@pytest.mark.parametrize("vectors", [1, 3])
def test_forward_populations_match_plain_propagator(fad, trp, vectors):
    import torch

    import rpm_b200 as rb
    from rpm_b200 import synthetic
    from rpm_b200.adjoint import AdjointYieldGradient, ParametricRadicalPair

    system = synthetic.make_system(5, fad, trp)
    model = ParametricRadicalPair(system, pulse_start_us=0.005, pulse_duration_us=0.01)
    times = np.arange(21) * 0.00125
    psi = synthetic.random_phase_vectors(system.dimensions, vectors, 3)
    fwd = AdjointYieldGradient(model).forward([50.0, 0.7, 0.3, 0.0, 1.0], torch.from_numpy(psi).to("cuda"), times, 1.0)
    pops = fwd["populations"].cpu().numpy()
    fwd["workspace"].close()
    h = rb.CompiledFullPairHamiltonian(system.dimensions, system.terms(0.7, 0.3), left_axes=system.left_axes,
                                       right_axes=system.right_axes)
    prop = rb.AdaptiveLanczosPropagator(h, minimum_dimension=8, maximum_dimension=40, state_error_budget=1e-12)
    for b in range(vectors):
        ref = prop.propagate(psi[b], times, rb.SingletPopulationObservable(system.dimensions)).observable_values
        np.testing.assert_allclose(pops[b], ref, rtol=0.0, atol=1e-9)

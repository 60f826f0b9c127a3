"""H psi of a batch against its vectors one at a time, bit for bit: the kernels
that take two vectors per thread (from some hundred blocks on) add in the order
of the one-vector kernel, so that a vector's result does not depend on how many
are beside it (GPU)."""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (spin-1, spin-1/2) per radical; batches below, at and above the lines of either
# precision, three vectors (kept single), odd ones (a last vector alone)
CASES = [((2, 5), (1, 6), (2, 3, 4, 5, 9)), ((2, 4), (1, 5), (4, 5, 6, 7, 17)), ((2, 3), (1, 4), (3, 21, 22, 23, 55)),
         ((2, 2), (1, 3), (84, 85, 171)), ((1, 4), (1, 4), (32, 33))]


@pytest.mark.parametrize("left,right,batches", CASES)
@pytest.mark.parametrize("precision", [128, 64])
@pytest.mark.parametrize("rates", [None, (1.0, 2.0)])
def test_a_vector_does_not_depend_on_its_neighbours(left, right, batches, precision, rates):
    import torch

    import rpm_b200 as rb
    from rpm_b200 import synthetic

    s = synthetic.make_system(7, left, right)
    h = rb.CompiledFullPairHamiltonian(s.dimensions, s.terms(math.pi / 4, 0.3), left_axes=s.left_axes,
                                       right_axes=s.right_axes)
    if rates:
        h.set_recombination_rates(*rates)
    rng = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((max(batches), s.dimension), generator=rng, device="cuda", dtype=torch.complex128)
    x = x.to(torch.complex64) if precision == 64 else x
    want = torch.empty_like(x)
    for k in range(max(batches)):
        h.apply(x[k:k + 1], want[k:k + 1], batch=1, precision=precision)
    for batch in batches:
        out = torch.full_like(x[:batch], 7.0)
        h.apply(x[:batch], out, batch=batch, precision=precision)
        assert torch.equal(torch.view_as_real(out), torch.view_as_real(want[:batch]))

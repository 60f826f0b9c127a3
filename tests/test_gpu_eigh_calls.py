"""Hermitian eigen-solver: calls of several host threads, matrices that are not finite (GPU)."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sizes_solved_by_several_threads_at_once():
    """Threads that solve different sizes (their kernels need 4 to 224 KB of shared
    memory) on streams of their own get the bits of calls one after the other."""
    import torch

    from rpm_b200.factorized import hermitian_eigh

    rng = np.random.default_rng(2)
    inputs = []
    for n in (4, 118, 40, 96):
        a = rng.normal(size=(2, n, n)) + 1j * rng.normal(size=(2, n, n))
        inputs.append(torch.from_numpy(a + a.conj().transpose(0, 2, 1)).to("cuda"))
    want = [hermitian_eigh(a) for a in inputs]
    torch.cuda.synchronize()
    failures = []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(60):
                    lam, vec = hermitian_eigh(inputs[k])
                    if not (torch.equal(lam, want[k][0]) and
                            torch.equal(torch.view_as_real(vec), torch.view_as_real(want[k][1]))):
                        failures.append((k, "result"))
        except Exception as e:  # noqa: BLE001
            failures.append((k, str(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(inputs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failures == []


# in shared memory and one block of eigenvector rows; in global memory and several
@pytest.mark.parametrize("n", [6, 72, 160])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_matrices_that_are_not_finite_are_reported(n, bad):
    """An error, and the solver goes on working."""
    import torch

    from rpm_b200 import _lib
    from rpm_b200.factorized import hermitian_eigh

    rng = np.random.default_rng(n)
    a = rng.normal(size=(3, n, n)) + 1j * rng.normal(size=(3, n, n))
    a = torch.from_numpy(a + a.conj().transpose(0, 2, 1)).to("cuda")
    broken = a.clone()
    broken[1, 2, 1] = broken[1, 1, 2] = bad
    with pytest.raises(_lib.RpmError) as e:
        hermitian_eigh(broken)
    assert e.value.code == _lib.RPM_E_NUMERIC
    lam, _ = hermitian_eigh(a)
    np.testing.assert_allclose(lam.cpu().numpy(), np.linalg.eigvalsh(a.cpu().numpy()), atol=1e-12 * n)

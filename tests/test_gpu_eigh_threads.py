"""Hermitian eigen-solver calls of several host threads (GPU)."""

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

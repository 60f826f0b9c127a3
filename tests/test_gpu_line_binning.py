"""Transition lines on a frequency grid: the single-pair entry point against NumPy,
lines outside the grid (GPU)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(d, seed):
    rng = np.random.default_rng(seed)
    lam = np.sort(rng.uniform(-3, 3, d))
    ops = rng.normal(size=(2, d, d)) + 1j * rng.normal(size=(2, d, d))
    return lam, ops[0], ops[1]


def _bin(lam, p, q, scale, delta, half):
    import torch

    from rpm_b200 import _lib

    grid = torch.zeros(2 * half + 1, dtype=torch.complex128, device="cuda")
    bad = torch.zeros(1, dtype=torch.int32, device="cuda")
    dev = [torch.from_numpy(np.ascontiguousarray(x)).to("cuda") for x in (lam, p, q)]
    _lib.call("rpm_bin_transition_lines", *(_lib.ptr(x) for x in dev), lam.size, scale, delta, half, _lib.ptr(grid),
              _lib.ptr(bad), _lib.stream_handle())
    return grid.cpu().numpy(), int(bad.item())


@pytest.mark.parametrize("d", [1, 2, 17, 72])
def test_binned_lines_match_numpy(d):
    """Bar 1e-12 of the largest possible bin: FP64 sums of at most d^2 lines in any order."""
    lam, p, q = _inputs(d, d)
    delta = 0.07
    half = int(np.ceil((lam[-1] - lam[0]) / delta)) + 3
    got, bad = _bin(lam, p, q, 0.5, delta, half)
    pos = (lam[:, None] - lam[None, :]) / delta + half
    low, w = np.floor(pos).astype(int), 0.5 * p * q.T
    want = np.zeros(2 * half + 1, complex)
    np.add.at(want, low, w * (1.0 - (pos - low)))
    np.add.at(want, low + 1, w * (pos - low))
    assert bad == 0
    np.testing.assert_allclose(got, want, rtol=0.0, atol=1e-12 * np.sum(np.abs(w)))


# just outside at either end, far outside, beyond the range of integers, infinite, NaN
@pytest.mark.parametrize("lam,delta", [((0.0, 10.0), 1.0), ((0.0, 1e9), 1.0), ((0.0, 1e19), 1.0), ((0.0, 1e300), 1e-10),
                                       ((0.0, np.inf), 1.0), ((0.0, np.nan), 1.0)])
def test_lines_outside_the_grid_are_reported(lam, delta):
    import torch

    from rpm_b200 import _lib

    half = 10
    op = np.ones((2, 2), complex)
    grid, bad = _bin(np.array(lam), op, op, 1.0, delta, half)
    assert bad == 1 and np.all(np.isfinite(grid))
    # all nine pairs of both radicals at once
    lam_d = torch.tensor([lam], dtype=torch.float64, device="cuda")
    vec = torch.eye(2, dtype=torch.complex128, device="cuda")[None].contiguous()
    halves = np.array([half], dtype=np.int64)
    need = np.zeros(1, dtype=np.int64)
    _lib.call("rpm_factorized_workspace", 2, 2, 1, halves.ctypes.data, halves.ctypes.data, 1, need.ctypes.data)
    work = torch.empty(int(need[0]), dtype=torch.uint8, device="cuda")
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    times = np.array([1.0])
    _lib.call("rpm_factorized_yields", 2, 2, 1, _lib.ptr(lam_d), _lib.ptr(vec), _lib.ptr(lam_d), _lib.ptr(vec), delta,
              halves.ctypes.data, halves.ctypes.data, times.ctypes.data, 1, _lib.ptr(out), _lib.ptr(flag),
              _lib.ptr(work), _lib.stream_handle())
    assert int(flag.item()) == 1

"""Eigen-solver and lifetime-sum kernels of the factorized yields at the edges of their ranges (GPU)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check_eigh(a, lam, vec):
    """numpy's eigenvalues, residual and orthonormality at the bars of the solver's other test."""
    n = a.shape[-1]
    for b in range(a.shape[0]):
        ref = np.linalg.eigvalsh(a[b])
        scale = np.max(np.abs(ref))
        grow = max(1.0, n / 64)
        assert np.max(np.abs(lam[b] - ref)) <= 1e-12 * scale * grow
        assert np.max(np.abs(a[b] @ vec[b] - vec[b] * lam[b][None, :])) <= 1e-11 * scale * grow
        assert np.max(np.abs(vec[b].conj().T @ vec[b] - np.eye(n))) <= 1e-12 * grow


# 118 / 119: the last matrix held in shared memory; 157 .. 160: eigenvector rows
# of one and of two CTAs; 1024: the cap, 24 rows per CTA; 65 / 66: one more
# rotation than a ring slot holds
@pytest.mark.parametrize("na,nb", [(2, 33), (65, 66), (118, 119), (157, 160), (32, 1024)])
def test_eigh_pair_sizes(na, nb):
    import torch

    from rpm_b200.factorized import _eigh_pair

    rng = np.random.default_rng(na)
    mats = []
    for n in (na, nb):
        a = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))
        a = a + a.conj().transpose(0, 2, 1)
        a[1] = np.diag(np.repeat(rng.standard_normal((n + 1) // 2), 2)[:n])  # already diagonal, twofold values
        mats.append(a)
    # a skew part goes: the solver takes 0.5 (A + A^H)
    skew = [torch.from_numpy(a + np.triu(np.full(a.shape[1:], 0.25), 1) - np.tril(np.full(a.shape[1:], 0.25), -1))
            for a in mats]
    lam_a, vec_a, lam_b, vec_b = (t.cpu().numpy() for t in _eigh_pair(*(s.to("cuda") for s in skew)))
    _check_eigh(mats[0], lam_a, vec_a)
    _check_eigh(mats[1], lam_b, vec_b)


@pytest.mark.parametrize("scale", [1e-120, 1.0, 1e120])
def test_eigh_scales_and_graded_entries(scale):
    """Squares of the entries leave the range of the short rotation formulas; decoupled and graded blocks."""
    import torch

    from rpm_b200.factorized import hermitian_eigh

    rng = np.random.default_rng(8)
    n = 40
    a = rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))
    a = a + a.conj().transpose(0, 2, 1)
    a[1, :20, 20:] = a[1, 20:, :20] = 0.0
    a[1, 20:, 20:] *= 1e-30
    a *= scale
    lam, vec = hermitian_eigh(torch.from_numpy(a).to("cuda"))
    _check_eigh(a / scale, lam.cpu().numpy() / scale, vec.cpu().numpy())


def _reference(lam_a, ops_a, lam_b, ops_b, delta, ha, hb, lifetimes):
    def grid(lam, ops, half, p, q):
        g = np.zeros(2 * half + 1, complex)
        d = lam.size
        pos = (lam[:, None] - lam[None, :]) / delta + half
        low = np.floor(pos).astype(int)
        w = ops[p] * ops[q].T / (d // 2)
        np.add.at(g, low.ravel(), (w * (1 - (pos - low))).ravel())
        np.add.at(g, low.ravel() + 1, (w * (pos - low)).ravel())
        return g

    n = 1 << (2 * (ha + hb)).bit_length()
    total = sum(np.fft.fft(grid(lam_a, ops_a, ha, p, q), n) * np.fft.fft(grid(lam_b, ops_b, hb, p, q), n)
                for p in range(3) for q in range(3))
    conv = np.fft.ifft(total)[:2 * (ha + hb) + 1]
    w = (np.arange(conv.size) - (ha + hb)) * delta
    rows = [0.25 + conv.sum().real]
    rows += [0.25 + (conv / (1 - 1j * w * t)).sum().real for t in lifetimes]
    return rows


# grid half widths per orientation: FFT lengths below, at and above one tile
# (2^11), within one column pass (<= 2^19), with a second one (2^20), mixed
@pytest.mark.parametrize("halves", [[(6, 9)], [(255, 256), (511, 512)], [(700, 400), (9000, 3000), (40, 20)],
                                    [(150000, 130000), (2000, 1000)]])
@pytest.mark.parametrize("da,db", [(2, 34), (18, 16)])
def test_lifetime_sums_match_numpy(halves, da, db):
    """Bar 1e-11: sums of fewer than 2^20 terms of total size ~1, rounding 1e-16 x log2(length) each, all of one sign
    at the worst 2e-9, as random signs 2^10 x 20 x 1e-16 = 2e-12."""
    import torch

    from rpm_b200 import _lib

    rng = np.random.default_rng(da)
    batch, lifetimes = len(halves), np.array([1.0, 0.05, 7.0])
    delta = 0.01
    ha, hb = (np.array([h[k] for h in halves], dtype=np.int64) for k in (0, 1))

    def radical(d, half):
        lam = np.sort(rng.uniform(-0.5, 0.5, (batch, d)), axis=1) * (half[:, None] - 3) * delta
        q, _ = np.linalg.qr(rng.standard_normal((batch, d, d)) + 1j * rng.standard_normal((batch, d, d)))
        return np.ascontiguousarray(lam), np.ascontiguousarray(q)

    spin = [np.array([[0, .5], [.5, 0]]), np.array([[0, -.5j], [.5j, 0]]), np.array([[.5, 0], [0, -.5]])]
    (la, va), (lb, vb) = radical(da, ha), radical(db, hb)
    size = ctypes.c_longlong()
    _lib.call("rpm_factorized_workspace", da, db, batch, ha.ctypes.data, hb.ctypes.data, 3, ctypes.byref(size))
    work = torch.full((size.value,), 255, dtype=torch.uint8, device="cuda")  # NaN where nothing is written
    dev = [torch.from_numpy(x).to("cuda") for x in (la, va, lb, vb)]
    out = torch.empty((batch, 4), dtype=torch.float64, device="cuda")
    bad = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run():
        _lib.call("rpm_factorized_yields", da, db, batch, *(_lib.ptr(x) for x in dev), delta, ha.ctypes.data,
                  hb.ctypes.data, lifetimes.ctypes.data, 3, _lib.ptr(out), _lib.ptr(bad), _lib.ptr(work),
                  _lib.stream_handle())

    run()
    assert int(bad.item()) == 0
    got = out.cpu().numpy()
    for b in range(batch):
        ops = [[v[b].conj().T @ np.kron(s, np.eye(d // 2)) @ v[b] for s in spin] for v, d in ((va, da), (vb, db))]
        want = _reference(la[b], ops[0], lb[b], ops[1], delta, int(ha[b]), int(hb[b]), lifetimes)
        assert np.max(np.abs(got[b] - want)) <= 1e-11
    # a line outside its grid is reported, not written
    dev[0][0, -1] = 2.0 * float(ha[0]) * delta
    run()
    assert int(bad.item()) == 1


def test_orientations_in_several_calls(monkeypatch):
    """The workspace limit splits the orientations into calls with the same results."""
    import rpm_b200 as rb
    from rpm_b200 import factorized, synthetic

    s = synthetic.make_system(3, (1, 2), (1, 1), exchange_J_mT=0.0, dipolar_D_mT=0.0)
    hams = [rb.CompiledFullPairHamiltonian(s.dimensions, s.terms(0.2 * k, 0.1), left_axes=s.left_axes,
                                           right_axes=s.right_axes) for k in range(5)]
    one = factorized.factorized_singlet_yields(hams, [1.0, 0.3])
    monkeypatch.setattr(factorized, "_WORKSPACE_BYTES", 1)
    many = factorized.factorized_singlet_yields(hams, [1.0, 0.3])
    for a, b in zip(one, many):
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-12)

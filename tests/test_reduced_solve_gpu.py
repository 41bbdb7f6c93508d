"""One-launch reduced eigensolve and reduced-matrix update, against NumPy (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pencil(n, seed, spread=1.0):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    y = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    h = (x + x.conj().T) * spread
    s = np.eye(n) + 0.2 / n * (y @ y.conj().T)
    return h, s


def _solve(h, s, roots, stream=None):
    import torch

    from qe_python_b200.eigensolver import ReducedSolve

    n = h.shape[0]
    storage = torch.zeros((n + 3, n + 3), dtype=torch.complex128, device="cuda")
    storage[:n, :n] = torch.from_numpy(h)
    solver = ReducedSolve(stream or torch.cuda.current_stream())
    solver.launch(storage[:n, :n], torch.from_numpy(s).cuda(), roots)
    values, vectors = solver.result()
    assert np.array_equal(solver.host_values(), values.cpu().numpy())
    return values.cpu().numpy(), vectors.cpu().numpy()


@pytest.mark.parametrize("n,roots", [(1, 1), (2, 1), (3, 3), (8, 8), (15, 4), (16, 8), (31, 31),
                                     (32, 1), (32, 32), (33, 5)])
def test_lowest_pairs(cuda_device, n, roots):
    import scipy.linalg
    import torch

    h, s = _pencil(n, n)
    want = scipy.linalg.eigh(h, s, eigvals_only=True)[:roots]
    scale = np.abs(scipy.linalg.eigh(h, s, eigvals_only=True)).max()
    tol = 40 * n * 2.2e-16  # backward error of n eps, condition of S below 3
    for stream in (None, torch.cuda.Stream()):
        e, c = _solve(h, s, roots, stream)
        assert np.max(np.abs(e - want)) <= tol * scale
        assert np.max(np.abs(h @ c - (s @ c) * e)) <= 10 * tol * scale
        assert np.max(np.abs(c.conj().T @ s @ c - np.eye(roots))) <= 10 * tol


def test_degenerate_diagonal_and_scaled(cuda_device):
    import scipy.linalg

    h = np.diag([2.0, -1.0, 2.0, 0.0, -1.0, 2.0]).astype(complex)
    e, c = _solve(h, np.eye(6, dtype=complex), 4)
    assert np.array_equal(e, [-1.0, -1.0, 0.0, 2.0])
    for spread in (1e-9, 1e9, 1e-140, 1e140):  # the last two: the library route
        h, s = _pencil(12, 5, spread)
        e, _ = _solve(h, s, 12)
        want = scipy.linalg.eigh(h, s, eigvals_only=True)
        assert np.max(np.abs(e - want)) <= 1e-13 * np.abs(want).max()


def _status(h, s, roots):
    """What the one-launch solver reports of the pencil."""
    import torch

    from qe_python_b200 import _lib

    n = h.shape[0]
    hd, sd = (torch.from_numpy(np.ascontiguousarray(m)).cuda() for m in (h, s))
    values = torch.zeros(roots + 1, dtype=torch.float64, device="cuda")
    vectors = torch.zeros((roots, n), dtype=torch.complex128, device="cuda")
    _lib.check("qeb_small_generalized_eigh", _lib.load().qeb_small_generalized_eigh(
        n, roots, hd.data_ptr(), n, sd.data_ptr(), n, values.data_ptr(), vectors.data_ptr(), n,
        int(torch.cuda.current_stream().cuda_stream)))
    return values.cpu().numpy()[roots]


def _with_smallest(smallest):
    """A pencil whose overlap has one eigenvalue ``smallest`` and nine ones."""
    h, s = _pencil(10, 3)
    u = np.linalg.qr(s)[0]
    weights = np.array([smallest] + [1.0] * 9)
    s = (u * weights) @ u.conj().T
    return h, 0.5 * (s + s.conj().T), u


def test_indefinite_overlap_takes_the_canonical_route(cuda_device):
    h, s, u = _with_smallest(-1e-6)
    assert 1 <= _status(h, s, 4) <= 10  # the Cholesky factorisation fails
    e, c = _solve(h, s, 4)
    # the pencil on the nine directions that are left, where S is the identity
    kept = u[:, 1:]
    want = np.linalg.eigvalsh(kept.conj().T @ h @ kept)[:4]
    scale = np.linalg.norm(h, 2)
    tol = 40 * 10 * 2.2e-16
    assert np.max(np.abs(e - want)) <= tol * scale
    assert np.max(np.abs(c.conj().T @ s @ c - np.eye(4))) <= 10 * tol
    assert np.max(np.abs(u[:, :1].conj().T @ c)) <= 10 * tol  # nothing of the dropped one
    residual = kept.conj().T @ (h @ c - (s @ c) * e)
    assert np.max(np.abs(residual)) <= 10 * tol * scale


def test_nearly_singular_overlap_stays_on_its_route(cuda_device):
    import scipy.linalg

    h, s, u = _with_smallest(1e-8)
    assert _status(h, s, 4) == 0.0
    e, c = _solve(h, s, 4)
    # backward error n eps of L^-1 H L^-H, whose norm is that of H over 1e-8
    tol = 40 * 10 * 2.2e-16 * np.linalg.norm(h, 2) * 1e8
    assert np.max(np.abs(e - scipy.linalg.eigh(h, s, eigvals_only=True)[:4])) <= tol
    assert np.max(np.abs(c.conj().T @ s @ c - np.eye(4))) <= 40 * 10 * 2.2e-16 * 1e8


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("first,active", [(0, 1), (0, 17), (5, 6), (24, 61)])
def test_update_reduced(cuda_device, dtype, first, active):
    import torch

    from qe_python_b200 import kernels as K
    from qe_python_b200.device import to_device_f

    rng = np.random.default_rng(active)
    m = active - first
    rows = [(rng.standard_normal((m, active)) + 1j * rng.standard_normal((m, active))).astype(dtype)
            for _ in range(2)]
    dev = [to_device_f(r, getattr(torch, dtype), torch.device("cuda")) for r in rows]
    lam = rng.standard_normal(first)
    for shift in (None, lam):
        mats = [torch.zeros((active + 2, active + 2), dtype=torch.complex128, device="cuda")
                for _ in range(2)]
        K.update_reduced(mats[0], mats[1], first, dev[0], dev[1],
                         None if shift is None else torch.from_numpy(shift).cuda())
        wide = [r.astype(np.complex128) for r in rows]
        if shift is not None:
            wide[0][:, :first] += wide[1][:, :first] * shift
        for got, r in zip(mats, wide):
            want = np.zeros((active + 2, active + 2), dtype=complex)
            want[first:active, :active] = r
            want[:first, first:active] = r[:, :first].conj().T
            block = r[:, first:]
            want[first:active, first:active] = 0.5 * (block + block.conj().T)
            assert np.max(np.abs(got.cpu().numpy() - want)) <= 4e-16 * np.max(np.abs(r))

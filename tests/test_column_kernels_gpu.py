"""Column kernels at the edges of their runs, blocks and clusters, against
NumPy (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("rows,cols", [
    (1, 1), (2, 3), (1023, 2), (1024, 5), (1025, 1), (8191, 3),
    (8192, 2),      # two blocks per column
    (40001, 7),     # a cluster per column, odd rows
    (70000, 200),
])
def test_edges(cuda_device, dtype, rows, cols):
    import torch

    from qe_python_b200 import kernels as K

    rng = np.random.default_rng(rows + cols)
    u = np.finfo(np.float32 if dtype == "complex64" else np.float64).eps / 2
    tdtype = getattr(torch, dtype)

    def matrix(odd, offset):
        """Column-major device matrix (an odd leading dimension, or a first
        value half a 16-byte word into its buffer) and its values."""
        ld = rows + (1 - rows % 2 + 2 if odd else rows % 2)
        storage = torch.full((cols * ld + offset,), float("nan"), dtype=tdtype, device="cuda")
        view = storage[offset:].reshape(cols, ld).T[:rows]
        values = (rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols))).astype(dtype)
        view.copy_(torch.from_numpy(values))
        return view, values.astype(np.complex128)

    diag = rng.uniform(-2.0, 20.0, rows)
    energies = rng.uniform(-1.0, 1.0, cols)
    diag_dev, e_dev = torch.from_numpy(diag).cuda(), torch.from_numpy(energies).cuda()
    for odd, offset in ((False, 0), (True, 0), (False, 1)):
        a, av = matrix(odd, offset)
        b, bv = matrix(odd, offset)
        # FP64 sums of `rows` terms (of exact squares for complex64)
        tol = 4 * rows * 1.2e-16
        norms = np.sum(np.abs(av) ** 2, axis=0)
        assert np.all(np.abs(K.column_squared_norms(a).cpu().numpy() - norms) <= tol * norms)
        got = K.column_diagonal_expectations(a, diag_dev).cpu().numpy()
        assert np.all(np.abs(got - diag @ np.abs(av) ** 2) <= tol * (np.abs(diag) @ np.abs(av) ** 2))
        got = K.column_inner_products(a, b).cpu().numpy()
        assert np.all(np.abs(got - np.sum(av.conj() * bv, axis=0))
                      <= 2 * tol * np.sum(np.abs(av) * np.abs(bv), axis=0))
        x = 2.0 * (diag[:, None] - energies[None, :])
        want = av * (2.0 / (0.5 * (1.0 + x + np.sqrt(1.0 + (x - 1.0) ** 2))))
        out, _ = matrix(odd, offset)
        K.precondition(a, e_dev, diag_dev, out)
        # one rounding of each part to the vectors' type on top of FP64 arithmetic
        assert np.all(np.abs(out.cpu().numpy() - want) <= (1.5 * u + 1e-14) * np.abs(want))
        order = rng.permutation(cols)
        K.normalize_columns(a, torch.from_numpy(norms).cuda(), torch.from_numpy(order).cuda(), out)
        want = av[:, order] / np.sqrt(norms[order])
        assert np.all(np.abs(out.cpu().numpy() - want) <= (1.5 * u + 1e-15) * np.abs(want))
        K.subtract_band_energies(out, a, e_dev)
        want = want - energies[None, :] * av
        assert np.all(np.abs(out.cpu().numpy() - want)
                      <= 6 * u * (np.abs(want) + np.abs(energies[None, :] * av)) + 3 * u)


def test_precondition_extremes(cuda_device):
    """Far-off energies, infinities and NaN behave as the formula does."""
    import torch

    from qe_python_b200 import kernels as K

    diag = np.array([0.0, 1e6, -1e6, 1e160, -1e3, np.inf, np.nan, 1e-30])
    for dtype, u in ((torch.complex64, 6e-8), (torch.complex128, 1.2e-16)):
        ones = torch.ones((1, 8), dtype=dtype, device="cuda").T
        got = K.precondition(ones, torch.zeros(1, dtype=torch.float64, device="cuda"),
                             torch.from_numpy(diag).cuda()).cpu().numpy()[:, 0]
        with np.errstate(all="ignore"):
            x = 2.0 * diag
            want = 2.0 / (0.5 * (1.0 + x + np.sqrt(1.0 + (x - 1.0) ** 2)))
        finite = np.isfinite(want)
        assert np.array_equal(np.isfinite(got.real), finite)
        # x = -2e6: 1 + x + sqrt(...) cancels to 2 with an absolute error of 2e6 u64
        assert np.all(np.abs(got.real - want)[finite] <= (2 * u + 2e-9) * np.abs(want[finite]) + 1e-45)

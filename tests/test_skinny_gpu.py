"""Narrow products (one output side of at most 16 columns) at the edges of
their blocks and widths, against NumPy (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("conj,m,n,k", [
    (True, 1, 1, 1),
    (True, 8, 8, 579),       # warps of a block split K
    (True, 33, 3, 64),
    (True, 5, 200, 63),      # the narrow side is A's (conjugate transpose written)
    (True, 16, 17, 129),
    (True, 864, 5, 4097),
    (True, 300, 16, 30001),  # K split over blocks, odd tail
    (True, 1000, 11, 9000),
    (False, 1, 1, 1),
    (False, 63, 2, 7),       # one row short of a block, fewer K values than warps
    (False, 64, 9, 8),
    (False, 65, 16, 9),
    (False, 1001, 5, 864),
])
def test_edges(cuda_device, dtype, conj, m, n, k):
    import torch

    from qe_python_b200 import kernels as K

    rng = np.random.default_rng(m + 7 * n + 13 * k)
    real = np.float32 if dtype == "complex64" else np.float64
    tdtype = getattr(torch, dtype)

    def matrix(rows, cols, ld, offset=0):
        """A column-major device matrix at the given leading dimension, whose
        first value lies ``offset`` values into its buffer, and its values."""
        storage = torch.full((cols * ld + offset,), float("nan"), dtype=tdtype, device="cuda")
        view = storage[offset:].reshape(cols, ld).T[:rows]
        values = (rng.standard_normal((rows, cols)) + 1j * rng.standard_normal((rows, cols)))
        values = values.astype(dtype)
        view.copy_(torch.from_numpy(values))
        return view, values.astype(np.complex128)

    code = K.OP_C if conj else K.OP_N
    alpha, beta = 0.7 - 0.2j, -0.3 + 1.1j
    ar, ac = (k, m) if conj else (m, k)
    u = np.finfo(real).eps / 2
    # aligned columns, odd leading dimensions, and a start half a 16-byte word in
    for odd, offset in ((False, 0), (True, 0), (False, 1)):
        pad = (lambda r: r + 1 - r % 2 + 2) if odd else (lambda r: r + r % 2)
        a, av = matrix(ar, ac, pad(ar), offset)
        b, bv = matrix(k, n, pad(k), offset)
        c, cv = matrix(m, n, pad(m), offset)
        op = av.conj().T if conj else av
        # rounding of a k-term complex dot product: (2k + 4) u sum |a||b| on
        # each part, sqrt(2) on the modulus
        scale = np.sqrt(2) * (2 * k + 4) * u * (np.abs(op) @ np.abs(bv))
        got = K.gemm(code, a, b, tensor=False).cpu().numpy()
        assert np.all(np.abs(got - op @ bv) <= scale)
        K.gemm(code, a, b, c, alpha=alpha, beta=beta, tensor=False)
        want = alpha * (op @ bv) + beta * cv
        assert np.all(np.abs(c.cpu().numpy() - want) <= scale + 8 * u * (np.abs(want) + np.abs(cv)))

"""FP64 tensor-pipe GEMM at the edges of its tiles, against NumPy (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("m,n,k", [
    (17, 17, 1),       # smallest sides past the skinny kernels, one K value
    (32, 48, 7),       # one 32 x 48 tile, a partial K step
    (33, 49, 8),       # one past those edges, one whole K step
    (48, 64, 33),      # one past four K steps
    (49, 65, 31),
    (64, 96, 64),
    (65, 33, 129),
    (579, 40, 130),    # many row tiles
    (140, 37, 11636),  # K split over blocks (A^H B)
    (97, 200, 4099),   # a last slice shorter than the others
])
def test_tile_edges(cuda_device, conj, m, n, k):
    import torch

    from qe_python_b200 import kernels as K
    from qe_python_b200.device import to_device_f

    rng = np.random.default_rng(m * 1000 + n + k)

    def values(*shape):
        return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)

    a, b, c0 = values(*((k, m) if conj else (m, k))), values(k, n), values(m, n)
    alpha, beta = 0.7 - 0.2j, -0.3 + 1.1j
    op = a.conj().T if conj else a
    device = torch.device("cuda")
    a_dev = to_device_f(a, torch.complex128, device)
    b_dev = to_device_f(b, torch.complex128, device)
    code = K.OP_C if conj else K.OP_N
    # rounding of a k-term complex dot product: (2k + 4) u sum |a||b| on each
    # part, sqrt(2) on the modulus, doubled for the reference's own
    scale = 2 * np.sqrt(2) * (2 * k + 4) * 1.2e-16 * (np.abs(op) @ np.abs(b))
    got = K.gemm(code, a_dev, b_dev).cpu().numpy()
    assert np.all(np.abs(got - op @ b) <= scale)
    c_dev = to_device_f(c0, torch.complex128, device)
    got = K.gemm(code, a_dev, b_dev, c_dev, alpha=alpha, beta=beta).cpu().numpy()
    assert np.all(np.abs(got - (alpha * (op @ b) + beta * c0)) <= scale + 4e-15 * np.abs(c0))
    # an odd leading dimension: a view inside a larger matrix
    wide = to_device_f(np.vstack([a, values(1, a.shape[1])]), torch.complex128, device)
    view = torch.empty(wide.shape[1], a.shape[0] | 1, dtype=torch.complex128, device=device)
    odd = view.T[:a.shape[0]]
    odd.copy_(wide[:a.shape[0]])
    got = K.gemm(code, odd, b_dev).cpu().numpy()
    assert np.all(np.abs(got - op @ b) <= scale)

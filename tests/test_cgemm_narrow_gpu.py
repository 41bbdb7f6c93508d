"""Split-TF32 GEMM on both sides of its 64- and 128-column tiles, against NumPy (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conj,m,n,k", [
    (True, 1, 17, 16), (True, 256, 64, 4001), (True, 130, 63, 23847), (True, 96, 65, 2000),
    (True, 300, 33, 513),
    (False, 127, 17, 1), (False, 1000, 64, 130), (False, 23847, 61, 256),  # a split last wave
    (False, 257, 65, 33), (False, 129, 128, 31),
])
def test_tile_widths(cuda_device, conj, m, n, k):
    import torch

    from qe_python_b200 import kernels as K
    from qe_python_b200.device import to_device_f

    rng = np.random.default_rng(m + n + k)

    def values(*shape):
        return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)

    a, b, c = values(*((k, m) if conj else (m, k))), values(k, n), values(m, n)
    dev = [to_device_f(x, torch.complex64, torch.device("cuda")) for x in (a, b, c)]
    op = (a.conj().T if conj else a).astype(np.complex128)
    want = op @ b
    # 22-bit split products and the FP32 accumulation of 2 k terms
    tol = 2e-6 * np.sqrt(2 * k) * np.sqrt(2) * 2
    code = K.OP_C if conj else K.OP_N
    got = K.cgemm_tf32x3(code, dev[0], dev[1]).cpu().numpy()
    assert np.max(np.abs(got - want)) <= tol
    K.cgemm_tf32x3(code, dev[0], dev[1], dev[2], alpha=0.5 - 1j, beta=0.25 + 0.5j)
    want = (0.5 - 1j) * want + (0.25 + 0.5j) * c
    assert np.max(np.abs(dev[2].cpu().numpy() - want)) <= 2 * tol
    assert K.tf32_error() == 0

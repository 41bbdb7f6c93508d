"""FP64 products A^H B: chains of additions no longer than K over the number of
slices that fill the GPU twice, and the rounding that goes with them."""

from __future__ import annotations

import numpy as np
import pytest

SHAPES = [(512, 40, 11019), (864, 100, 20000), (256, 61, 23847), (97, 97, 5000), (512, 256, 11019),
          (17, 17, 700), (300, 200, 300)]


def _slices(m, n, k):
    """Two waves of 64 x 64 tiles on 148 SMs, slices of at least 256 values."""
    tiles = -(-m // 64) * -(-n // 64)
    return max(1, min(-(-2 * 148 // tiles), k // 256, 64))


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_slices(m, n, k):
    from qe_python_b200 import _lib
    from qe_python_b200 import kernels as K

    nbytes = int(_lib.load().qeb_zgemm_scratch_bytes(K.OP_C, m, n, k, _lib.QEB_F64))
    assert max(1, nbytes // (16 * m * n)) >= _slices(m, n, k)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", SHAPES[:4])
def test_rounding(cuda_device, m, n, k):
    """The error against extended precision is that of FP64 chains of that
    length, the two products of each part added one after the other (2 depth
    additions: one addition of their sum would round half as often)."""
    import torch

    from qe_python_b200 import kernels as K
    from qe_python_b200.device import to_device_f

    rng = np.random.default_rng(k)
    a, b = (rng.standard_normal((k, c)) + 1j * rng.standard_normal((k, c)) for c in (m, n))
    got = K.gemm(K.OP_C, *(to_device_f(v, torch.complex128, torch.device("cuda")) for v in (a, b)))
    i, j = np.arange(0, m, max(1, m // 32)), np.arange(0, n, max(1, n // 24))
    got = got.cpu().numpy()[np.ix_(i, j)]
    a, b = a[:, i].conj(), b[:, j]
    ar, ai, br, bi = (v.astype(np.longdouble) for v in (a.real, a.imag, b.real, b.imag))
    exact = (ar.T @ br - ai.T @ bi, ar.T @ bi + ai.T @ br)
    depth = -(-k // _slices(m, n, k))
    chained = np.zeros((len(i), len(j)), dtype=complex)
    for start in range(0, k, depth):
        part = np.zeros_like(chained)
        for row in range(start, min(k, start + depth)):
            x, y = a[row][:, None], b[row][None, :]
            part.real += x.real * y.real
            part.imag += x.real * y.imag
            part.real -= x.imag * y.imag
            part.imag += x.imag * y.real
        chained += part

    def error(v):
        return np.sqrt(float(((v.real - exact[0]) ** 2 + (v.imag - exact[1]) ** 2).sum()))

    # both are sums of about a thousand independent roundings' walks: within a
    # fifth of each other
    assert error(got) <= 1.2 * error(chained)

"""Rounding of the line transforms against extended precision, beside the
generic Stockham kernels' (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from qe_python_b200.basis import LocalPotentialWorkspace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bands,precision", [(36, 8, "f64"), (36, 8, "f32"), (144, 1, "f32")])
def test_factors_round_no_more_than_the_generic_kernels(cuda_device, monkeypatch, n, bands, precision):
    """Two equal factors: one layer of twiddles between DFTs without any.  (With
    4 x 9 and 16 x 9, whose DFT9 and DFT16 have twiddles of their own, the
    errors were 1.04 to 1.06 of the generic kernels'.)"""
    import scipy.fft
    import torch

    from qe_python_b200.device import to_device_f

    axis = np.arange(-int(0.205 * n), int(0.205 * n) + 1)
    m = np.stack([a.ravel() for a in np.meshgrid(axis, axis, axis, indexing="ij")], axis=1)
    m = m[np.sum(m ** 2, axis=1) <= axis[-1] ** 2].astype(np.int32)
    rng = np.random.default_rng(n)
    psi = (rng.standard_normal((len(m), bands)) + 1j * rng.standard_normal((len(m), bands)))
    psi = psi.astype(np.complex64).astype(np.complex128)  # exact in either precision
    v = rng.uniform(-1, 1, (n, n, n)).astype(np.float32).astype(float)
    where = tuple(m[:, a] % n for a in range(3))
    exact = np.empty(psi.shape, dtype=np.clongdouble)
    for b in range(bands):
        grid = np.zeros((n, n, n), dtype=np.clongdouble)
        grid[where] = psi[:, b]
        grid = scipy.fft.ifftn(grid, norm="forward", workers=4) * v.astype(np.longdouble)
        exact[:, b] = scipy.fft.fftn(grid, norm="forward", workers=4)[where]
    errors = []
    for generic in ("0", "1"):
        monkeypatch.setenv("QEB_FORCE_GENERIC", generic)
        ws = LocalPotentialWorkspace(m, (n, n, n), precision=precision)
        assert ws.line_passes == (generic == "0")
        got = ws.apply(torch.from_numpy(v).cuda(),
                       to_device_f(psi, ws.complex_dtype, torch.device("cuda"))).cpu().numpy()
        errors.append(float(np.sqrt(np.sum(np.abs(got - exact) ** 2))))
    assert errors[0] <= errors[1]

"""Densities of several streams added to one grid (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from qe_python_b200.basis import LocalPotentialWorkspace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("bands", [3, 24])  # atomics straight into the density; with a grid
def test_two_streams_into_one_density(cuda_device, precision, bands):
    import torch

    shape, calls = (64, 60, 64), 40
    rng = np.random.default_rng(bands)
    axes = np.arange(-9, 10)
    m = np.stack([a.ravel() for a in np.meshgrid(axes, axes, axes, indexing="ij")], axis=1)
    m = m[np.sum(m ** 2, axis=1) <= 81].astype(np.int32)
    psi = torch.from_numpy(rng.standard_normal((bands, len(m)))
                           + 1j * rng.standard_normal((bands, len(m)))).cuda().T
    weights = torch.from_numpy(rng.uniform(0.5, 2.0, bands)).cuda()
    spaces = [LocalPotentialWorkspace(m, shape, precision=precision) for _ in range(2)]
    psi = psi.to(spaces[0].complex_dtype).T.contiguous().T
    once = torch.zeros(shape, dtype=torch.float64, device="cuda")
    spaces[0].accumulate_density(once, psi, weights)
    rho = torch.zeros_like(once)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in spaces]
    for _ in range(calls):
        for space, stream in zip(spaces, streams):
            with torch.cuda.stream(stream):
                space.accumulate_density(rho, psi, weights)
    torch.cuda.synchronize()
    # sums of positive FP64 terms, in any order: (2 calls bands) u relative
    want = 2 * calls * once
    assert float(((rho - want).abs() / want.clamp_min(1e-300)).max()) <= 2 * calls * bands * 1.2e-16

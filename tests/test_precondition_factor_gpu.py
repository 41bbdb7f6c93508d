"""The preconditioner's FP64 factor behind complex64 vectors (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_factor_is_rounded_in_fp64(cuda_device):
    """The products' roundings to 24 bits against a NumPy FP64 factor.  Two
    factors r apart (relative) round a product to different values for a share
    of about r / 2^-24 of the components: a factor good to 1e-13 shows in some 7
    of the 4 million here (six were seen of approximate reciprocals with Newton
    steps), the last bits in which two FP64 evaluations differ (3e-16 on these
    x, about 5e-9 per component) in none."""
    import torch

    from qe_python_b200 import kernels as K

    rng = np.random.default_rng(4)
    rows, cols = 40000, 50
    r = (rng.standard_normal((cols, rows)) + 1j * rng.standard_normal((cols, rows))).astype(np.complex64)
    diag, energies = rng.uniform(0.0, 30.0, rows), rng.uniform(-1.0, 0.0, cols)
    got = K.precondition(torch.from_numpy(r).cuda().T, torch.from_numpy(energies).cuda(),
                         torch.from_numpy(diag).cuda()).cpu().numpy().T
    x = 2.0 * (diag[None, :] - energies[:, None])
    s = 2.0 / (0.5 * (1.0 + x + np.sqrt(1.0 + (x - 1.0) * (x - 1.0))))
    differing = sum(int(np.count_nonzero((s * part.astype(np.float64)).astype(np.float32) != out))
                    for part, out in ((r.real, got.real), (r.imag, got.imag)))
    assert differing <= 3


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_cancelled_denominator_gives_infinity(cuda_device, dtype):
    """x below -2^53: 1 + x + sqrt(1 + (x - 1)^2) is zero and the quotient infinite."""
    import torch

    from qe_python_b200 import kernels as K

    diag = torch.tensor([-1e20, -1e100, 2.0], dtype=torch.float64, device="cuda")
    ones = torch.full((1, 3), 1 - 1j, dtype=getattr(torch, dtype), device="cuda").T
    got = K.precondition(ones, torch.zeros(1, dtype=torch.float64, device="cuda"), diag)
    got = got.cpu().numpy()[:, 0]
    assert np.all(got.real[:2] == np.inf) and np.all(got.imag[:2] == -np.inf)
    assert np.isfinite(got[2])

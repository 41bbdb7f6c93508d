"""Column reductions over clusters of blocks: the form of their barrier, and
clusters of every size against NumPy."""

from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

SOURCE = Path(__file__).resolve().parents[1] / "qe_python_b200/csrc/davidson_kernels.cu"


def test_cluster_barrier_needs_no_converged_warp():
    """Thread 0 of a block reaches the barriers from branches of its own (it
    stores and adds the partial sums), and barrier.cluster's .aligned form is
    undefined in a warp that has not reconverged."""
    barriers = re.findall(r"barrier\.cluster\.(?:arrive|wait)[.\w]*", SOURCE.read_text())
    assert len(barriers) == 2 and not any("aligned" in b for b in barriers)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("rows,cols", [(8191, 5), (8192, 3), (16384, 3), (32769, 148), (65536, 1)])
def test_cluster_sizes(cuda_device, dtype, rows, cols):
    """One, two, four, four and eight blocks per column, many times over."""
    import torch

    from qe_python_b200 import kernels as K

    rng = np.random.default_rng(rows)
    a, b = ((rng.standard_normal((cols, rows)) + 1j * rng.standard_normal((cols, rows))).astype(dtype)
            for _ in range(2))
    ta, tb = torch.from_numpy(a).cuda().T, torch.from_numpy(b).cuda().T
    a, b = a.astype(np.complex128), b.astype(np.complex128)
    norms = np.sum(np.abs(a) ** 2, axis=1)
    inner = np.sum(a.conj() * b, axis=1)
    # FP64 sums of `rows` terms, in another order than NumPy's
    tol = 4 * rows * 1.2e-16
    first = None
    for _ in range(20):
        got = K.column_squared_norms(ta).cpu().numpy(), K.column_inner_products(ta, tb).cpu().numpy()
        assert np.all(np.abs(got[0] - norms) <= tol * norms)
        assert np.all(np.abs(got[1] - inner) <= 2 * tol * np.sum(np.abs(a) * np.abs(b), axis=1))
        if first is not None:  # a fixed order of the sums
            assert np.array_equal(got[0], first[0]) and np.array_equal(got[1], first[1])
        first = got

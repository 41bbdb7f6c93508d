"""A refused plan is an error of its own call only (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from qe_python_b200 import _lib
from qe_python_b200.basis import LocalPotentialWorkspace

pytestmark = pytest.mark.gpu


def test_refused_plan_leaves_no_pending_error(cuda_device):
    """An FP64 plane past shared memory is refused on the host; the next
    library and torch calls of the thread do not report it."""
    import torch

    axis = np.arange(-90, 91)
    miller = np.stack([m.ravel() for m in np.meshgrid(axis, axis, [0], indexing="ij")], axis=1)
    with pytest.raises(_lib.NativeError):
        LocalPotentialWorkspace(miller.astype(np.int32), (192, 192, 16), precision="f64")
    x = torch.rand(4, dtype=torch.float64, device="cuda").sum()
    assert 0.0 <= float(x) <= 4.0
    small = LocalPotentialWorkspace(np.zeros((1, 3), dtype=np.int32), (16, 16, 16))
    assert small.plane_waves == 1

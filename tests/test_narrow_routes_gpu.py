"""Narrow products on both sides of the rules that choose their kernels, against
NumPy (GPU)."""

from __future__ import annotations

import pytest

from tests import test_skinny_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("conj,m,n,k", [
    # one thread per row from so many thousand rows on, by width and K
    (False, 28000, 1, 10),
    (False, 65001, 2, 9),
    (False, 27999, 2, 10),
    (False, 16000, 16, 10),
    (False, 15999, 16, 10),
    (False, 50001, 4, 65),     # a K step past the staged 64
    (False, 65537, 8, 151),
    (False, 20001, 11, 49),
    (False, 36255, 7, 128),    # one row short of a block of 256
    (False, 34001, 13, 151),   # the last wave full enough (complex128), and not
    (False, 38001, 10, 65),
    # 9 to 16 columns: few steps for many wide columns, or about a hundred long ones
    (True, 512, 9, 1536),
    (True, 511, 9, 1536),
    (True, 605, 16, 33),
    (True, 10, 600, 300),      # the narrow side is A's
    (True, 64, 13, 16384),
    (True, 192, 16, 16511),    # K split over blocks, odd tail
    (True, 13, 97, 20001),
    (True, 97, 12, 20001),
])
def test_routes(cuda_device, dtype, conj, m, n, k):
    test_skinny_gpu.test_edges(cuda_device, dtype, conj, m, n, k)

"""Narrow products on both sides of the rules that choose their kernels, against
NumPy (GPU)."""

from __future__ import annotations

import pytest

from tests import test_skinny_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("conj,m,n,k", [
    # one thread per row from so many thousand rows on, by width and K
    (False, 46000, 1, 10),
    (False, 60001, 2, 9),
    (False, 45999, 2, 10),
    (False, 12000, 16, 10),
    (False, 11999, 16, 10),
    (False, 52001, 4, 65),     # a K step past the staged 64
    (False, 65537, 8, 151),
    (False, 32001, 11, 47),    # groups of eight, of four and a rest
    (False, 36255, 7, 128),    # one row short of a block
    (False, 24001, 12, 3),
    (False, 16001, 12, 300),   # 11 and 12 complex128 columns in the kernel of 16
    # slices in whole waves for 9 to 16 columns against at most 192
    (True, 192, 9, 3071),
    (True, 193, 9, 12288),
    (True, 192, 16, 12289),
    (True, 13, 97, 20001),     # the narrow side is A's
    (True, 97, 12, 20001),
    (True, 1, 16, 6145),
])
def test_routes(cuda_device, dtype, conj, m, n, k):
    test_skinny_gpu.test_edges(cuda_device, dtype, conj, m, n, k)

"""Line-transform passes over the lengths, shapes and k-point batches at which
their kernels change, against the oracle (GPU)."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import native_fft as oracle
from qe_python_b200.basis import LocalPotentialWorkspace, grid_slots

pytestmark = pytest.mark.gpu

LENGTHS = [16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96,
           100, 108, 120, 128, 135, 144, 150, 160, 180, 192]


def _basis(shape, fraction, seed, shift=0):
    """Miller indices of an ellipsoid that spans ``fraction`` of the grid, in
    random order (``shift``: moved along x)."""
    reach = [max(1, int(fraction * n / 2)) for n in shape]
    axes = [np.arange(-r, r + 1) for r in reach]
    m = np.stack([a.ravel() for a in np.meshgrid(*axes, indexing="ij")], axis=1)
    m = m[np.sum((m / (np.array(reach) + 1e-9)) ** 2, axis=1) <= 1.0]
    m[:, 0] += shift
    return np.random.default_rng(seed).permutation(m).astype(np.int32)


def _check(shape, miller, precision, bands=2, seed=0, density=True):
    import torch

    rng = np.random.default_rng(seed)
    npw = len(miller)
    psi = np.asfortranarray(rng.standard_normal((npw, bands)) + 1j * rng.standard_normal((npw, bands)))
    if precision == "f32":
        psi = np.asfortranarray(psi.astype(np.complex64).astype(np.complex128))
    v = np.ascontiguousarray(rng.uniform(-1, 1, shape))
    kinetic = rng.uniform(0, 4, npw)
    linear, *_ = grid_slots(miller, shape)
    size = int(np.prod(shape))
    grid = np.zeros((bands, size), dtype=np.complex128)
    plan = oracle.NativeFFTWPlan(grid, shape, bands, 1, size)
    want = np.zeros_like(psi)
    oracle.apply_serial(grid, psi, v, linear, plan, size, size, want, 0, kinetic)
    ws = LocalPotentialWorkspace(miller, shape, precision=precision)
    got = ws.apply(torch.from_numpy(v).cuda(), torch.from_numpy(psi).cuda(),
                   diagonal=torch.from_numpy(kinetic).cuda()).cpu().numpy()
    # rounding of a transform: a few u per butterfly level and axis, both ways
    tol = (1.2e-7 if precision == "f32" else 2.3e-16) * 12 * np.log2(size)
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want)) * 4
    if density:
        full = np.zeros((bands, size), dtype=np.complex128)
        full[:, linear] = psi.T
        w = rng.uniform(0.5, 2.0, bands)
        psi_r = np.fft.ifftn(full.reshape(bands, *shape), axes=(1, 2, 3), norm="forward")
        rho = np.einsum("b,bxyz->xyz", w, np.abs(psi_r) ** 2)
        acc = torch.ones(shape, dtype=torch.float64, device="cuda")
        ws.accumulate_density(acc, torch.from_numpy(psi).cuda(), torch.from_numpy(w).cuda())
        assert np.max(np.abs(acc.cpu().numpy() - 1.0 - rho)) <= tol * np.max(rho) * 4
    return ws


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n", LENGTHS)
def test_every_length(cuda_device, n, precision):
    """A square plane of every listed length (static kernel; its sphere as wide
    as ecutrho = 4 ecutwfc makes it), z lines of another one."""
    nz = LENGTHS[(LENGTHS.index(n) * 7 + 3) % len(LENGTHS)] if n <= 96 else 20
    # (FP64 planes of wider spheres are refused from 160 points on)
    fraction = 0.47 if n < 160 else (0.28 if n < 192 else 0.24)
    ws = _check((n, n, nz), _basis((n, n, nz), fraction, n), precision, density=n <= 96)
    # the static kernel's rows of 192 FP64 points exceed shared memory: run-time kernel
    assert ws.line_passes and (ws.pruned_plane > 0) == ((n, precision) != (192, "f64"))


@pytest.mark.parametrize("n,nz,fraction,precision,lines,kept", [
    (192, 20, 0.24, "f64", True, 0),   # the occupied blocks' rows fit where the kept ones do not
    (192, 20, 0.28, "f64", False, 0),  # neither fit: generic kernels, no blocks reported
    (192, 20, 0.28, "f32", True, 4),
    (64, 125, 0.47, "f64", False, 0),  # z without a split
])
def test_plane_layout(cuda_device, n, nz, fraction, precision, lines, kept):
    ws = _check((n, n, nz), _basis((n, n, nz), fraction, 3), precision, density=False)
    assert (ws.line_passes, ws.pruned_plane) == (lines, kept)


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape,fraction,shift", [
    ((45, 50, 90), 0.47, 0),     # unequal plane: run-time kernel
    ((50, 45, 24), 0.47, 1),
    ((16, 192, 18), 0.47, 0),
    ((48, 48, 20), 0.95, 0),     # a sphere past the static kernel's kept rows
    ((36, 36, 24), 0.45, 9),     # sticks away from x = 0
    ((24, 24, 125), 0.47, 0),    # z length without two small factors: generic kernels
    ((125, 24, 24), 0.47, 0),
    ((8, 10, 12), 0.6, 0),
])
def test_other_shapes(cuda_device, shape, fraction, shift, precision):
    _check(shape, _basis(shape, fraction, 5, shift), precision, bands=3)


def test_sparse_sticks(cuda_device):
    """Few scattered sticks (33: one more than a z block), one entry each."""
    rng = np.random.default_rng(3)
    cells = rng.choice(32 * 32, 33, replace=False)
    miller = np.stack([cells // 32, cells % 32, rng.integers(0, 20, 33)], axis=1).astype(np.int32)
    for precision in ("f32", "f64"):
        _check((32, 32, 20), miller, precision)


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_batch_of_unequal_spheres(cuda_device, precision):
    """k points of one grid whose spheres keep different numbers of blocks (two
    static plane kernels and the run-time one): the bits of each alone."""
    import torch

    from qe_python_b200.basis import apply_local_multi
    from qe_python_b200.device import empty_f, to_device_f

    shape = (90, 90, 36)
    millers = [_basis(shape, f, 7) for f in (0.30, 0.36, 0.47, 0.36, 0.7)]
    rng = np.random.default_rng(9)
    v = torch.from_numpy(rng.uniform(-1, 1, shape)).cuda()
    ws = [LocalPotentialWorkspace(m, shape, precision=precision) for m in millers]
    assert [w.pruned_plane for w in ws] == [2, 2, 3, 2, 0]
    blocks = [to_device_f(rng.standard_normal((len(m), nb)) + 1j * rng.standard_normal((len(m), nb)),
                          ws[0].complex_dtype, torch.device("cuda"))
              for m, nb in zip(millers, (3, 1, 4, 0, 2))]
    targets = [empty_f(b.shape[0], b.shape[1], b.dtype, b.device) for b in blocks]
    apply_local_multi(ws, ws[0].native_potential(v), blocks, [None] * 5, targets)
    for w, block, target in zip(ws, blocks, targets):
        if block.shape[1]:
            assert torch.equal(target, w.apply(v, block))

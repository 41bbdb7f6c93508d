"""The scratch that a captured H|psi> graph records stays the graph's: a density
of as many bands leaves the stick buffer alone, and a larger apply on the same
workspace replaces the buffer without taking it from the graph."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest


def test_density_leaves_the_stick_buffer(monkeypatch):
    """Host side of accumulate_density on CPU buffers, the library faked."""
    import torch

    from qe_python_b200 import basis

    calls = []
    lib = SimpleNamespace(
        qeb_local_scratch_bytes=lambda plan, nb: 1024 * nb,
        qeb_density_scratch_bytes=lambda plan, nb: 1024 * nb + 4096,
        qeb_density_grid_bytes=lambda plan, nb: 4096,
        qeb_accumulate_density=lambda *a: calls.append(a) or 0,
        qeb_accumulate_density_grid=lambda *a: calls.append(a) or 0,
    )
    monkeypatch.setattr(basis, "_lib", SimpleNamespace(load=lambda: lib, check=lambda *a: None))
    monkeypatch.setattr(basis, "stream_handle", lambda: 0)
    monkeypatch.setattr(basis, "to_device_f", lambda v, dtype, device: v)
    ws = object.__new__(basis.LocalPotentialWorkspace)
    ws._plan = None
    ws.shape, ws.device = (4, 4, 4), torch.device("cpu")
    ws.complex_dtype, ws.serial_fft_batch_size = torch.complex128, None
    ws.scratch_pool = basis.FFTScratchPool()
    sticks, nbytes = ws._scratch(6)
    ws.accumulate_density(torch.zeros(4, 4, 4, dtype=torch.float64),
                          torch.zeros(6, 5, dtype=torch.complex128).T, torch.ones(6).double())
    assert len(calls) == 1 and calls[0][1] == sticks.data_ptr() and calls[0][2] == nbytes
    assert ws._scratch(6)[0] is sticks


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_replay_after_density_and_larger_apply(cuda_device, precision):
    import torch

    from qe_python_b200.basis import LocalPotentialWorkspace, make_bases
    from qe_python_b200.device import to_device_f
    from qe_python_b200.diagonalization import HpsiGraph, PlaneWaveHamiltonian
    from qe_python_b200.workloads import hpsi_microbench

    work = hpsi_microbench(nbands=48)
    basis = make_bases(work.reciprocal, np.zeros(3), 30.0)[0]
    ws = LocalPotentialWorkspace(basis, work.shape, precision=precision)
    ham = PlaneWaveHamiltonian(basis, None, ((work.beta, work.coupling),), local_workspace=ws,
                               real_potential=torch.from_numpy(work.potential).cuda(),
                               potential_average=0.0)
    psi = to_device_f(work.psi, ham.dtype, ham.device)
    block = psi[:, :32]  # 32 bands of 64^3 points: the density takes its grid
    graph = HpsiGraph(ham, 32)
    sticks = graph._sticks
    assert sticks is ws._scratch(32)[0]
    want = ham.apply(block).clone()
    assert torch.equal(graph(block), want)

    rho = torch.zeros(ws.shape, dtype=torch.float64, device="cuda")
    ws.accumulate_density(rho, block, torch.ones(32, dtype=torch.float64, device="cuda"))
    assert ws._scratch(32)[0] is sticks
    ham.apply(psi)  # 48 bands: the pool's buffer moves, the graph keeps the old one
    assert ws._scratch(48)[0].data_ptr() != sticks.data_ptr() and graph._sticks is sticks
    others = [torch.full((sticks.numel() // n,), 7, dtype=torch.uint8, device="cuda")
              for n in (1, 1, 2, 2, 4)]
    assert torch.equal(graph(block), want)
    assert all(bool((t == 7).all()) for t in others)

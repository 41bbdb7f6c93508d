"""The one-launch eigensolver is asked for no more columns than it takes."""

from __future__ import annotations

from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("limit,n,route", [(32, 32, "small"), (32, 33, "library"),
                                           (8, 8, "small"), (8, 9, "library")])
def test_route_follows_the_kernel_limit(monkeypatch, limit, n, route):
    import torch

    from qe_python_b200 import eigensolver

    lib = SimpleNamespace(qeb_small_eigh_max=lambda: limit)
    monkeypatch.setattr(eigensolver, "_lib", SimpleNamespace(load=lambda: lib))
    solver = eigensolver.ReducedSolve(None)
    taken = []
    monkeypatch.setattr(solver, "_launch_small", lambda *a: taken.append("small"))
    monkeypatch.setattr(solver, "_launch_library", lambda *a: taken.append("library"))
    matrix = SimpleNamespace(shape=(n, n), dtype=torch.complex128, is_cuda=True,
                             stride=lambda axis: (n, 1)[axis])
    solver.launch(matrix, matrix, 4)
    assert taken == [route]

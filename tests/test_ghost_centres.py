"""Dirichlet data at the ghost centres of a grid whose coordinates change in place,
and of one made in inference mode."""

from __future__ import annotations

import torch

import pyshocks_gb300 as gb
from pyshocks_gb300 import scalar
from pyshocks_gb300.burgers import c_boundary


def _values(bc, grid):
    return list(c_boundary(bc, grid, (0.0, 0.0, 0.0)).dirichlet)[:6]


def _expected(grid):
    g, n = grid.nghosts, grid.ncells
    return [float(grid.x[g - 1 - k]) for k in range(3)] + [float(grid.x[g + n + k]) for k in range(3)]


def test_centres_follow_the_grid():
    bc = scalar.make_dirichlet_boundary(lambda t, x: x)
    grid = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=8, nghosts=3, device="cpu")
    assert _values(bc, grid) == _expected(grid)
    assert _values(bc, grid) == _expected(grid)
    before = _expected(grid)
    grid.x.add_(0.25)
    assert _expected(grid) != before
    assert _values(bc, grid) == _expected(grid)


def test_centres_of_an_inference_grid():
    bc = scalar.make_dirichlet_boundary(lambda t, x: 2.0 * x.requires_grad_() if torch.is_grad_enabled() else x)
    with torch.inference_mode():
        grid = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=8, nghosts=3, device="cpu")
        assert _values(bc, grid) == _expected(grid)
    assert _values(bc, grid) == [2.0 * v for v in _expected(grid)]
    plain = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=8, nghosts=3, device="cpu")
    with torch.inference_mode():
        assert _values(bc, plain) == _expected(plain)
    assert _values(bc, plain) == [2.0 * v for v in _expected(plain)]

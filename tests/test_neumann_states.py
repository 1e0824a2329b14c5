"""``apply_boundary`` with Neumann sides on states that are not a grid's own
(other length, type or rank): the results and refusals of the index form, from
its own formula ``u[ito] = u[ifrom] + side (x[ifrom] - x[ito]) g(t)``."""

from __future__ import annotations

import pytest
import torch

import pyshocks_gb300 as gb
from pyshocks_gb300 import apply_boundary, scalar


def _indexed(sides, grid, gn, u):
    u = u.clone()
    g, n = grid.nghosts, u.shape[0]
    for side in sides:
        ifrom = torch.arange(*grid.gi_[side].indices(n))
        ito = torch.arange(g - 1, -1, -1) if side == -1 else torch.arange(n - 1, n - g - 1, -1)
        u[ito] = u[ifrom] + side * (grid.x[ifrom] - grid.x[ito]) * gn
    return u


STATES = {
    "own": torch.arange(10.0, dtype=torch.float64),
    "float32": torch.arange(10.0),
    "integer": torch.arange(10),
    "two columns": torch.arange(20.0, dtype=torch.float64).reshape(10, 2),
    "three columns": torch.arange(30.0, dtype=torch.float64).reshape(10, 3),
    "longer": torch.arange(12.0, dtype=torch.float64),
    "shorter": torch.arange(8.0, dtype=torch.float64),
}


@pytest.mark.parametrize("state", list(STATES))
@pytest.mark.parametrize("gn", [0.0, 0.5])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("sides", [(-1,), (1,), (-1, 1)])
def test_states_of_any_shape_and_type(sides, dtype, gn, state):
    grid = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=6, nghosts=2, device="cpu", dtype=dtype)
    bc = (scalar.make_neumann_boundary(lambda t: gn) if len(sides) == 2
          else scalar.NeumannBoundary(side=sides[0], g=lambda t: gn))
    u = STATES[state]
    try:
        ref = _indexed(sides, grid, gn, u)
    except (RuntimeError, IndexError) as exc:
        with pytest.raises(type(exc)):
            apply_boundary(bc, grid, 0.0, u)
        return
    out = apply_boundary(bc, grid, 0.0, u)
    assert out.dtype == ref.dtype and torch.equal(out, ref)

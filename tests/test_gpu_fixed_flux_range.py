"""Inputs at the edges of what the float pairs of ``csrc/fixed_flux.cuh`` hold:
smoothness parameters whose products leave float's range."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R

pytestmark = pytest.mark.gpu


def _scheme(flux, eps):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers

    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=eps)
    return burgers.make_scheme_from_name(flux, rec=rec)


@pytest.mark.parametrize("flux", ["rusanov", "lf"])
@pytest.mark.parametrize(("eps", "amp"), [(1e-40, 1e-16), (1e-38, 1e-16), (1e-36, 1e-14), (1e-30, 1e-12), (1e-24, 1e-10),
                                          (1e-6, 1e-3), (1e24, 1e10), (1e30, 1e12)])
def test_steps_for_any_smoothness_parameter(eps, amp, flux):
    """Three steps of states of size *amp* (eps small against their differences'
    squares) against the oracle: 1e-13 of the largest value, as for the other
    fixed-flux steps (about 900 roundings). (Smaller states at eps = 1e-40 are out of
    reach of the FP64 formula too: its products of eight smoothness sums fall below
    the smallest normal double.)"""
    from pyshocks_gb300.batched import BatchedSolver

    sizes = [17, 40, 61, 100, 127]
    nsteps = 3
    u0, refs = [], []
    for n in sizes:
        og = R.make_uniform_cell_grid(-amp, amp, n, 3)
        x = (np.arange(n) + 0.5) / n
        u = amp * (0.3 + np.sin(2 * np.pi * x) + 0.1 * np.cos(6 * np.pi * x + 0.3))
        ug = np.zeros(n + 6)
        ug[3:-3] = u
        ref, _ = R.evolve(R.SchemeSpec(flux_kind=flux, eps=eps), og, ug, theta=0.9, maxit=nsteps)
        u0.append(u)
        refs.append(ref[3:-3])
    for tile in (0, 64):
        solver = BatchedSolver(_scheme(flux, eps), sizes, [2.0 * amp / n for n in sizes], theta=0.9, tile=tile)
        solver.reset(torch.tensor(np.concatenate(u0)))
        solver.step(nsteps)
        assert solver.status() == 0
        for b, n in enumerate(sizes):
            err = np.max(np.abs(solver.instance(b).cpu().numpy() - refs[b])) / np.max(np.abs(u0[b]))
            assert err < 1.0e-13, (n, tile, err)

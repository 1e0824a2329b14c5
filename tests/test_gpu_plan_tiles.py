"""Which tiles a plan takes does not depend on the kernel that steps it: the FP64
formula's layout (seven windows of the tile and its halo in one SM) is the limit also
where the integer fluxes need less."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(flux, alpha, tile, ctas):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers
    from pyshocks_gb300.batched import BatchedSolver

    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6)
    n = 20000
    s = BatchedSolver(burgers.make_scheme_from_name(flux, rec=rec, alpha=alpha), [n], 2.0 / n, tile=tile,
                      ctas_per_sm=ctas)
    s.reset(0.5 + 0.3 * torch.sin(0.01 * torch.arange(n, dtype=torch.float64)))
    return s


@pytest.mark.parametrize("flux", ["rusanov", "lf"])
@pytest.mark.parametrize("alpha", [1.0, 0.9])  # integer fluxes, FP64 formula
def test_longest_tile(flux, alpha):
    s = _solver(flux, alpha, 4096, 0)
    s.step(1)
    assert s.status() == 0
    for tile in (4200, 8192):
        with pytest.raises(Exception):
            _solver(flux, alpha, tile, 0)
        if alpha == 1.0:  # (with named CTAs the step refuses)
            s = _solver(flux, alpha, tile, 1)
            with pytest.raises(Exception):
                s.step(1)

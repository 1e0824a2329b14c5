"""The autotuner's candidates for the integer-flux plans, and that the plan's own
choice is among them."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from pyshocks_gb300 import autotune


def _scheme(eps=1.0e-6, alpha=1.0, flux="rusanov"):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers

    return burgers.make_scheme_from_name(flux, rec=gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=eps),
                                         alpha=alpha)


def test_which_schemes_run_on_the_integer_fluxes():
    assert autotune.integer_flux(_scheme(), 0.01)
    assert autotune.integer_flux(_scheme(flux="lf"), 0.01)
    assert not autotune.integer_flux(_scheme(eps=1.0e-40), 0.01)
    assert not autotune.integer_flux(_scheme(alpha=0.9), 0.01)


@pytest.mark.parametrize("adjoint", [False, True])
def test_candidates_of_integer_flux_plans(adjoint):
    cands = autotune.candidates(torch.float64, 16384, False, adjoint, True, True)
    assert cands[0] == (0, 0)
    assert len(set(cands)) == len(cands)
    for tile, c in cands:
        per = autotune._smem_bytes(tile, torch.float64, False, True, True)
        assert max(c, 1) * per <= autotune.SMEM_PER_SM
    # 946 cells: 27 KB a CTA, eight of them
    assert adjoint or (946, 8) in cands
    assert (0, 0) in autotune.candidates(torch.float32, 300, weno5=True)


@pytest.mark.gpu
@pytest.mark.parametrize("max_steps", [0, 6])
def test_short_instances_are_timed_with_the_plans_own_choice(tmp_path, monkeypatch, max_steps):
    from pyshocks_gb300.batched import BatchedSolver

    monkeypatch.setenv("PYSHOCKS_GB300_CACHE", str(tmp_path / "tune.json"))
    autotune._MEMO.clear()
    sizes = np.arange(100, 340, 10)
    scheme = _scheme()
    s = BatchedSolver(scheme, sizes, 2.0 / sizes, tile="auto", max_steps=max_steps)
    res = autotune.tune(scheme, sizes, 2.0 / sizes, adjoint=max_steps > 0)
    own = [ms for tile, c, ms in res.table if (tile, c) == (0, 0)]
    assert len(own) == 1 and res.ms_per_step <= own[0]
    assert (s.tile, s.ctas_per_sm) == (res.tile, res.ctas_per_sm)
    u0 = torch.sin(0.05 * torch.arange(int(sizes.sum()), dtype=torch.float64))
    d = BatchedSolver(scheme, sizes, 2.0 / sizes, max_steps=max_steps)
    for x in (s, d):
        x.reset(u0)
        x.step(4)
    assert torch.equal(s.u, d.u)

"""Short single-instance calls at the lengths where one CTA hands over to a launch
per piece (``kBlockDtCells`` in ``csrc/forward.cu``, ``kGhBlockCells`` in ``csrc/ghosted.cu``)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8191, 8192, 8193, 20000])
def test_predicted_timestep(n):
    """theta (cfl / max|u|) with the maximum at either end: exact."""
    from pyshocks_gb300 import _lib as L

    s = L.ShkScheme(flux=L.SHK_FLUX_RUSANOV, rec=L.SHK_REC_WENOJS53, eps=1.0e-6, nu=1.0, speed=1.0)
    dt = torch.empty((), dtype=torch.float64, device="cuda")
    for at in (0, n - 1):
        u = torch.full((n + 6,), 0.25, dtype=torch.float64, device="cuda")
        u[3 + at] = -1.7
        u[:3] = 9.0
        u[n + 3 :] = -9.0
        assert L.lib().shk_predict_timestep_f64(s, u.data_ptr(), n, 3, 0.125, 0.5, dt.data_ptr(), L.stream_handle()) == 0
        assert float(dt) == 0.5 * (0.125 / 1.7)


@pytest.mark.parametrize("extra", [0, 1])
@pytest.mark.parametrize(("fk", "limit"), [("lf", 2560), ("rusanov", 1536), ("rusanov", 2048)])
def test_ghosted_step_and_transpose(fk, limit, extra):
    """The constant reconstruction's lines (step and transpose), at the bars of the
    other ghosted tests."""
    from test_gpu_block_paths import test_ghosted_step_and_transpose as check

    check("constant", fk, 1, limit, extra)


@pytest.mark.parametrize("theta", [0.5, 1, torch.tensor([0.25, 0.5], dtype=torch.float64), torch.tensor(0.5)])
def test_time_step_factor_of_any_kind(theta):
    """The driver's ``theta * predict_timestep``: a number, or a tensor that
    broadcasts and keeps its gradient."""
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers, scalar, timestepping
    from pyshocks_gb300.schemes import predict_timestep

    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6)
    grid = gb.make_uniform_cell_grid(a=-1.0, b=1.0, n=64, nghosts=3)
    bc = scalar.PeriodicBoundary()
    scheme = gb.bind(burgers.Rusanov(rec=rec), grid, bc)
    u = torch.sin(grid.x)
    if torch.is_tensor(theta):
        theta = theta.cuda().requires_grad_()
    dt = timestepping.TimestepPredictor(scheme, grid, bc, theta)(0.0, u)
    ref = theta * predict_timestep(scheme, grid, bc, 0.0, u)
    assert dt.shape == ref.shape and torch.equal(dt.detach(), ref.detach())
    assert dt.requires_grad == ref.requires_grad

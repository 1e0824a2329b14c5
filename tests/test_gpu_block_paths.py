"""The one-CTA forms of the short single-instance calls at the sizes where they
hand over to a launch per piece: the ghosted step and its transpose
(``csrc/ghosted.cu``: 512 cells with ghosts for WENO-JS5, 3072 for the constant
reconstruction) and the CFL step (32768 cells)."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R
from oracle import torch_ref as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize(("rec", "fk", "g", "limit"), [("constant", "lf", 1, 3072), ("wenojs53", "lf", 3, 512),
                                                       ("wenojs53", "rusanov", 3, 512)])
def test_ghosted_step_and_transpose(rec, fk, g, limit, extra):
    """Same bars as the smaller ghosted tests: 1e-12 of the largest value for
    the step, 1e-11 for the transpose."""
    from test_gpu_ghosted import _c_args, _ws

    from pyshocks_gb300 import _lib as L

    n = limit + extra - 2 * g
    grid = R.make_uniform_cell_grid(-1.0, 1.0, n, g)
    x = np.asarray(grid.x)
    u = 0.4 + 0.7 * np.sin(np.pi * x) + 0.2 * np.cos(4 * np.pi * x)
    dt = 0.4 * grid.dx_min / np.max(np.abs(u))
    tb = {"left": "periodic", "right": "periodic", "dirichlet": np.zeros((3, 2, 3)), "neumann": np.zeros((3, 2))}
    s, b = _c_args(L, rec, fk, 1.0, tb, g, grid.dx_min)
    ws = _ws(L, n, g)
    ud = torch.tensor(u, device="cuda")
    p = np.random.default_rng(3).standard_normal(u.size)
    pd = torch.tensor(p, device="cuda")
    out = torch.empty_like(ud)
    st = L.lib().shk_ssprk33_step_ghosted_f64(s, ctypes.byref(b), ud.data_ptr(), out.data_ptr(), n, g, grid.dx_min,
                                              dt, ws.data_ptr(), ws.numel(), L.stream_handle())
    assert st == 0, L.errstr(st)
    spec = R.SchemeSpec(flux_kind=fk, rec=rec, eps=1.0e-6)
    ref = R.ssprk33(lambda t, v: R.apply_operator(spec, grid, v, t, None), dt, 0.0, u)
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1.0e-12 * np.max(np.abs(ref))
    st = L.lib().shk_ssprk33_vjp_ghosted_f64(s, ctypes.byref(b), ud.data_ptr(), pd.data_ptr(), out.data_ptr(), n, g,
                                             grid.dx_min, dt, ws.data_ptr(), ws.numel(), L.stream_handle())
    assert st == 0, L.errstr(st)
    ref = T.ghosted_step_vjp(torch.tensor(u), torch.tensor(p), dt, grid.dx_min, g, tb, torch.tensor(x), rec=rec,
                             flux_kind=fk, eps=1.0e-6, nu=1.0).numpy()
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1.0e-11 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1025, 32768, 32769])
def test_predicted_timestep(n):
    """cfl / max|u| with the maximum at either end: exact."""
    from pyshocks_gb300 import _lib as L

    s = L.ShkScheme(flux=L.SHK_FLUX_RUSANOV, rec=L.SHK_REC_WENOJS53, eps=1.0e-6, nu=1.0, speed=1.0)
    dt = torch.empty((), dtype=torch.float64, device="cuda")
    for at in (0, n - 1):
        u = torch.full((n + 6,), 0.25, dtype=torch.float64, device="cuda")
        u[3 + at] = -1.7
        u[:3] = 9.0
        u[n + 3:] = -9.0
        st = L.lib().shk_predict_timestep_f64(s, u.data_ptr(), n, 3, 0.125, 0.5, dt.data_ptr(), L.stream_handle())
        assert st == 0
        assert float(dt) == 0.5 * (0.125 / 1.7)


@pytest.mark.parametrize("ctas", [1, 0])
@pytest.mark.parametrize(("dtype", "flux"), [("float32", "burgers"), ("float32", "lwr"), ("float64", "lwr")])
def test_many_items_per_cta_report_every_maximum(dtype, flux, ctas):
    """A CTA's tiles report their maximum and completion with its next item (or
    after its last): with 64-cell tiles a CTA takes up to about forty, of instances
    that end at every point of its list, and states and times must equal, bit for
    bit, those of one CTA per tile."""
    from test_gpu_adjoint import _scheme

    from pyshocks_gb300.batched import BatchedSolver

    sizes = [n for n in (20011, 7, 333, 64, 65, 4097, 15, 1999) for _ in range(12)]
    rng = np.random.default_rng(61)
    u0 = torch.tensor(np.concatenate([0.5 + 0.3 * np.sin(2 * np.pi * (np.arange(n) / n + rng.uniform()))
                                      * rng.uniform(0.2, 1.0) for n in sizes]))
    out = []
    for tile, c in ((64, ctas), (2048, 0)):
        s = BatchedSolver(_scheme(*(("lwr",) if flux == "lwr" else ())), sizes, [2.0 / n for n in sizes], tile=tile,
                          ctas_per_sm=c, dtype=getattr(torch, dtype))
        s.reset(u0)
        s.step(5)
        assert s.status() == 0
        out.append((s.u.clone(), s.time()))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])

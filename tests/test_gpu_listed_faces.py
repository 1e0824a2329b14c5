"""Faces and cells that the integer / float-pair forms leave to FP64 (``csrc/stencil.cuh``
``fx_listed_faces``, ``fx_listed_tile``, ``csrc/adjoint.cu`` ``weno53_listed_vjp``): states of noise, of runs of
it, and random ones, at the window lengths where the list, the chunks of 60 faces and
their threshold change."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R
from oracle import torch_ref as T

pytestmark = pytest.mark.gpu

SIZES = [5, 31, 46, 47, 75, 76, 77, 78, 106, 107, 165, 166, 167, 168, 226, 400, 1000]
KINDS = ["noise", "runs", "random", "zeros"]


def _state(kind, n, rng):
    x = (np.arange(n) + 0.5) / n
    u = 0.3 + np.sin(2 * np.pi * x) + 0.1 * np.cos(6 * np.pi * x)
    if kind == "noise":
        return u + 0.005 * rng.standard_normal(n)
    if kind == "random":
        return rng.uniform(-1.0, 1.0, n)
    if kind == "zeros":  # random stretches between exact zeros
        return np.where((np.arange(n) // 29) % 2 == 0, rng.uniform(-1.0, 1.0, n), 0.0)
    mask = np.zeros(n, dtype=bool)  # runs of 1 to 70 noisy cells
    i = 0
    while i < n:
        run = int(rng.integers(1, 71))
        mask[i : i + run] = True
        i += run + int(rng.integers(1, 60))
    return u + np.where(mask, 0.05 * rng.standard_normal(n), 0.0)


def _scheme(flux):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers

    return burgers.make_scheme_from_name(flux, rec=gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6))


@pytest.mark.parametrize("flux", ["rusanov", "lf"])
@pytest.mark.parametrize("kind", KINDS)
def test_steps_match_oracle_and_do_not_depend_on_the_tile(kind, flux):
    """Three steps: 1e-13 of the largest value (about 900 roundings) from the
    oracle; bit for bit the same in every tile, resident or launched, however the
    faces were shared out."""
    from pyshocks_gb300.batched import BatchedSolver

    nsteps = 3
    rng = np.random.default_rng(17)
    u0 = [_state(kind, n, rng) for n in SIZES]
    out = []
    for tile in (0, 16, 60, 90, 180, 226, 466, 1024):
        s = BatchedSolver(_scheme(flux), SIZES, [2.0 / n for n in SIZES], theta=0.9, tile=tile)
        s.reset(torch.tensor(np.concatenate(u0)))
        s.step(nsteps)
        assert s.status() == 0
        out.append((s.u.clone(), s))
    for u, _ in out[1:]:
        assert torch.equal(u, out[0][0])
    for b, n in enumerate(SIZES):
        og = R.make_uniform_cell_grid(-1.0, 1.0, n, 3)
        ug = np.zeros(n + 6)
        ug[3:-3] = u0[b]
        ref, _ = R.evolve(R.SchemeSpec(flux_kind=flux), og, ug, theta=0.9, maxit=nsteps)
        err = np.max(np.abs(out[0][1].instance(b).cpu().numpy() - ref[3:-3])) / np.max(np.abs(u0[b]))
        assert err < 1.0e-13, (n, err)


@pytest.mark.parametrize("kind", KINDS)
def test_gradient_does_not_depend_on_the_tile(kind):
    """Checkpointed gradients through stored stages, bit for bit, and against
    autograd: 1e-11 of the largest entry per step (as the transposed step), four
    steps."""
    from pyshocks_gb300.adjoint import CheckpointedSolve
    from pyshocks_gb300.batched import BatchedSolver

    nsteps = 4
    sizes = [31, 77, 166, 400, 1000]
    rng = np.random.default_rng(23)
    u0 = torch.tensor(np.concatenate([_state(kind, n, rng) for n in sizes]))
    p = torch.tensor(rng.standard_normal(sum(sizes))).cuda()
    out = []
    for tile in (0, 64, 216, 448):
        s = BatchedSolver(_scheme("rusanov"), sizes, [2.0 / n for n in sizes], theta=0.5, tile=tile, max_steps=nsteps)
        c = CheckpointedSolve(s, nsteps)
        c.forward(u0.cuda())
        out.append(c.backward(p).clone())
        dts = s.dt_history()
    for g in out[1:]:
        assert torch.equal(g, out[0])
    o = 0
    for b, n in enumerate(sizes):
        states = [u0[o : o + n]]
        for k in range(nsteps - 1):
            states.append(T.ssprk33(states[-1][None], float(dts[k][b]), 2.0 / n)[0])
        q = p[o : o + n].cpu()
        for k in reversed(range(nsteps)):
            q = T.step_vjp(states[k][None], q[None], float(dts[k][b]), 2.0 / n)[0]
        err = float((out[0][o : o + n].cpu() - q).abs().max() / q.abs().max())
        assert err < nsteps * 1.0e-11, (n, err)
        o += n


@pytest.mark.parametrize("n", [31, 95, 96, 97, 127, 128, 129, 130, 470])
@pytest.mark.parametrize("kind", ["noise", "random"])
def test_single_step_and_transpose_on_coarse_grids(kind, n):
    """The single-instance step and its transpose at the lengths where the FP64
    formula hands over (96, 128 cells): 1e-13 and 1e-11 of the largest value."""
    from pyshocks_gb300 import _lib as L

    rng = np.random.default_rng(n)
    u = torch.tensor(_state(kind, n, rng))
    p = torch.tensor(rng.standard_normal(n))
    dx = 2.0 / n
    dt = 0.4 * dx / float(u.abs().max())
    cs = _scheme("rusanov").c_scheme(dx)
    ud, pd = torch.cat([u[-3:], u, u[:3]]).cuda(), torch.cat([p[-3:], p, p[:3]]).cuda()
    out = torch.empty_like(ud)
    lib = L.lib()
    assert lib.shk_ssprk33_step_f64(cs, ud.data_ptr(), out.data_ptr(), n, 3, dx, dt, L.stream_handle()) == 0
    ref = T.ssprk33(u[None], dt, dx)[0]
    assert float((out.cpu()[3:-3] - ref).abs().max()) <= 1.0e-13 * float(u.abs().max())
    assert lib.shk_ssprk33_vjp_f64(cs, ud.data_ptr(), pd.data_ptr(), out.data_ptr(), n, 3, dx, dt, L.stream_handle()) == 0
    ref = T.step_vjp(u[None], p[None], dt, dx)[0]
    assert float((out.cpu()[3:-3] - ref).abs().max()) <= 1.0e-11 * float(ref.abs().max())


def test_lax_friedrichs_where_the_state_is_small():
    """Random cells of size 1e-10 far from cells of size 1: their fluxes carry the
    instance's speed and are exact to (speed x their own size), so two steps keep
    1e-13 of 1e-10 (about 900 roundings) away from the large cells' reach."""
    from pyshocks_gb300.batched import BatchedSolver

    rng = np.random.default_rng(31)
    sizes, nsteps = [400, 1201], 2
    u0 = []
    for n in sizes:
        x = (np.arange(n) + 0.5) / n
        u0.append(np.where(x < 0.5, 0.4 + np.sin(2 * np.pi * x), 1.0e-10 * rng.uniform(-1.0, 1.0, n)))
    for tile in (0, 64):
        s = BatchedSolver(_scheme("lf"), sizes, [2.0 / n for n in sizes], theta=0.9, tile=tile)
        s.reset(torch.tensor(np.concatenate(u0)))
        s.step(nsteps)
        assert s.status() == 0
        for b, n in enumerate(sizes):
            og = R.make_uniform_cell_grid(-1.0, 1.0, n, 3)
            ug = np.zeros(n + 6)
            ug[3:-3] = u0[b]
            ref, _ = R.evolve(R.SchemeSpec(flux_kind="lf"), og, ug, theta=0.9, maxit=nsteps)
            far = slice(n // 2 + 40, n - 40)
            err = np.max(np.abs(s.instance(b).cpu().numpy()[far] - ref[3:-3][far]))
            assert err < 1.0e-23, (n, tile, err)

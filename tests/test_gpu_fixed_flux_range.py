"""Inputs at the edges of what the float pairs of ``csrc/fixed_flux.cuh`` hold:
smoothness parameters whose products leave float's range, cotangents of compact
support, and cotangents whose magnitudes cross the range of a warp's scale."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R
from oracle import torch_ref as T

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


def _vjp(u, p, dt, dx):
    from pyshocks_gb300 import _lib as L

    n = u.numel()
    ud = torch.cat([u[-3:], u, u[:3]]).cuda()
    pd = torch.cat([p[-3:], p, p[:3]]).cuda()
    out = torch.empty_like(ud)
    st = L.lib().shk_ssprk33_vjp_f64(_scheme("rusanov", 1e-6).c_scheme(dx), ud.data_ptr(), pd.data_ptr(),
                                     out.data_ptr(), n, 3, dx, dt, L.stream_handle())
    assert st == 0, L.errstr(st)
    return out.cpu()[3:-3]


def _local_error(got, ref, floor):
    """Largest error against the largest of an entry and its neighbours, over the
    entries whose surroundings are at least *floor* of the largest."""
    a = ref.abs()
    size = torch.stack([a.roll(-1), a, a.roll(1)]).amax(0)
    m = size > floor * a.max()
    return float(((got - ref).abs()[m] / size[m]).max())


# Entry by entry: the reverse step and autograd differ by the operator's second
# derivative (at most about 1e3 per unit) times a step's roundings of 1e-16, and
# an entry's terms exceed it and its neighbours by at most some 1e3 (the
# farthest taps, 2 / 60 of a face value, thrice): 1e-7 leaves three digits.
LOCAL_BAR = 1.0e-7


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("n", [1025, 1100])
def test_transposed_step_of_compact_cotangents(n, flat):
    """Cotangents that end (or begin) at every cell around the edge of a 512-cell
    tile and of a warp's 58 cells, on a smooth state or one whose left part is
    constant."""
    x = (torch.arange(n, dtype=torch.float64) + 0.5) / n
    u = 0.8 + 0.3 * torch.sin(40 * np.pi * x) + 0.1 * torch.cos(22 * np.pi * x)
    if flat:
        u[200:480] = 0.7
    dx = 2.0 / n
    dt = 0.4 * dx / float(u.abs().max())
    rng = np.random.default_rng(3)
    p0 = torch.tensor(rng.uniform(0.5, 1.0, n))
    for edge in list(range(484, 540)) + list(range(40, 76)):
        for side in (0, 1):
            p = p0.clone()
            if side:
                p[:edge] = 0.0
            else:
                p[edge:] = 0.0
            ref = T.step_vjp(u[None], p[None], dt, dx)[0]
            err = _local_error(_vjp(u, p, dt, dx), ref, 1.0e-30)
            assert err < LOCAL_BAR, (edge, side, err)


@pytest.mark.parametrize(("lo", "hi"), [(-290, -285), (-292, -276), (240, 255), (246, 250), (-260, 260)])
def test_transposed_step_of_cotangents_across_the_scales(lo, hi):
    """Cotangents rising from 10^lo to 10^hi over the cells: inside a few warps
    they pass the magnitudes that the pairs of floats are scaled for."""
    n = 400
    x = (torch.arange(n, dtype=torch.float64) + 0.5) / n
    u = 0.8 + 0.3 * torch.sin(16 * np.pi * x) + 0.1 * torch.cos(10 * np.pi * x)
    dx = 2.0 / n
    dt = 0.4 * dx / float(u.abs().max())
    rng = np.random.default_rng(4)
    p = torch.tensor(rng.uniform(0.5, 1.0, n) * 10.0 ** np.linspace(lo, hi, n))
    ref = T.step_vjp(u[None], p[None], dt, dx)[0]
    inner = slice(20, n - 20)  # (away from the jump of the periodic continuation)
    got = _vjp(u, p, dt, dx)
    a = ref.abs()
    size = torch.stack([a.roll(-1), a, a.roll(1)]).amax(0)
    assert float(((got - ref).abs() / size)[inner].max()) < LOCAL_BAR

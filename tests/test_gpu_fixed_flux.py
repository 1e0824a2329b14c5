"""The integer / float-pair fluxes of the double Burgers step (``csrc/fixed_flux.cuh``)
at the sizes and states where they can go wrong: shorter than a stencil, around
a warp's 60 faces, odd lengths; states whose faces all stay on the integers,
all fall to the FP64 formula, or mix; zero and constant stretches; scales in
and beyond the accepted powers of two.

Tolerance: three steps of three stages, each a handful of roundings of 2^-53
of the largest value, the operator's Lipschitz constant under the CFL bound a
few units: 1e-13 of the largest value (about 900 roundings), against the
oracle's own double arithmetic.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R

pytestmark = pytest.mark.gpu

SIZES = [3, 4, 5, 7, 33, 59, 60, 61, 62, 63, 121, 127, 600, 1031]


def _state(kind, n, rng):
    x = (np.arange(n) + 0.5) / n
    if kind == "smooth":
        return 0.3 + np.sin(2 * np.pi * x) + 0.1 * np.cos(6 * np.pi * x)
    if kind == "noise":
        return rng.uniform(-1.0, 1.0, n)
    if kind == "front":
        return np.where((x > 0.3) & (x < 0.6), 1.0, -0.7) + 0.05 * np.sin(2 * np.pi * x)
    if kind == "plateaus":
        return np.where((x > 0.3) & (x < 0.6), 0.8, 0.0)
    # magnitudes from 1e-12 to 1
    return np.exp(-27.0 * np.abs(2.0 * x - 1.0)) * np.where(x > 0.5, 1.0, -1.0)


@pytest.mark.parametrize("flux", ["rusanov", "lf"])
@pytest.mark.parametrize(("kind", "amp"), [("smooth", 1.0), ("noise", 1.0), ("front", 1.0),
                                           ("plateaus", 1.0), ("range", 1.0), ("smooth", 1e-22),
                                           ("front", 1e-17), ("smooth", 1e17), ("front", 1e19)])
def test_steps_match_oracle(kind, amp, flux):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers
    from pyshocks_gb300.batched import BatchedSolver

    nsteps = 3
    rng = np.random.default_rng(11)
    u0, refs = [], []
    for n in SIZES:
        og = R.make_uniform_cell_grid(-amp, amp, n, 3)
        u = amp * _state(kind, n, rng)
        ug = np.zeros(n + 6)
        ug[3:-3] = u
        ref, _ = R.evolve(R.SchemeSpec(flux_kind=flux), og, ug, theta=0.9, maxit=nsteps)
        u0.append(u)
        refs.append(ref[3:-3])
    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6)
    solver = BatchedSolver(burgers.make_scheme_from_name(flux, rec=rec), SIZES, [2.0 * amp / n for n in SIZES], theta=0.9)
    solver.reset(torch.tensor(np.concatenate(u0)))
    solver.step(nsteps)
    assert solver.status() == 0
    for b, n in enumerate(SIZES):
        err = np.max(np.abs(solver.instance(b).cpu().numpy() - refs[b])) / np.max(np.abs(u0[b]))
        assert err < 1.0e-13, (n, err)


@pytest.mark.parametrize("kind", ["smooth", "noise", "front", "range"])
@pytest.mark.parametrize("scale", [1.0, 1e-250, 1e-30, 1e200, 1e280])
def test_transposed_step_matches_autograd(kind, scale):
    """One reverse step (``fx_vjp_stage``) around a warp's 58 cells and the
    tile of 512, with cotangents of any scale (the pairs of floats work relative
    to the warp's largest). The oracle's step is differentiated at its own
    rounding of the stages; the operator's second derivative is at most about
    1 / sqrt(eps) = 1e3 per unit, so 1e-11 of the largest entry leaves two
    digits over 1e3 times a step's roundings."""
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import _lib as L
    from pyshocks_gb300 import burgers

    from oracle import torch_ref as T

    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6)
    scheme = burgers.Rusanov(rec=rec)
    rng = np.random.default_rng(5)
    for n in [13, 57, 58, 59, 116, 117, 500, 512, 513, 1025]:
        dx = 2.0 / n
        u = torch.tensor(_state(kind, n, rng))
        p = torch.tensor(rng.standard_normal(n)) * torch.tensor(np.exp(-0.05 * np.arange(n)))
        dt = 0.4 * dx / float(u.abs().max())
        ref = T.step_vjp(u[None], p[None], dt, dx)[0]
        ud = torch.cat([u[-3:], u, u[:3]]).cuda()
        pd = torch.cat([p[-3:], p, p[:3]]).cuda() * scale
        out = torch.empty_like(ud)
        st = L.lib().shk_ssprk33_vjp_f64(scheme.c_scheme(dx), ud.data_ptr(), pd.data_ptr(), out.data_ptr(), n, 3, dx,
                                         dt, L.stream_handle())
        assert st == 0, L.errstr(st)
        got = (out / scale).cpu()[3:-3]
        assert float((got - ref).abs().max()) <= 1.0e-11 * float(ref.abs().max()), n

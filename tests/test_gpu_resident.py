"""Plans whose instances each have a CTA for all steps of a call
(``resident_steps_kernel``) against the same plan stepped launch by launch (a
named tile): states, both ping-pong buffers, times, dt history and the next
call's maxima, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import numpy_ref as R

pytestmark = pytest.mark.gpu

SIZES = [3, 5, 9, 47, 61, 250, 1000, 1536]


@pytest.mark.parametrize("copies", [1, 40])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("mode", ["cfl", "tfinal", "fixed", "dirichlet", "neumann"])
def test_resident_steps_equal_launched_steps(dtype, mode, copies):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers
    from pyshocks_gb300.batched import BatchedSolver

    sizes = SIZES if copies == 1 else [n for n in SIZES if n <= 250] * copies
    rng = np.random.default_rng(5)
    u0 = torch.tensor(np.concatenate([R.random_fourier_ic(rng, np.linspace(-1, 1, n + 1)) for n in sizes]))
    rec = gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=1.0e-6)
    out = []
    for tile in (0, 512):
        s = BatchedSolver(burgers.Rusanov(rec=rec), sizes, [2.0 / n for n in sizes], theta=0.8, tile=tile,
                          dtype=dtype, max_steps=12)
        if mode in ("dirichlet", "neumann"):
            s.set_boundary(mode, dirichlet=[0.3, -0.2], neumann=[0.1, 0.0])
        s.reset(u0, tfinal=None if mode != "tfinal" else 0.004)
        if mode == "fixed":
            s.set_fixed_dt(torch.tensor([1e-4, 2e-4, 0.0, 1e-4, 3e-5]))
        for k in (1, 4, 2, 3):
            s.step(k)
        assert s.status() == 0
        out.append((s.buf_a.clone(), s.buf_b.clone(), s.time(), s.dt_history()))
    for a, b in zip(*out):
        assert torch.equal(a, b)

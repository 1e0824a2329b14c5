"""Resident plans (all steps of a call in one launch) at their limits: a wait that
runs out, batches of mixed lengths on either side of the rule that chooses them, and
calls longer than one launch."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scheme(eps=1.0e-6):
    import pyshocks_gb300 as gb
    from pyshocks_gb300 import burgers

    return burgers.Rusanov(rec=gb.reconstruction.make_reconstruction_from_name("wenojs53", eps=eps))


def test_a_timed_out_window_writes_no_state():
    """The hook lets the window's bounded wait expire: the plan reports it, and
    neither buffer changes, as with the launched step."""
    from test_gpu_bounds_check import library

    from pyshocks_gb300 import _build
    from pyshocks_gb300 import _lib as L
    from pyshocks_gb300.batched import BatchedSolver

    if not L.CHECK_LIB_PATH.exists():
        _build.build(variants=("check",))
    checked = L.load_check_library()
    n = 1024
    u0 = torch.linspace(0.5, 1.5, n, dtype=torch.float64)
    for tile in (0, 512):
        with library(checked):
            s = BatchedSolver(_scheme(), [n], 2.0 / n, tile=tile)
            s.buf_b.fill_(7.0)
            s.reset(u0)
            assert checked.shk_check_force_timeout(16, 1024) == 0
            try:
                s.step(1)
                torch.cuda.synchronize()
                assert s.status() & L.ERR_TIMEOUT
            finally:
                assert checked.shk_check_force_timeout(0, 0) == 0
            assert torch.equal(s.buf_a.cpu(), u0)
            assert torch.all(s.buf_b == 7.0)


@pytest.mark.parametrize("long_share", [2, 10, 400])
@pytest.mark.parametrize("batch", [300, 456, 760])
def test_mixed_lengths_equal_launched_steps(batch, long_share):
    """Every second, every tenth instance, or one, has 1500 cells and the others 200
    (two, three and five instances an SM): bit for bit the launched steps."""
    from pyshocks_gb300.batched import BatchedSolver

    sizes = np.where(np.arange(batch) % long_share, 200, 1500)
    if long_share == 400:
        sizes[1:] = 200
    rng = np.random.default_rng(9)
    x = np.concatenate([(np.arange(n) + 0.5) / n for n in sizes])
    u0 = torch.tensor(0.4 + np.sin(2 * np.pi * x) * np.repeat(rng.uniform(0.2, 1.0, batch), sizes))
    out = []
    for tile in (0, 466):
        s = BatchedSolver(_scheme(), sizes, 2.0 / sizes, theta=0.9, tile=tile)
        s.reset(u0)
        s.step(3)
        s.step(2)
        assert s.status() == 0
        out.append((s.u.clone(), s.time()))
    assert torch.equal(out[0][0], out[1][0])
    assert torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nsteps", [511, 512, 513, 1025])
def test_long_calls_equal_launched_steps(nsteps, dtype):
    """A call of more than 512 steps takes several launches: both buffers and the
    times of the launched steps, bit for bit, and of the call after it."""
    from pyshocks_gb300.batched import BatchedSolver

    sizes = np.array([40, 77, 128])
    x = np.concatenate([(np.arange(n) + 0.5) / n for n in sizes])
    out = []
    for tile in (0, 64):
        s = BatchedSolver(_scheme(), sizes, 2.0 / sizes, theta=0.9, tile=tile, dtype=dtype)
        s.reset(torch.tensor(0.4 + np.sin(2 * np.pi * x)))
        s.step(nsteps)
        s.step(2)
        assert s.status() == 0
        out.append((s.buf_a.clone(), s.buf_b.clone(), s.time()))
    for a, b in zip(*out):
        assert torch.equal(a, b)

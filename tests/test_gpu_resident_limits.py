"""Resident plans (all steps of a call in one launch) at their limits: a wait that
runs out."""

from __future__ import annotations

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

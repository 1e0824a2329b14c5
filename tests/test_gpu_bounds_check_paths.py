"""The integer-flux, resident, one-CTA and listed-face tests again under the
bounds-check build (see ``test_gpu_bounds_check.py``): every parameter set, the
library swapped, and no violation in the log."""

from __future__ import annotations

import importlib

import pytest

from test_gpu_bounds_check import _param_sets, checked, library, read_log  # noqa: F401

pytestmark = pytest.mark.gpu

RERUN = [
    ("test_gpu_fixed_flux", "test_steps_match_oracle"),
    ("test_gpu_fixed_flux", "test_transposed_step_matches_autograd"),
    ("test_gpu_fixed_flux_range", "test_steps_for_any_smoothness_parameter"),
    ("test_gpu_fixed_flux_range", "test_transposed_step_of_cotangents_across_the_scales"),
    ("test_gpu_listed_faces", "test_steps_match_oracle_and_do_not_depend_on_the_tile"),
    ("test_gpu_listed_faces", "test_gradient_does_not_depend_on_the_tile"),
    ("test_gpu_listed_faces", "test_single_step_and_transpose_on_coarse_grids"),
    ("test_gpu_resident", "test_resident_steps_equal_launched_steps"),
    ("test_gpu_resident_limits", "test_mixed_lengths_equal_launched_steps"),
    ("test_gpu_block_paths", "test_ghosted_step_and_transpose"),
    ("test_gpu_block_paths", "test_predicted_timestep"),
    ("test_gpu_block_paths", "test_many_items_per_cta_report_every_maximum"),
    ("test_gpu_short_calls", "test_predicted_timestep"),
    ("test_gpu_short_calls", "test_ghosted_step_and_transpose"),
]


def _cases():
    out = []
    for modname, fname in RERUN:
        fn = getattr(importlib.import_module(modname), fname)
        for i, kw in enumerate(_param_sets(fn)):
            out.append(pytest.param(modname, fname, kw, id=f"{modname}-{fname}-{i}"))
    return out


@pytest.mark.parametrize(("modname", "fname", "kwargs"), _cases())
def test_no_bounds_violation(checked, modname, fname, kwargs):  # noqa: F811
    fn = getattr(importlib.import_module(modname), fname)
    with library(checked):
        read_log(checked, reset=True)
        fn(**kwargs)
        log = read_log(checked, reset=True)
    assert log["flag"] == 0, log

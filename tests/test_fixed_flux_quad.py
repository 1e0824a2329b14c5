"""The integer / float-pair arithmetic of ``csrc/fixed_flux.cuh``, built for the host,
against 113-bit arithmetic (``fixed_flux_quad.cpp``): smooth to slightly noisy states
of any accepted scale, eps from 1e-24 to 1e24.

Units: 2^-53 of the largest of a face's four cells, squared for fluxes. A flux is a
sum of integers of 2^-57 of that and two pairs of floats whose error stays below
2^-54: a few units, and no more in the mean than the FP64 formula. The backward's
terms carry pairs of about 45 bits times at most 1/8: 2^-44, 512 units of the
largest seed."""

from __future__ import annotations

import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "pyshocks_gb300" / "csrc"


@pytest.fixture(scope="module")
def values(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path_factory.mktemp("quad") / "fixed_flux_quad"
    # (no contraction: the sums of two floats are error-free as written)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC), "-o", str(exe),
                    str(HERE / "fixed_flux_quad.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {k: float(v) for k, v in (line.split() for line in out.splitlines())}


def test_enough_faces_of_each_kind(values):
    for kind in ("rusanov", "lf", "listed", "rough", "lf_rough", "grad"):
        assert values[f"{kind}.count"] > 10000


def test_fluxes(values):
    assert values["rusanov.rms"] <= values["formula.rms"]
    for kind in ("rusanov", "lf", "faces", "listed", "rough", "lf_rough"):
        assert values[f"{kind}.max"] <= 8.0, kind


def test_backward_of_the_weights(values):
    assert values["grad.max"] <= 512.0


def test_conversions(values):
    """Integers to doubles to the nearest; doubles to pairs and back, at most
    2^80 below the pair's scale: 24 bits truncated and the other 29 rounded to 24,
    2^-48 (32 units)."""
    assert values["to_double.max"] <= 1.0
    assert values["split.max"] <= 32.0

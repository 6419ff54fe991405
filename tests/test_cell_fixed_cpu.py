"""The fixed-point collision of the FP64 form (csrc/cell_fixed.h), compiled for the
CPU, against 113-bit arithmetic and against the same update in double.

Bound: a result of the fixed-point update is off by a few units of 2^-56 of the cell's
largest value (rounded products) and by its own rounding to double, the double update
by a rounding of up to 2^-53 at each of about ten dependent operations; so over cells of
every kind the fixed-point error must not exceed the double one, neither its largest
value nor its root mean square.  Fluid cells get the same bits with and without the
solid terms, zeros stay zeros, and cells outside the range are refused.
"""
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("fixed") / "cell_fixed_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{PKG / 'csrc'}",
                    str(ROOT / "tests" / "cell_fixed_check.cpp"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_error_no_larger_than_double(program, seed):
    out = subprocess.run([str(program), "4000", str(seed)], check=True, capture_output=True, text=True).stdout
    lines = [ln.split() for ln in out.splitlines()]
    kinds = [ln for ln in lines if len(ln) == 11]
    assert len(kinds) == 14
    for name, fx, fr, dx, dr, ffx, ffr, fdx, fdr, bits, left_out in kinds:
        if int(left_out) < 3900:
            assert float(fx) <= float(dx) and float(fr) <= float(dr), name
            assert float(ffx) <= float(fdx) and float(ffr) <= float(fdr), name
        assert int(bits) == 0, name
        if name in ("fluid", "solid", "slow_fluid", "slow_solid", "noise", "faint_fluid", "resting_bed",
                    "driven_fluid", "driven_solid", "pushed_fluid", "pushed_solid"):
            assert int(left_out) == 0, name
    assert ["zero", "1"] in lines and ["refused", "5"] in lines

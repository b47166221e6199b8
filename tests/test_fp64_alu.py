"""The FP64 division, square root and ordering on the integer units
(csrc/fp64_alu.cuh), compiled for the host: the bits of the host's IEEE
operations over random and edge operands, with the FP32 seed as it is and moved
by up to two units in the last place (the approximate reciprocals of a GPU are
good to one)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("ulps", [-2, -1, 0, 1, 2])
def test_integer_division_and_square_root_are_ieee(tmp_path, ulps):
    exe = str(tmp_path / "alu")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DE2D_SEED_ULPS={ulps}",
                    os.path.join(ROOT, "tests", "fp64_alu_driver.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe, "1000000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0 and res.stdout.strip() == "0", res.stdout

"""The FP64 form's forward register rounds (tests/host/fp64_round_check.c):
with only the named outputs reduced, values stay in the FP64 quotient's range
and every output within what the next round accepts, exactly congruent.  And
its CRT (tests/host/crt56_check.c): the coefficient's base-2^56 digits from any
representatives the inverse transforms leave."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
@pytest.mark.parametrize("bits", [1, 2, 3, 4])
def test_forward_round_ranges(tmp_path, bits):
    exe = tmp_path / "fp64_round_check"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "host", "fp64_round_check.c"), "-lm"], check=True)
    out = subprocess.run([str(exe), str(bits), "200000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("bad=0"), out.stdout + out.stderr


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
@pytest.mark.parametrize("terms", [1, 2])
@pytest.mark.parametrize("row_bits", [4, 5, 9, 10, 11, 12, 13])
def test_middle_round_ranges(tmp_path, row_bits, terms):
    """The last forward and the first inverse round of a row without the products
    by one (tests/host/fp64_middle_check.c)."""
    exe = tmp_path / "fp64_middle_check"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe),
                    os.path.join(HERE, "host", "fp64_middle_check.c"), "-lm"], check=True)
    out = subprocess.run([str(exe), str(row_bits), str(terms), "50000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("bad=0"), out.stdout + out.stderr


@pytest.mark.skipif(shutil.which("gcc") is None, reason="gcc not available")
def test_crt_digits_exact(tmp_path):
    exe = tmp_path / "crt56_check"
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", str(exe), os.path.join(HERE, "host", "crt56_check.c"),
                    "-lm"], check=True)
    out = subprocess.run([str(exe), "300000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("bad=0"), out.stdout + out.stderr


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_short_column_passes_meet_the_rows_in_range(tmp_path):
    """Column passes of one to three bits (and the round beside the twiddles of
    longer ones) from the largest pieces into a row's first round, and from the
    largest values a row leaves to what the CRT accepts: the device templates
    themselves, built for the host (tests/host/fp64_columns_check.cpp)."""
    exe = tmp_path / "fp64_columns_check"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(HERE, "host", "cuda_shim"),
                    "-I", os.path.join(os.path.dirname(HERE), "piculator_b200", "csrc"), "-o", str(exe),
                    os.path.join(HERE, "host", "fp64_columns_check.cpp")], check=True)
    out = subprocess.run([str(exe), "20000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("bad=0"), out.stdout + out.stderr

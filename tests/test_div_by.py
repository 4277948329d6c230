"""The clouds' division by the cell width through its reciprocal (div_by) gives the bits of the
division, which the gathered velocities' equality with the oracle rests on."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("div_by") / "div_by")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "host", "div_by.cpp")], check=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_quotients_have_the_bits_of_the_division(program, seed):
    r = subprocess.run([program, "2000000", str(seed)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    assert "6000002 quotients" in r.stdout

"""The integer-pipe quotient over the exponents that the solvers' quotient()
accepts (i64fp::in_window<400>), against the host's IEEE binary64 one, bit for
bit."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_quotients_match_ieee_over_the_solvers_range(tmp_path, seed):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "fp64_int_quotient_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "arcanefem_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "fp64_int_quotient_check.cc"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, "8000000", str(seed)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert list(map(int, out.stdout.split())) == [0, 0]

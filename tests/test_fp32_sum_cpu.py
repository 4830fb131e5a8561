"""The compensated FP32 sums of arcanefem_gb300/csrc/afem_fp32_sum.cuh: never
further from the sum in double than the plain tree over a thread per value that
they stand for, and infinities and NaN as plain additions give them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_compensated_sums_are_no_further_off_than_a_tree(tmp_path, seed):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "fp32_sum_check")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", "-I",
                        os.path.join(ROOT, "arcanefem_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "fp32_sum_check.cc"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe, "2000", str(seed)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    *rows, special = out.stdout.strip().split("\n")
    assert special.split() == ["1"] * 6
    assert len(rows) == 6
    for row in rows:
        mine, tree = map(float, row.split())
        assert mine <= tree

"""The plan of Pauli strings on the host, no GPU (tests/pauli_plan_check.cu)."""
import os
import subprocess

import pytest

from test_batch_program_host import HERE, ROOT, _nvcc


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_plans_equal_a_walk_and_take_linear_time(tmp_path):
    exe = str(tmp_path / "pauli_plan_check")
    cmd = [_nvcc(), "-std=c++17", "-O2", "-x", "cu", "-I" + os.path.join(ROOT, "ruqu_b200", "csrc"),
           "-I" + os.path.join(ROOT, "include"), "-o", exe, os.path.join(HERE, "pauli_plan_check.cu")]
    b = subprocess.run(cmd, capture_output=True, text=True)
    assert b.returncode == 0, b.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert r.stdout.rstrip().endswith(" 0 failures")

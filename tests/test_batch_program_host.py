"""The programs of the batched QAOA and VQE engines (ruqu_b200/csrc/rq_plan.cuh) on the host, no GPU:
tests/batch_program_check.cu runs each one tile by tile and phase by phase as the kernels do and
compares it with the circuit on the whole state (see the program's header)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _nvcc():
    for c in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if c and os.path.exists(c):
            return c
    return None


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_symmetric_and_packed_programs_equal_the_circuit(tmp_path):
    exe = str(tmp_path / "batch_program_check")
    cmd = [_nvcc(), "-std=c++17", "-O2", "-x", "cu", "-I" + os.path.join(ROOT, "ruqu_b200", "csrc"),
           "-I" + os.path.join(ROOT, "include"), "-o", exe, os.path.join(HERE, "batch_program_check.cu")]
    b = subprocess.run(cmd, capture_output=True, text=True)
    assert b.returncode == 0, b.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert r.stdout.rstrip().endswith(" 0 failures")

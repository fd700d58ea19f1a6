"""The integer-pipe square root of the Givens rotations (hsr_device.cuh:
ip_sqrt, ip_recip_root) compiled for the host and compared bit for bit with
the host's IEEE square root and division on 2e7 seeded operands.  Both are
correctly rounded, so the device's FP64 instructions give the same bits; the
device build of the same code is checked by every bitwise test against the
oracle."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_integer_pipe_square_root_on_host(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "intsqrt_check")
    src = os.path.join(HERE, "native", "intsqrt_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-o", exe, src],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe, "20000000"], check=False, capture_output=True, text=True, timeout=600)
    roots, bad, quots, badq = (int(v) for v in out.stdout.strip().split()[-4:])
    assert out.returncode == 0 and bad == 0 and badq == 0, out.stdout
    assert roots == 20000000 and quots > 0.8 * roots

"""The conversions of digit sums to FP64 (hsr_digits.cuh: dg_value) compiled
for the host: sums next to powers of two, whose rounding carries through every
bit, and seeded ones, against exact integer arithmetic."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_digit_sums_to_fp64_on_host(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "digitsum_check")
    src = os.path.join(HERE, "native", "digitsum_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-o", exe, src],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe, "1000000"], check=False, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout
    sums, bad1, bad2 = (int(v) for v in out.stdout.strip().split()[-3:])
    assert bad1 == 0 and bad2 == 0 and sums > 2000000, out.stdout


def test_failed_product_marks_every_part(tmp_path):
    """A digit product whose wait ran out leaves NaN in all its parts."""
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "digitpoison_check")
    src = os.path.join(HERE, "native", "digitpoison_check.cu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-o", exe, src],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe], check=False, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout

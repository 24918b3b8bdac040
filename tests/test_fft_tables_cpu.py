"""The tables of the transform stages' twiddles, for every plan: the bits of the
roots of unity they are laid out from."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_stage_tables_of_every_plan(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "tables")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-diag-suppress", "177", "-I" + os.path.join(ROOT, "colore_gb300", "csrc"),
                    "-o", exe, os.path.join(HERE, "fft_tables_check.cu")], check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert [int(v) for v in out[0::2]] == [64, 96, 128, 192, 256, 384, 512, 1024, 2048]
    assert all(int(v) == 0 for v in out[1::2]), out

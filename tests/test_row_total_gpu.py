"""A row's triangles are summed in 64 bits: a block's row with more than 2^32 of them."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_row_of_more_than_2_32_triangles(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "row_total")
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Wno-deprecated-gpu-targets", os.path.join(HERE, "native", "row_total.cu"),
                    "-o", exe], check=True)
    f, rounds = 1100, 3640                       # two chunks of members
    hits = f * f * rounds
    assert hits > 1 << 32
    run = subprocess.run([exe, str(f), str(rounds)], check=True, capture_output=True, text=True,
                         timeout=120)
    assert run.stdout.split("\n")[:2] == [f"{hits} {hits} 1", f"0 {hits} 1"]

"""CPU check of the operand copies of the CUDA-core FP32, plain FP64 and grouped kernels
(csrc/fp32_copy.cuh, csrc/fp64_copy.cuh): tests/copy_maps.cpp compiles the headers
themselves for the host and runs every thread's copies for tiles inside and at the edges
of operands of any alignment and leading dimension."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gemm_avx512f_b200", "csrc")


def test_copies_stay_inside_and_land_where_fragments_read(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "copy_maps")
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "copy_maps.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout

"""The step loop of the FP64 stream's normal sum counts groups of four draws in
64 bits: 2^34 steps and more are accepted by the pathwise Greeks, and 2^32
groups in 32 bits are none.  Such a path takes minutes on the GPU, so the
count is checked where the kernel takes it from, at compile time."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = """
#include "ref_stream.cuh"
static_assert(sizeof(of::draw_groups(int64_t{1})) == 8, "the loop counter holds any step count");
static_assert(of::draw_groups((int64_t{1} << 34) + 3) == int64_t{1} << 32, "2^34 + 3 steps");
static_assert(of::draw_groups(3) == 0 && of::draw_groups(4) == 1, "small step counts");
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_group_count_holds_any_step_count(tmp_path):
    src = tmp_path / "groups.cu"
    src.write_text(SOURCE)
    r = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--fmad=false", "-I",
                        os.path.join(ROOT, "openferric_b200", "csrc"), "-I", os.path.join(ROOT, "include"), "-c",
                        str(src), "-o", str(tmp_path / "groups.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

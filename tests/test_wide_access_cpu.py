"""Objects that kernels read and write through 16-byte accesses are aligned for
them by their type, wherever the compiler places them."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "gpu_testbed_poisson-gravity_b200", "csrc")

SOURCE = """
#include "gravity.cuh"
static_assert(alignof(gpg::FluidRun<float>) == 16, "FP32 run");
static_assert(alignof(gpg::FluidRun<double>) == 16, "FP64 run");
static_assert(sizeof(gpg::FluidRun<float>) == 5 * 16 && sizeof(gpg::FluidRun<double>) == 5 * 16, "rows stay aligned");
"""


def test_fluid_runs(tmp_path):
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    nvcc = nvcc if os.path.exists(nvcc) else shutil.which("nvcc")
    if not nvcc:
        pytest.skip("no nvcc")
    src = tmp_path / "align.cu"
    src.write_text(SOURCE)
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                        "-I", CSRC, "-c", str(src), "-o", str(tmp_path / "align.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]

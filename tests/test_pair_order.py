"""The tile order of the CTA-pair Gram kernels (gputools_gb300/csrc/gram_core.cuh),
checked on the host by tests/pair_order_check.cu, built by nvcc and run without
a GPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_pair_order_covers_each_tile_once(tmp_path):
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"),
                                                "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "pair_order_check"
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "gputools_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", str(exe),
                    os.path.join(HERE, "pair_order_check.cu"), "-lcuda"],
                   check=True, timeout=600)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr

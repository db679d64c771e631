"""A guiding step that failed on the device leaves the network as it was.

A backward CTA that gives up waiting on its tensor cores raises the error word and leaves no row of
gradient sums. The word is set from the host here (no wait is made to fail), the rows are NaN, and the
step's kernels are launched as the library launches them: tests/native/guide_failed_step.cu, compiled
against the library's own sources.
"""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def build(exe):
    src = os.path.join(ROOT, "photon-v2_b200", "csrc")
    subprocess.run([os.path.join(CUDA, "bin", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                    "--expt-relaxed-constexpr", "-I", src, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "native", "guide_failed_step.cu"),
                    os.path.join(src, "guide_train.cu"), os.path.join(src, "guide_mlp.cu"),
                    os.path.join(src, "pg_runtime.cpp"), "-o", str(exe)], check=True)


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which(os.path.join(CUDA, "bin", "nvcc")) is None, reason="needs nvcc")
def test_failed_step_leaves_the_network_alone(gpu_lib, tmp_path):
    exe = tmp_path / "guide_failed_step"
    build(exe)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.strip() == "ok"

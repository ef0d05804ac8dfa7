"""The FP64 inverse square root of the sampled direct sums (csrc/wide.cuh,
rsqrt64): the SFU's estimate is as near as its one step needs, and the result as
near as its comment derives, 2^-53 + 2^-54 + 2^-55 < 2^-52."""

import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.mark.gpu
def test_rsqrt64_and_its_estimate(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "rsqrt64_check"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    str(ROOT / "tests" / "cuda" / "rsqrt64_check.cu"), "-o", str(exe)],
                   check=True)
    f = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    print(f)
    assert 0 < float(f[f.index("estimate") + 1]) < 2.0 ** -18
    assert 0 < float(f[f.index("result") + 1]) < 2.0 ** -52

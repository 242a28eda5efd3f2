"""The word by which a solve tells the host of its iterations, past the counts
that the word's bits hold: a small program built with nvcc, run on the CPU."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT


def test_the_host_follows_long_solves(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "checks")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "published_word_checks.cu"), "-o", exe],
                   check=True, capture_output=True, text=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout == "bad 0\n"

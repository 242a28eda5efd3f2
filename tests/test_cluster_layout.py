"""Host construction of the cluster-resident smoothing layout: a small program
around cluster_layout.h, built with nvcc, run on the CPU."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("cluster") / "checks")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "cluster_layout_checks.cu"), "-L", PKG, "-lgpusolver_b200",
                    "-Xlinker", f"-rpath={PKG}", "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def test_messages_stay_inside_the_cluster(program):
    out = subprocess.run([program], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split("\n")[0] == "bad 0"


def test_new_values_go_to_their_places(program):
    """Refreshed in place, the layout equals one built from the new values."""
    out = subprocess.run([program], check=True, capture_output=True, text=True, timeout=120).stdout
    assert out.split("\n")[1] == "stale 0"

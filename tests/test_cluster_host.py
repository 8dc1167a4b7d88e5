"""Layouts and index arithmetic of the cluster-resident lens (cmblensing_b200/csrc/lf_cluster.cuh), on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not found")
def test_cluster_layouts(tmp_path):
    exe = tmp_path / "cluster_check"
    subprocess.check_call(["nvcc", "-std=c++17", "-Wno-deprecated-gpu-targets", "-gencode",
                           "arch=compute_100a,code=sm_100a", "-o", str(exe),
                           os.path.join(HERE, "native", "cluster_check.cu")])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert len(r.stdout.strip().splitlines()) == 6

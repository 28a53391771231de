"""The waits of the aggregation pipelines for ranks that share a GPU, compiled for the host with a warp of 32 threads
(csrc/tests/one_gpu_waits_model.cc)."""
import os
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "p4app-switchML_b200")


@pytest.fixture(scope="module")
def output(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("waits") / "one_gpu_waits_model")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", "-I" + os.path.join(PKG, "include"), "-I" + os.path.join(PKG, "csrc"),
                    "-I" + cuda, os.path.join(PKG, "csrc", "tests", "one_gpu_waits_model.cc"), "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True, timeout=120).stdout


@pytest.mark.parametrize("case", ["lanes_that_read_different_counts", "a_wait_that_runs_out_is_reported"])
def test_case(output, case):
    assert "ok   " + case in output, output

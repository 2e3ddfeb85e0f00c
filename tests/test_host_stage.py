"""The pinned staging of host arrays, on the CPU: host_stage.cu over a stand-in for the CUDA runtime (host_stage_check.cpp)."""
import os
import subprocess

from conftest import ROOT


def test_staging_leaves_nothing_in_flight(tmp_path):
    exe = str(tmp_path / "host_stage_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-x", "c++",
                    os.path.join(ROOT, "llama2.rs_b200", "csrc", "host_stage.cu"), os.path.join(ROOT, "tests", "host_stage_check.cpp"),
                    "-o", exe, "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

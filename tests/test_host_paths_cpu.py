"""Failure paths of the library's host code, against a CUDA runtime without a
GPU whose calls fail on demand (tests/fake_cudart.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "pagani-toolkit_b200")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("host")
    inc = os.path.join(os.path.dirname(HERE), "include")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(NVCC))), "include")
    objs, exe = [], str(d / "host_paths")
    for src in (os.path.join(PKG, "csrc", "api_core.cu"), os.path.join(PKG, "csrc", "tune.cu"), os.path.join(HERE, "host_paths.cpp")):
        objs.append(str(d / (os.path.basename(src) + ".o")))
        subprocess.run([NVCC, "-x", "cu", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", f"-I{inc}",
                        "-c", src, "-o", objs[-1]], check=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{cuda}", os.path.join(HERE, "fake_cudart.cpp"), *objs,
                    "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("name", ["large_copy_that_fails", "large_copy_without_staging", "idle_buffers_make_room",
                                  "saved_choice_that_does_not_fit", "error_that_is_over"])
def test_host_path(harness, name, tmp_path):
    r = subprocess.run([harness, name], capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, PAGANI_TUNE_CACHE=str(tmp_path / "tune.txt")))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr

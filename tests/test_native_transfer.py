"""The native transfer code against a CUDA runtime that is played by the CPU (``native/fake_cuda.h``): what happens when a
launch fails, and what a GPU may still have to do when a call returns."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "flexkv_b200", "csrc")


def _run(tmp_path, program, sources):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if cxx is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no C++ compiler or no CUDA headers")
    exe = str(tmp_path / program)
    cmd = [cxx, "-std=c++17", "-O1", "-g", f"-I{CSRC}", f"-I{include}", os.path.join(HERE, "native", program + ".cpp"),
           *(os.path.join(CSRC, s) for s in sources), "-pthread", "-o", exe]
    subprocess.run(cmd, check=True, timeout=300)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and "OK" in p.stdout, (p.stdout + p.stderr)[-4000:]


TRANSFER = ("transfer_group.cpp", "ce_copy.cpp", "ptr_table.cpp", "kv_copy_host.cpp")


def test_failed_launch_leaves_nothing_in_flight(tmp_path):
    _run(tmp_path, "failed_launch", TRANSFER)


def test_failed_layerwise_restore_leaves_nothing_in_flight(tmp_path):
    _run(tmp_path, "failed_layerwise", ("layerwise_group.cpp",) + TRANSFER)


def test_threads_share_a_group(tmp_path):
    _run(tmp_path, "shared_group", TRANSFER)


def test_staging_memory_is_taken_only_where_it_can_be_used(tmp_path):
    _run(tmp_path, "device_memory", ("layerwise_group.cpp",) + TRANSFER)

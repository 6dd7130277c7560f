"""Kernels' shared-memory limits under concurrent callers, on the host: compiles tests/smem_attr_check.cpp
against torchfsm_gb300/csrc/fsm_smem_attr.h with a stand-in for the attribute call."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "torchfsm_gb300", "csrc")


def test_limits_only_grow(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "smem_attr_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC,
                    os.path.join(HERE, "smem_attr_check.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr

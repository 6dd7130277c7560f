"""How the parts of a split batch are enqueued and joined, on the host: compiles tests/split_check.cpp
against torchfsm_gb300/csrc/fsm_split.h with stand-in streams, every call failing in turn."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "torchfsm_gb300", "csrc")


def test_parts_are_joined_whatever_fails(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "split_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, os.path.join(HERE, "split_check.cpp"),
                    "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr

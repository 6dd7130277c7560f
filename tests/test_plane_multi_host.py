"""What the multi-plan column launch refuses, on the host: compiles tests/plane_multi_check.cu against
the library (the refusals come before any call to the device)."""

import os
import subprocess

import pytest

from torchfsm_gb300 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_multi_plan_column_launch_refusals(tmp_path):
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    _lib.load()
    exe = str(tmp_path / "plane_multi_check")
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                    os.path.join(build.REPO, "include"), os.path.join(HERE, "plane_multi_check.cu"), build.LIB,
                    "-Xlinker", "-rpath=" + build.BUILD, "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr

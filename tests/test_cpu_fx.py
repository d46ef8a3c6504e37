"""The fixed-point columns (adg_fx.cuh) compiled for the host, where their
results can be compared with wider arithmetic (tests/cxx/test_fx.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX_DIR = os.path.join(ROOT, "tests", "cxx")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    c = shutil.which("g++") or shutil.which("c++")
    if not c:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("fx") / "test_fx")
    r = subprocess.run([c, "-std=gnu++17", "-O2", "-I", CXX_DIR, "-I", os.path.join(ROOT, "ader-dg-amr_gb300", "csrc"),
                        os.path.join(CXX_DIR, "test_fx.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("check", ["pressure_floor", "flux_accuracy", "zero_columns"])
def test_fixed_point_columns(exe, check):
    r = subprocess.run([exe, check], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr

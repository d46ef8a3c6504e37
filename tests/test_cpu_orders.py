"""The sample orders of training epochs on their way to the GPU
(adg_orders.hpp), over a copy queue that reads its sources late."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX_DIR = os.path.join(ROOT, "tests", "cxx")


def test_every_epoch_gets_its_own_order(tmp_path):
    c = shutil.which("g++") or shutil.which("c++")
    if not c:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "test_orders")
    r = subprocess.run([c, "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "ader-dg-amr_gb300", "csrc"),
                        os.path.join(CXX_DIR, "test_orders.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout

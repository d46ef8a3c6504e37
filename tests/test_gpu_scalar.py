"""The kernels' own reciprocal, square root and conversions give what CUDA's
operators give, bit for bit, and the 60-bit reciprocal its units
(tests/cxx/test_scalar.cu): 2^27 arguments, the borders of the fast ranges,
ties and subnormal numbers among them."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scalar_functions(tmp_path):
    from adg_gb300 import build

    exe = str(tmp_path / "test_scalar")
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O2", "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cxx", "test_scalar.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = {f: (int(n), first) for f, n, first in (line.split() for line in r.stdout.splitlines())}
    assert set(rows) == {"fast_rcp", "fast_sqrt", "to_float", "to_double", "fx_reciprocal"}
    assert all(n == 0 for n, _ in rows.values()), rows

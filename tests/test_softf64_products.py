"""The special products of csrc/svm_softf64.cuh (a square, the exact product of two floats, a sign flip),
compiled for the host: bit for bit the IEEE results."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_special_products(tmp_path, seed):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "curvedspacevertexmodel_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "softf64_products_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "2000000", str(seed)], capture_output=True, text=True, timeout=300, check=True)
    out = json.loads(r.stdout)
    assert out.pop("cases") == 2000000 and not any(out.values()), out

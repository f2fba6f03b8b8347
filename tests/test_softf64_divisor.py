"""The divisor forms of csrc/svm_softf64.cuh (a reciprocal kept for several quotients, a square root used
as a divisor) and the FP32 sign filter of csrc/svm_det_filter.h, compiled for the host: bit for bit the
IEEE results whatever the seeds' last bits, and never another sign than the FP64 determinant's."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "curvedspacevertexmodel_gb300", "csrc")


def _run(tmp_path, source, *flags):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", *flags, "-I" + CSRC,
                    os.path.join(ROOT, "tests", "native", source), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    return r.returncode, json.loads(r.stdout)


@pytest.mark.parametrize("ulps", [-4, 0, 4])
def test_quotients_by_kept_divisors_and_roots(tmp_path, ulps):
    rc, out = _run(tmp_path, "softf64_divisor_check.cpp", f"-DSF_HOST_SEED_ULPS={ulps}")
    assert rc == 0 and not any(out.values()), out


def test_determinant_sign_filter(tmp_path):
    rc, out = _run(tmp_path, "det_filter_check.cpp")
    assert rc == 0 and out["wrong"] == 0, out
    assert out["undecided"] < 0.01 * out["ordinary"], out   # it decides nearly all ordinary triangles

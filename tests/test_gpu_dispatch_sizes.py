"""Both sides of the sizes at which a single FP64 sphere's kernels change: 3000 vertices (hardware or
integer-pipe products), 20,000 cells (two threads a cell or one), 50,000 vertices (one corner kernel or
two; the T1 pass over a cluster of blocks or a cooperative grid).  A sphere of n cells has 2n - 4
vertices, so most are no multiple of the 32 vertices of a force or corner block.  With one arccosine on
both sides the device and the oracle agree bit for bit (test_gpu_portable_acos.py); the energy is a tree
sum there, so it is held to the rounding of a sum of that many terms."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("cells", [(33, 100, 1501, 1502, 1503), (10003,), (19999, 20001), (25001, 25003)])
@pytest.mark.parametrize("jitter,threshold,flips", [(0.1, 0.04, False), (0.3, 0.15, True)])
def test_steps_match_oracle_bit_for_bit(svm_lib, jitter, threshold, flips, cells):
    lib = os.path.join(ROOT, "curvedspacevertexmodel_gb300", "libsvm_pacos.so")
    assert os.path.exists(lib), "libsvm_pacos.so was not built"
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "dispatch_sizes_run.py"), str(jitter),
                        str(threshold), *map(str, cells)],
                       env=dict(os.environ, SVM_LIBRARY=lib), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    for rep in json.loads(r.stdout.strip().splitlines()[-1]):
        assert rep["steps"] == 3 and rep["checks"] == 3 and (rep["flips"] > 0 or not flips or rep["cells"] < 1000), rep
        for key in ("pos_bits_differ", "flips_differ", "topology_differ", "area_perimeter_bits_differ",
                    "energy_cpu_order_bits_differ", "force_bits_differ", "status"):
            assert rep[key] == 0, rep
        assert rep["energy_reduction_rel"] < 2 * rep["cells"] * 2.0 ** -53, rep

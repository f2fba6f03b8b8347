"""Calls whose device memory is refused raise, and can be made again (tests/refused_memory_run.py)."""
import json
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def run(svm_lib, oracle_mod, tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = str(tmp_path_factory.mktemp("shim") / "refuse_malloc.so")
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", os.path.join(ROOT, "tests", "native", "refuse_malloc.cpp"), "-o", so,
                    "-ldl"], check=True)

    def go(*args):
        r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "refused_memory_run.py"), *map(str, args)],
                           env=dict(os.environ, LD_PRELOAD=so), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-3000:]
        return json.loads(r.stdout.strip().splitlines()[-1])

    return go


@pytest.mark.parametrize("blocks", [0, 1, 4])
def test_ring_growth_refused_before_a_pass(run, blocks):
    rep = run("growth", blocks)
    assert rep.pop("refused") == [True, True, True], rep
    assert rep == dict(flips=True, neighbours=True, growths=1, status=0, step=True), rep


@pytest.mark.parametrize("first,samples", [(0, 512), (1, 1500)])
def test_training_refused_room_for_its_sums(run, first, samples):
    """The refused call has taken no step: Adam's bias corrections go on from the last step taken, and a batch
    that fitted before fits again."""
    assert run("train", first, samples) == dict(refused=True, losses=True, weights=True)


@pytest.mark.parametrize("slots", [2, 64])
def test_neighbour_list_refused_room_to_grow(run, slots):
    rep = run("lists", slots)
    assert rep.pop("longest") > 4 and rep == dict(refused=[True, True], same=True), rep

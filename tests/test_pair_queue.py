"""The queue through which a CTA pair's scheduler hands claimed tasks to the roles of both CTAs (``csrc/mmoe_pair_queue.h``): every reader
gets every task, and no slot is overwritten before all reads of it are known to be over.  No GPU involved."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def queue(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ is not installed")
    exe = str(tmp_path_factory.mktemp("queue") / "pair_queue")
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-o", exe, os.path.join(ROOT, "tests", "pair_queue.cpp")], check=True)

    def run(tasks, epilogue, seed, scope="cluster"):
        out = subprocess.run([exe, str(tasks), str(epilogue), str(seed), scope], check=True, capture_output=True, text=True, timeout=120).stdout
        return tuple(int(v) for v in out.split())

    return run


@pytest.mark.parametrize("epilogue", [4, 8])
@pytest.mark.parametrize("tasks", [0, 1, 3, 4, 5, 8, 9, 60])
def test_every_role_reads_every_task_and_no_slot_is_overwritten_early(queue, tasks, epilogue):
    for seed in range(3):
        assert queue(tasks, epilogue, seed) == (0, 0, (2 * epilogue + 3) * (tasks + 1))       # the last number means "no more"


@pytest.mark.parametrize("epilogue", [4, 8])
def test_barriers_that_order_only_their_own_cta_are_found_to_race(queue, epilogue):
    """With everything that crosses the pair in CTA scope, the tasks arrive all the same, by latency; the order is nobody's promise."""
    races, wrong, _ = queue(9, epilogue, 0, "cta")
    assert races > 0 and wrong == 0

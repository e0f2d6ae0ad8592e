"""The steps of a single-GPU call as the C interface takes them (``csrc/mmoe_abi.cu``), with launches that fail.  No GPU involved."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ERR_CUDA = 3


@pytest.fixture(scope="module")
def forward(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not installed")
    exe = str(tmp_path_factory.mktemp("sequence") / "forward_sequence")
    subprocess.run([nvcc, "-std=c++17", "-Wno-deprecated-gpu-targets", "-o", exe, os.path.join(ROOT, "tests", "forward_sequence.cpp")],
                   check=True, capture_output=True)

    def run(tokens, layer_mask=0, engine=0, failing="none"):
        out = subprocess.run([exe, str(tokens), str(layer_mask), str(engine), failing], check=True, capture_output=True, text=True).stdout
        status, *steps = out.split()
        return int(status), steps

    return run


@pytest.mark.parametrize("m", [1, 16, 17, 192, 256, 3840])
def test_a_call_whose_combine_fails_leaves_no_claimed_tasks(forward, m):
    """The combine zeroes the counters of the launch of both GEMMs.  Where it is not launched, the call zeroes them some other way."""
    before = [] if m <= 16 else ["route"]
    assert forward(m) == (0, before + ["experts", "combine"])
    assert forward(m, failing="combine") == (ERR_CUDA, before + ["experts", "combine", "zero"])
    assert forward(m, failing="experts") == (ERR_CUDA, before + ["experts"])
    assert forward(m, layer_mask=1, failing="combine") == (ERR_CUDA, ["route", "experts", "combine"])
    assert forward(m, engine=1, failing="combine") == (ERR_CUDA, ["route", "experts", "combine"])

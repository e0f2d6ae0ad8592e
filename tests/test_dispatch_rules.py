"""The host-side rules that choose how a call is run (``csrc/mmoe_common.cuh``), compiled for the host and checked over
everything they accept.  No GPU involved."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NEVER = 0x7fffffff


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    """``rules("forms")`` -> the table's rows as tuples of integers."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not installed")
    exe = str(tmp_path_factory.mktemp("rules") / "dispatch_rules")
    subprocess.run([nvcc, "-std=c++17", "-Wno-deprecated-gpu-targets", "-o", exe, os.path.join(ROOT, "tests", "dispatch_rules.cpp")],
                   check=True, capture_output=True)

    def table(name):
        text = subprocess.run([exe, name], check=True, capture_output=True, text=True).stdout
        rows = [tuple(int(v) for v in line.split()[1:]) for line in text.splitlines()]
        assert rows
        return rows

    return table


def test_staged_tokens_replace_placed_rows_on_one_gpu_only(rules):
    """GEMM1 may multiply this rank's staged tokens only where every row is one of them: one rank, the routed tiles in the
    launch, no expert on the pair kernels, at most 16 tokens in pool blocks of 16."""
    for ranks, pair_above, select, peers, block_m, m, pairs, small, staged in rules("forms"):
        case = (ranks, pair_above, select, peers, block_m, m)
        want = ranks == 1 and select != 2 and pair_above != 0 and 1 <= m <= 16 and block_m == 16
        assert staged == want, case
        if staged:
            assert small and not pairs, case


def test_pair_launches_of_small_calls(rules):
    """No launch on CTA pairs where none can be worth it: one GPU with no more tokens than the line, several ranks with few
    routes (6 per token, 192 or 48 of 384 experts here) -- but a rank without tokens, or with the pair kernels forced on, keeps
    them.  The shared expert by itself takes one launch, by its own tokens."""
    for ranks, pair_above, select, peers, block_m, m, pairs, small, staged in rules("forms"):
        case = (ranks, pair_above, select, peers, block_m, m)
        if select == 2:
            assert (pairs, small) == ((1, 0) if m > pair_above else (0, 1) if m > 0 else (0, 0)), case
        elif pair_above == NEVER:
            assert (pairs, small) == (0, 1), case
        elif ranks == 1:
            assert (pairs, small) == (m > pair_above, pair_above > 0 or m == 0), case
        else:
            few = pair_above > 0 and 0 < 6 * m <= min(3072, 96 * (384 // ranks))
            assert (pairs, small) == (not few, pair_above > 0), case


def test_launch_parameters_are_kept_for_every_layer_of_a_model(rules):
    """Keys that take turns are built once as long as they fit, from the parameters of a key with the same workspace where
    there is one; a value that was handed out stays valid when its entry is replaced."""
    for keys, rounds, built, siblings, wrong in rules("cache"):
        assert wrong == 0
        assert built == (keys if keys <= 16 else rounds * keys), keys
        assert siblings == built - min(keys, 4), keys


# sizes of the structures that cross the C boundary, by the version of the interface: a change needs a new version
ABI_SIZES = {3: (32, 37 * 8, 80, 32), 4: (32, 38 * 8, 80, 32)}


def test_structures_of_the_c_interface_and_its_version(rules):
    import ctypes
    from vllm_plugin_b200.backend import _native
    (version, *sizes), = rules("abi")
    assert tuple(sizes) == ABI_SIZES[version]
    assert tuple(sizes) == tuple(ctypes.sizeof(s) for s in (_native.MmoeGeometry, _native.MmoeLayout, _native.MmoeWeights, _native.MmoeOptions))


def test_cuts_fit_their_tiles_and_scale_chunks(rules):
    """However many rows an expert has (more than there are tokens, when tokens name it twice or come from other ranks): its
    tiles cover them, are no larger than the kernels' tiles, and no more than the scale chunks reserved for its pool blocks."""
    for block_m, pairs, cap, n, parts, step, tiles, chunks in rules("cuts"):
        case = (block_m, pairs, cap, n)
        assert step % 16 == 0 and step <= (128 if pairs else cap) and parts * step >= n and tiles <= parts, case
        assert tiles <= chunks, case


def test_experts_just_past_one_pair_task(rules):
    """Above the line experts run on pairs, unless a second task would be nearly empty and the weights-as-A kernels take no more
    than four tiles of 80 rows, or three of 112, instead -- in the call's own tile size."""
    for pair_above, cap, n, on_pairs, tiles, tasks in rules("pairs"):
        case = (pair_above, cap, n)
        if pair_above != 192:
            assert on_pairs == (pair_above == 0), case
        elif n <= 192 or 256 < n <= (320 if cap == 80 else 336):
            assert not on_pairs and tiles <= (4 if cap == 80 else 3), case
        else:
            assert on_pairs, case


def test_what_a_call_rewrites_is_not_read_as_constant():
    """The GEMM launches run beside the launches that write their inputs: nothing in them goes through the read-only path."""
    for name in ("mmoe_umma.cu", "mmoe_umma_tm.cu", "mmoe_tc.cuh", "mmoe_common.cuh"):
        with open(os.path.join(ROOT, "vllm_plugin_b200", "csrc", name)) as f:
            assert "__ldg(p." not in f.read().replace("__ldg(x_sf", "__ldg(p."), name

"""Failure detection without faulting a GPU: a bounded device-side wait that nobody satisfies must run out, leave a
status record the host can read, and leave the context usable.  Here a two-rank geometry is driven by ONE process: the
"peer" workspace is a second local buffer, so the peer's arrival flag is never written."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


class _LoneRankOfTwo:
    def size(self):
        return 2

    def rank(self):
        return 0

    def barrier(self):
        return None


def test_peer_wait_times_out_and_reports_status():
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.workspace import SymmBuffer
    lib = _native.load()
    mine = SymmBuffer(_LoneRankOfTwo(), 16, 1920, 4, 512, 256, 1)          # plain device memory: no rendezvous happens
    other = torch.zeros(mine.layout.total_bytes, dtype=torch.int8, device="cuda")
    ids = torch.randint(0, 16, (8, 4), dtype=torch.int64, device="cuda")
    mine.topk_idx[:8].copy_(ids)
    stream = torch.cuda.current_stream().cuda_stream
    geo = ctypes.byref(mine.geo)
    _native.check(lib.mmoe_dispatch_count(geo, mine.base_ptr, 8, stream))
    peers = (ctypes.c_void_p * 2)(mine.base_ptr, other.data_ptr())
    opts = _native.MmoeOptions(10.0, 1, 0, 300, 0)                         # 300 ms budget for every device-side wait
    _native.check(lib.mmoe_ep_dispatch(geo, mine.base_ptr, peers, 8, ctypes.byref(opts), stream))
    words = (ctypes.c_int32 * 8)()
    code = lib.mmoe_read_status(geo, mine.base_ptr, words, stream)
    assert code == _native.MMOE_ERR_DEVICE_TIMEOUT
    assert words[0] == 1 and words[1] in (10, 11) and words[2] == 1       # barrier kernel, missing rank = 1
    with pytest.raises(RuntimeError, match="device-side wait expired"):
        _native.check(code)
    # the context is still healthy: an ordinary single-rank call right after works
    import helpers as H
    from helpers import O
    layer = H.make_layer(512, 256, 8, 2, True, seed=1)
    hid = O.make_hidden(5, 512, 1)
    rid, w = O.make_routing(5, 8, 2, 2)
    y, _ = H.run_layer(layer, hid, rid, w)
    assert O.parity_metrics(y.cpu(), H.oracle_layer(layer, hid, rid, w))["rel_l2"] <= 1e-3
    # reading the status cleared it: the buffer that timed out reports healthy again
    assert lib.mmoe_read_status(geo, mine.base_ptr, words, stream) == _native.MMOE_OK and words[0] == 0


def test_eager_calls_notice_a_bad_status_without_blocking():
    """The production path never calls ``read_status``: eager calls copy the status words to pinned memory behind the
    launch (here after every call) and a later call raises.  The condition used is an expert id >= num_experts, which the
    dispatch counts and treats as masked; after the report the buffer is healthy again."""
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend.workspace import SingleRankGroup
    import helpers as H
    from helpers import O
    layer = H.make_layer(512, 256, 8, 2, True, seed=3)
    l1, l2, sl1, sl2 = H.kernel_weights(layer, "cuda")
    buf = api.get_symm_buffer_for_mega_moe(SingleRankGroup(), 8, 1920, 2, 512, 256, 1)
    hid = O.make_hidden(6, 512, 1).cuda()
    ids, w = O.make_routing(6, 8, 2, 2)
    bad = ids.clone()
    bad[0, 0] = 99
    y = torch.empty((6, 512), dtype=torch.bfloat16, device="cuda")
    api.set_kernel_options(status_poll_interval=1)
    try:
        def call(which):
            api.stage_inputs_for_mega_moe(buf, hid, which.cuda(), w.cuda())
            api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, activation_clamp=10.0)
        call(bad)
        torch.cuda.synchronize()
        with pytest.raises(AssertionError, match="expert ids"):
            for _ in range(3):                 # the copy was queued behind the first call; one of the next calls sees it
                call(ids)
                torch.cuda.synchronize()
        for _ in range(3):                     # re-armed: healthy calls stay quiet
            call(ids)
            torch.cuda.synchronize()
        api.read_status(buf)
    finally:
        api.set_kernel_options(status_poll_interval=32)
    ref = H.oracle_layer(layer, hid.cpu(), ids, w)
    assert O.parity_metrics(y.cpu(), ref)["rel_l2"] <= 1e-3


def test_host_side_argument_errors_map_to_the_reference_exception_classes():
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend.workspace import SingleRankGroup
    import helpers as H
    layer = H.make_layer(512, 256, 8, 2, True, seed=2)
    l1, l2, sl1, sl2 = H.kernel_weights(layer, "cuda")
    buf = api.get_symm_buffer_for_mega_moe(SingleRankGroup(), 8, 1920, 2, 512, 256, 1)
    y = torch.empty((4, 512), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(AssertionError):
        api.fp8_fp4_mega_moe(y, l1, l2, buf, None, None)                  # buffer has a shared expert, none given
    with pytest.raises(AssertionError):
        api.fp8_fp4_mega_moe(y.float(), l1, l2, buf, sl1, sl2)            # y must be BF16
    with pytest.raises(AssertionError):
        api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, recipe=(1, 1, 128))
    with pytest.raises(NotImplementedError):
        api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, activation_alpha=1.702)
    with pytest.raises(AssertionError):
        api.fp8_fp4_mega_moe(y, (l1[0], l1[1].contiguous()), l2, buf, sl1, sl2)   # scales must be MN-major


@pytest.mark.parametrize("m", [8, 100, 300])
def test_an_error_left_by_an_earlier_call_is_not_taken_for_a_failed_launch(m):
    """Reading the status on a capturing stream is an error of the host, which the CUDA runtime remembers.  The layer call behind it
    neither reports that error as its own nor stops halfway, and so is the call behind that one right as well."""
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    import helpers as H
    from helpers import O
    layer = H.make_layer(512, 256, 8, 2, True, seed=4)
    l1, l2, sl1, sl2 = weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, 512, 1).cuda()
    ids, w = O.make_routing(m, 8, 2, 2)
    want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    assert O.parity_metrics(want.cpu(), H.oracle_layer(layer, hid.cpu(), ids, w))["rel_l2"] <= 1e-3
    lib, rt = _native.load(), ctypes.CDLL("libcudart.so.12")
    side, graph, words = torch.cuda.Stream(), ctypes.c_void_p(), (ctypes.c_int32 * 8)()
    api.stage_inputs_for_mega_moe(buf, hid, ids.cuda(), w.cuda())
    assert rt.cudaStreamBeginCapture(ctypes.c_void_p(side.cuda_stream), 2) == 0                # 2: relaxed
    assert lib.mmoe_read_status(ctypes.byref(buf.geo), buf.base_ptr, words, side.cuda_stream) == _native.MMOE_ERR_CUDA
    rt.cudaStreamEndCapture(ctypes.c_void_p(side.cuda_stream), ctypes.byref(graph))
    rt.cudaGetLastError()                                                                      # this copy of the runtime, not the library's
    for _ in range(2):
        y = torch.zeros_like(want)
        api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, activation_clamp=10.0)
        api.read_status(buf)
        assert torch.equal(y, want)


@pytest.mark.parametrize("hidden,inter,m,missing", [(512, 256, 8, "routed"), (512, 256, 8, "shared"), (512, 256, 100, "routed"),
                                                    (2560, 1152, 16, "shared"), (2560, 1152, 150, "routed"), (2560, 1152, 300, "routed"),
                                                    (512, 256, 160, "restarted"), (2560, 1152, 160, "restarted")])
def test_rows_that_never_become_complete_and_the_call_behind(hidden, inter, m, missing):
    """GEMM2 waits for a count of GEMM1's finished parts.  Here the count of one expert starts far below zero, as if parts of it were
    lost: its GEMM2 tasks give up, every other task of the call is done, and the next call on the buffer is right.  "restarted": a skewed call,
    whose CTAs have started over with larger token slots."""
    import time
    from vllm_plugin_b200 import api
    import helpers as H
    from helpers import O
    e, k = 8, 3
    layer = H.make_layer(hidden, inter, e, k, True, seed=5)
    weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, hidden, 1)
    ids, w = O.make_routing(m, e, k, 2)
    if missing == "restarted":
        ids[:] = torch.tensor([6, 1, 4])
        api.set_kernel_options(block_m=16)
    want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    rows = buf.ret[:m * k].clone()
    assert O.parity_metrics(want.cpu(), H.oracle_layer(layer, hid, ids, w))["rel_l2"] <= 1e-3
    assert buf.plan_words[7] == 80 or missing != "restarted"
    lost = e if missing == "shared" else int(ids[0, 0])
    done = buf._view(buf.layout.plan, (16 + 5 * e + 4 + e + 1,), torch.int32)[16 + 5 * e + 4:]
    api.set_kernel_options(timeout_ms=200)
    try:
        for _ in range(2):
            buf.ret.zero_()
            done[lost] = buf.plan_words[13] = -2 ** 30                    # 13: all experts' parts
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            with pytest.raises(RuntimeError, match="device wait expired: kernel 4"):
                H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
            assert 0.15 < time.perf_counter() - t0 < 2.0
            assert buf.plan_words[9:14].cpu().tolist() == [0] * 5 and not done.any()
            pos = buf.route_pos[:m].cpu().long()
            for x in range(e):
                if x != lost and bool((ids == x).any()):
                    assert torch.equal(buf.ret[pos[ids == x].cuda()], rows[pos[ids == x].cuda()]), x
            for _ in range(2):
                y, _ = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
                assert torch.equal(y, want)
    finally:
        api.set_kernel_options(timeout_ms=2000, block_m=0)


@pytest.mark.parametrize("missing", ["routed", "shared"])
def test_pairs_that_wait_for_lost_rows_and_the_call_behind(missing):
    """The same where the experts run on CTA pairs, whose GEMM2 starts behind GEMM1's finished parts as SMs come free."""
    from vllm_plugin_b200 import api
    import helpers as H
    from helpers import O
    e, k, m, hidden, inter = 4, 2, 1000, 512, 256
    layer = H.make_layer(hidden, inter, e, k, True, seed=6)
    weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, hidden, 1)
    ids, w = O.make_routing(m, e, k, 2)
    want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    assert O.parity_metrics(want.cpu(), H.oracle_layer(layer, hid, ids, w))["rel_l2"] <= 1e-3
    assert buf.plan_words[6] == 0                                         # every expert on pairs
    done = buf._view(buf.layout.plan, (16 + 5 * e + 4 + e + 3,), torch.int32)[16 + 5 * e + 4:]      # and the claimed tasks behind it
    api.set_kernel_options(timeout_ms=200)
    try:
        for _ in range(2):
            done[e if missing == "shared" else 1] = -2 ** 30
            with pytest.raises(RuntimeError, match="device wait expired: kernel 22"):
                H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
            assert not done.any()
            for _ in range(2):
                y, _ = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
                assert torch.equal(y, want)
    finally:
        api.set_kernel_options(timeout_ms=2000)


@pytest.mark.parametrize("missing", ["routed", "shared"])
def test_pairs_with_several_tasks_each_and_lost_rows(missing):
    """Five and more tasks per pair and layer, so that every slot of a pair's queue is used again, with roles that stop at different places
    of it.  Only what was lost is missing, the wait ends near its limit, and the calls behind are right."""
    import time
    from vllm_plugin_b200 import api
    import helpers as H
    from helpers import O
    e, k, m, hidden, inter = 12, 6, 1500, 2560, 1152
    layer = H.make_layer(hidden, inter, e, k, True, seed=8)
    weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, hidden, 1)
    ids, w = O.make_routing(m, e, k, 2)
    want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    shared_out = buf._view(buf.layout.shared_out, (m, hidden), torch.bfloat16)
    rows, shared_rows = buf.ret[:m * k].clone(), shared_out.clone()
    sample = torch.arange(0, m, 25)
    assert O.parity_metrics(want.cpu()[sample], H.oracle_layer(layer, hid[sample], ids[sample], w[sample]))["rel_l2"] <= 1e-3
    assert buf.plan_words[6] == 0                                         # every expert on pairs
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    tiles = (int(buf.plan_words[0]) + int(buf.plan_words[1])) // 2
    assert tiles * (2 * inter // 256) >= 5 * pairs and tiles * (hidden // 256) >= 5 * pairs
    lost = e if missing == "shared" else int(ids[0, 0])
    done = buf._view(buf.layout.plan, (16 + 6 * e + 8,), torch.int32)[16 + 5 * e + 4:]              # and what lies behind it
    api.set_kernel_options(timeout_ms=200)
    try:
        for _ in range(2):
            buf.ret.zero_()
            shared_out.zero_()
            done[lost] = -2 ** 30
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            with pytest.raises(RuntimeError, match="device wait expired: kernel 22"):
                H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
            assert 0.15 < time.perf_counter() - t0 < 2.0
            assert not done.any()
            pos = buf.route_pos[:m].cpu().long()
            for x in range(e):
                if x != lost:
                    assert torch.equal(buf.ret[pos[ids == x].cuda()], rows[pos[ids == x].cuda()]), x
            assert torch.equal(shared_out, shared_rows) == (missing != "shared")
            for _ in range(2):
                y, _ = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
                assert torch.equal(y, want)
    finally:
        api.set_kernel_options(timeout_ms=2000)


@pytest.fixture(scope="module")
def run_wait(tmp_path_factory):
    import os
    import shutil
    import subprocess
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not installed")
    so = str(tmp_path_factory.mktemp("waits") / "waits.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(os.path.dirname(__file__), "waits.cu")], check=True, capture_output=True)
    fn = ctypes.CDLL(so).run_wait
    fn.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p, ctypes.c_void_p]
    return fn


@pytest.mark.parametrize("which,name", list(enumerate(["the plan", "a task, whole warp", "a task, one lane polls", "a free slot for a task"])))
def test_every_other_wait_of_the_launch_of_both_gemms_gives_up(run_wait, which, name):
    """The waits that a call cannot be made to lose from outside, each in a kernel of one warp: for the plan of a launch that orders the
    routes itself, for the scheduler's next task, and the scheduler's own for a free slot."""
    plan, status, out = (torch.zeros(n, dtype=torch.int32, device="cuda") for n in (4096, 8, 1))
    stream = torch.cuda.current_stream().cuda_stream
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    assert run_wait(which, plan.data_ptr(), 8, status.data_ptr(), 100_000_000, out.data_ptr(), stream) == 0
    end.record()
    torch.cuda.synchronize()
    assert out.item() == 1 and status.tolist()[:4] == [1, 4, 10 + which, 0]
    assert 90 < start.elapsed_time(end) < 1000
    if which == 0:                                 # ... and ends at once where the flag is set
        plan[10] = 1
        assert run_wait(which, plan.data_ptr(), 8, status.data_ptr(), 100_000_000, out.data_ptr(), stream) == 0
        assert out.item() == 2

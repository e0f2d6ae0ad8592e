"""Expert parallelism on real GPUs: one process per GPU over NCCL (NVLS off), each rank checked against the oracle.
Skipped on machines with fewer GPUs than ranks."""

import pytest
import torch

from ep_harness import layer_body, run_ranks

pytestmark = pytest.mark.gpu


def _need(n):
    if torch.cuda.device_count() < n:
        pytest.skip(f"needs {n} GPUs")


SMALL = dict(hidden=512, inter=256, num_experts=16, num_topk=4, shared=True)


def test_redundant_physical_experts_under_cuda_graph():
    """Load-balancer geometry: 12 logical + 4 redundant physical experts over 2 ranks, decode-sized calls replayed from
    a CUDA graph."""
    _need(2)
    run_ranks(2, "nccl", layer_body, SMALL, (16, 64), 5, dict(zipf_s=1.2), 1920, "peer", True, 4, timeout=240)


@pytest.mark.parametrize("world,tokens,kw,transport,graph", [
    (2, (70, 33), dict(zipf_s=1.2, mask_frac=0.05, hot=2), "peer", False),
    (2, (70, 33), dict(zipf_s=1.2, mask_frac=0.05, hot=2), "peer-unfused", False),
    (2, (70, 33), dict(zipf_s=1.2, mask_frac=0.05, hot=2), "nccl", False),
    (2, (1, 0), {}, "peer", False),
    (2, (40, 130), dict(zipf_s=1.2, mask_frac=0.05), "peer", True),
    (4, (130, 64, 7, 300), dict(zipf_s=1.2, mask_frac=0.05), "peer", False),
])
def test_layer_matches_oracle_at_ep(world, tokens, kw, transport, graph):
    """Per-rank output against the oracle, receive counts / block offsets / statistics bit-exact; with the device-side
    peer exchange (write-back fused into GEMM2, checked bit-identical to the separate copy kernel; also replayed from a
    CUDA graph) and with the host-driven NCCL exchange."""
    _need(world)
    run_ranks(world, "nccl", layer_body, SMALL, tokens, 3, kw, 1920, transport, graph, timeout=240)


@pytest.mark.parametrize("world", [2, 8])
def test_draft_model_split_top3(world):
    """Configuration 2 of the benchmark at reduced H / I: E=128, top-3 (16 experts per rank at EP8), capacity 3840 per
    rank, prefill- and decode-sized calls on different ranks (including a rank without tokens)."""
    _need(world)
    geometry = dict(hidden=512, inter=256, num_experts=128, num_topk=3, shared=True)
    tokens = (300, 1, 32, 7, 130, 64, 0, 255)[:world]
    run_ranks(world, "nccl", layer_body, geometry, tokens, 9, dict(zipf_s=1.2, mask_frac=0.05, hot=2), 3840, "peer", False,
              timeout=300)
    run_ranks(world, "nccl", layer_body, geometry, (32,) * world, 10, {}, 3840, "peer", True, timeout=300)


@pytest.mark.parametrize("world", [1, 2, 8])
def test_redundant_experts_graphs_and_reload_under_a_reshuffled_map(world):
    """Configuration 4 of the benchmark at reduced H / I: 392 physical experts (384 + copies of the 8 hottest), top-6,
    decode-sized calls captured and replayed as CUDA graphs, weights reloaded in place under a reshuffled placement,
    graphs replayed again: bit-identical outputs, oracle parity and bit-exact counts both times."""
    _need(world)
    from ep_harness import eplb_body
    run_ranks(world, "nccl", eplb_body, (1, 4, 16, 64, 256), 17, timeout=420)


class _RankOf:
    def __init__(self, rank, world):
        self._rank, self._world = rank, world

    def size(self):
        return self._world

    def rank(self):
        return self._rank

    def barrier(self):
        return None


def run_ranks_in_turn(layer, hids, ids, ws, orientation=0):
    """Every rank's steps of the host-driven exchange on one GPU, one after the other (no kernel waits for another rank);
    the all-to-alls are copies between the ranks' workspaces.  Returns the ranks' outputs and buffers."""
    import ctypes
    import helpers as H
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.frontend import _weights_struct, check_mega_moe_arguments, read_status
    from vllm_plugin_b200.backend.workspace import SymmBuffer
    world, e_l = len(hids), layer.num_experts // len(hids)
    lib, stream = _native.load(), torch.cuda.current_stream().cuda_stream
    opts = _native.MmoeOptions(10.0, 1, 0, 2000, 0)
    api.precompile_mega_moe_variants(world, layer.num_experts, 1920, layer.num_topk, layer.hidden, layer.inter, 1)
    api.set_kernel_options(orientation=orientation)
    try:
        ranks = []
        for r in range(world):
            with pytest.warns(UserWarning, match="symmetric memory"):
                buf = SymmBuffer(_RankOf(r, world), layer.num_experts, 1920, layer.num_topk, layer.hidden, layer.inter, 1)
            l1, l2, s1, s2 = H.kernel_weights(layer, "cuda", r * e_l, (r + 1) * e_l)
            m = hids[r].shape[0]
            y = torch.empty((m, layer.hidden), dtype=torch.bfloat16, device="cuda")
            strides = check_mega_moe_arguments(y, l1, l2, buf, s1, s2, None, (1, 1, 32), "swiglu", 10.0, True, 1.0, 0.0)
            geo, base = ctypes.byref(buf.geo), buf.base_ptr
            bm = api.stage_inputs_for_mega_moe(buf, hids[r].cuda(), ids[r].cuda(), ws[r].cuda())
            _native.check(lib.mmoe_dispatch_count(geo, base, m, stream))
            _native.check(lib.mmoe_dispatch_pack(geo, base, m, stream))
            ranks.append((buf, geo, base, bm, m, y, _weights_struct(l1, l2, s1, s2, *strides), (l1, l2, s1, s2)))
        counts = [buf.send_count.view(world, e_l).cpu() for buf, *_ in ranks]            # [source][destination, expert]
        rows = [[int(counts[s][d].sum()) for d in range(world)] for s in range(world)]
        for d, (buf, geo, base, bm, m, y, wstruct, _) in enumerate(ranks):
            at = 0
            for s, (src, *_) in enumerate(ranks):
                buf.recv_count[s].copy_(counts[s][d])
                lo, n = sum(rows[s][:d]), rows[s][d]
                for name in ("x", "sf", "w"):
                    to, frm = getattr(buf, "recv_" + name)[at:at + n], getattr(src, "send_" + name)[lo:lo + n]
                    to.view(torch.uint8).copy_(frm.view(torch.uint8))
                at += n
            _native.check(lib.mmoe_dispatch_place(geo, base, m, bm, None, stream))
            _native.check(lib.mmoe_experts(geo, base, ctypes.byref(wstruct), ctypes.byref(opts), m, bm, stream))
        for s, (src, geo, base, bm, m, y, *_) in enumerate(ranks):
            for d, (buf, *_) in enumerate(ranks):
                at, lo, n = sum(rows[x][d] for x in range(s)), sum(rows[s][:d]), rows[s][d]
                src.ret_recv[lo:lo + n].copy_(buf.ret[at:at + n])
            _native.check(lib.mmoe_combine(geo, base, y.data_ptr(), m, stream))
            read_status(src)
        return [r[5] for r in ranks], [r[0] for r in ranks]
    finally:
        api.set_kernel_options(orientation=0)


@pytest.mark.parametrize("orientation", [0, 1])
@pytest.mark.parametrize("tokens", [(5, 9), (16, 1), (0, 12), (17, 16), (3, 400), (120, 500), (16, 2, 7, 1)])
def test_ranks_in_turn_match_the_oracle(tokens, orientation):
    """The layer's kernels at EP 2 and 4 without the transport: per rank a handful of tokens of its own, and rows of other
    ranks that it has never staged."""
    import helpers as H
    from helpers import O
    from test_gpu_layer import assert_parity
    layer = H.make_layer(512, 256, 16, 4, True, seed=4)
    hids = [O.make_hidden(m, 512, 10 + r) for r, m in enumerate(tokens)]
    routing = [O.make_routing(m, 16, 4, 20 + r, zipf_s=1.2, mask_frac=0.05) for r, m in enumerate(tokens)]
    ids, ws = [a for a, _ in routing], [b for _, b in routing]
    ys, _ = run_ranks_in_turn(layer, hids, ids, ws, orientation)
    want = O.moe_layer(hids, ids, ws, layer.experts, layer.shared, 10.0, None)
    for r, m in enumerate(tokens):
        if m > 0:
            assert_parity(ys[r], want[r], f"rank {r} of {tokens}, orientation {orientation}")

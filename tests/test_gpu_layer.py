"""GPU parity of the whole layer against the CPU oracle on identical seeded inputs, through the package's public API
(which calls the C ABI).  Tolerance of the BF16 output: relative L2 <= 1e-3 and max_abs <= 2e-2; one BF16 ulp of the
reference is larger than 2e-2 wherever |y| >= 4, and a one-ulp disagreement is inherent to the FP32 summation order, so
the element-wise bound is max(2e-2, one BF16 ulp of the reference value)."""

import pytest
import torch

import helpers as H
from helpers import O

pytestmark = pytest.mark.gpu

REL_L2 = 1e-3
MAX_ABS = 2e-2


def assert_parity(y, ref, what=""):
    a, b = y.float().cpu(), ref.float()
    assert torch.isfinite(a).all(), what
    rel = float((a - b).norm() / b.norm().clamp(min=1e-30))
    ulp = torch.pow(2.0, torch.floor(torch.log2(b.abs().clamp(min=2.0 ** -126))) - 7)
    bound = torch.clamp(ulp, min=MAX_ABS)
    worst = float(((a - b).abs() - bound).max())
    assert rel <= REL_L2, f"{what}: rel_l2 {rel}"
    assert worst <= 0, f"{what}: an element exceeds max(2e-2, 1 ulp) by {worst}"


SMALL = dict(hidden=512, inter=256, num_experts=8, num_topk=2)


@pytest.mark.parametrize("engine", [0, 1])
@pytest.mark.parametrize("m", [1, 5, 33, 130])
@pytest.mark.parametrize("shared", [True, False])
def test_small_layer_matches_oracle(engine, m, shared):
    layer = H.make_layer(shared=shared, seed=m, **SMALL)
    hid = O.make_hidden(m, layer.hidden, 1)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 2, mask_frac=0.1 if m > 1 else 0.0)
    y, buf = H.run_layer(layer, hid, ids, w, engine=engine)
    assert_parity(y, H.oracle_layer(layer, hid, ids, w), f"engine {engine} m {m}")
    # the dispatch tables of the call (M <= 128 takes the fused single-launch route/plan kernel) against the oracle
    hdr, total, block_off = buf.plan_tables()
    plan = O.dispatch_plan([ids], layer.num_experts, 0, hdr["block_m"])
    assert torch.equal(buf.send_count.cpu().long(), plan.recv_total) and torch.equal(total.long(), plan.recv_total)
    assert torch.equal(block_off.long(), plan.pool_block_offset)
    pos = buf.route_pos[:m].cpu()
    dst = buf.pool_dst.cpu()
    inv = {int(pos[t, s]): (t, s) for t in range(m) for s in range(layer.num_topk) if int(pos[t, s]) >= 0}
    for ex in range(layer.num_experts):
        base = int(block_off[ex]) * hdr["block_m"]
        assert [inv[int(dst[base + j])] for j in range(int(total[ex]))] == [(t, s) for (_, t, s) in plan.routes[ex]]


@pytest.mark.parametrize("bm", [16, 32, 64, 128, 192, 240])
def test_every_block_m_variant(bm):
    """Forced BLOCK_M with ~150 tokens per expert (Zipf: some experts far more): several pool blocks per expert,
    partially filled last blocks, and experts whose rows are cut into two or more equal tensor-core tiles that do not
    follow the block boundaries."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(shared=True, seed=3, **SMALL)
    m = 600
    hid = O.make_hidden(m, layer.hidden, 4)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 5, zipf_s=1.2)
    api.set_kernel_options(block_m=bm)
    try:
        y, buf = H.run_layer(layer, hid, ids, w)
        assert buf.plan_tables()[0]["block_m"] == bm
    finally:
        api.set_kernel_options(block_m=0)
    assert_parity(y, H.oracle_layer(layer, hid, ids, w), f"block_m {bm}")


@pytest.mark.parametrize("geom", [dict(hidden=512, inter=256, num_experts=8, num_topk=2),
                                  dict(hidden=1024, inter=384, num_experts=4, num_topk=2)])
@pytest.mark.parametrize("bm", [16, 64, 128, 192, 240])
def test_tokens_as_a_kernels_every_block_m(geom, bm):
    """The CTA-pair kernels forced on (they otherwise get the experts with many rows): tiles of up to 128 rows under every
    BLOCK_M pool layout, 256-row weight blocks of which each CTA of the pair loads half, an empty second tile where an expert's
    rows fit the first, scale chunks of blocks that a tile does not follow, the shared expert's tiles, masked routes and experts
    without tokens.  Against the oracle, and against the weights-as-A kernels on the same inputs."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(shared=True, seed=21, **geom)
    m = 600
    hid = O.make_hidden(m, layer.hidden, 4)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 5, zipf_s=1.2, mask_frac=0.05)
    ids[ids == 1] = -1                                      # an expert that receives nothing
    api.set_kernel_options(block_m=bm)
    try:
        y_tm, buf = H.run_layer(layer, hid, ids, w, orientation=2)
        assert buf.plan_tables()[0]["block_m"] == bm
        y_sa, _ = H.run_layer(layer, hid, ids, w, orientation=1)
    finally:
        api.set_kernel_options(block_m=0)
    ref = H.oracle_layer(layer, hid, ids, w)
    assert_parity(y_tm, ref, f"tokens-as-A block_m {bm}")
    assert_parity(y_sa, ref, f"weights-as-A block_m {bm}")
    diff = (y_tm.float() - y_sa.float()).abs().max().item()
    assert diff <= 2e-2, f"the two kernel families differ by {diff}"


@pytest.mark.parametrize("orientation", [2, 3])
@pytest.mark.parametrize("m", [1, 40, 129, 700])
def test_tokens_as_a_kernels_token_counts_and_options(m, orientation):
    """Forced pair kernels (2 and 3 name the same form) over small and ragged token counts (tiles of 1..128 rows, token boxes of
    32 to 128 rows), with the two-slice weight form, without clamp, and with the IEEE sigmoid."""
    layer = H.make_layer(shared=True, seed=23, hidden=1024, inter=512, num_experts=4, num_topk=2)
    hid = (O.make_hidden(m, layer.hidden, 1).float() * 3).to(torch.bfloat16)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 2, mask_frac=0.1 if m > 1 else 0.0)
    for clamp, fast, localized in ((10.0, True, False), (None, False, True)):
        y, _ = H.run_layer(layer, hid, ids, w, clamp=clamp, fast_math=fast, localized=localized, orientation=orientation)
        assert_parity(y, H.oracle_layer(layer, hid, ids, w, clamp=clamp), f"m {m} clamp {clamp} fast {fast}")


def test_options_fast_math_clamp_and_localized_weights():
    layer = H.make_layer(shared=True, seed=9, **SMALL)
    hid = (O.make_hidden(40, layer.hidden, 1).float() * 6).to(torch.bfloat16)       # large activations: the clamp bites
    ids, w = O.make_routing(40, layer.num_experts, layer.num_topk, 2)
    for clamp in (10.0, 0.5, None):
        ref = H.oracle_layer(layer, hid, ids, w, clamp=clamp)
        for fast in (True, False):
            y, _ = H.run_layer(layer, hid, ids, w, clamp=clamp, fast_math=fast)
            assert_parity(y, ref, f"clamp {clamp} fast_math {fast}")
    y0, _ = H.run_layer(layer, hid, ids, w)
    y1, _ = H.run_layer(layer, hid, ids, w, localized=True)                         # two-slice routed weights
    assert torch.equal(y0, y1)


@pytest.mark.parametrize("hidden", [256, 512, 768, 1280])
@pytest.mark.parametrize("m", [3, 60, 260])
def test_two_slice_weights_of_any_hidden_size(hidden, m):
    """Slices of W2 with an odd number of 128-row blocks: a task of 256 rows reaches from one slice into the other."""
    layer = H.make_layer(hidden, 256, 4, 2, True, seed=10)
    hid = O.make_hidden(m, hidden, 1)
    ids, w = O.make_routing(m, 4, 2, 2)
    y0, _ = H.run_layer(layer, hid, ids, w)
    y1, _ = H.run_layer(layer, hid, ids, w, localized=True)
    assert torch.equal(y0, y1)
    assert_parity(y0, H.oracle_layer(layer, hid, ids, w), f"hidden {hidden} m {m}")


def test_masked_tokens_padding_and_empty_call():
    layer = H.make_layer(shared=False, seed=11, **SMALL)
    m = 20
    hid = O.make_hidden(m, layer.hidden, 1)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 2)
    pad = torch.zeros(m, dtype=torch.bool)
    pad[[0, 7, 19]] = True
    y, _ = H.run_layer(layer, hid, ids, w, pad=pad)
    ref = H.oracle_layer(layer, hid, ids, w, pad=pad)
    assert_parity(y, ref, "padding")
    assert float(y[pad.cuda()].float().abs().max()) == 0.0          # no valid slot and no shared expert: exact zeros
    y_empty, _ = H.run_layer(layer, hid[:0], ids[:0], w[:0])
    assert y_empty.shape == (0, layer.hidden)


@pytest.mark.parametrize("m", [1, 40, 300])
def test_residual_added_in_the_combine_pass(m):
    """``residual=`` gives bit for bit what a separate BF16 addition after the layer gives, also in place (residual is y),
    at decode and prefill sizes (chained small-call path and the two-stream path)."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(shared=True, seed=12, **SMALL)
    hid = O.make_hidden(m, layer.hidden, 5)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 6, mask_frac=0.1)
    y, buf = H.run_layer(layer, hid, ids, w)
    dev = y.device
    res = (torch.randn(m, layer.hidden, generator=torch.Generator().manual_seed(3)) * 2).to(torch.bfloat16).to(dev)
    want = y + res                                           # the engine's own addition
    l1, l2, sl1, sl2 = H.kernel_weights(layer, dev)
    out = torch.empty_like(y)
    api.stage_inputs_for_mega_moe(buf, hid.to(dev), ids.to(dev), w.to(dev))
    api.fp8_fp4_mega_moe(out, l1, l2, buf, sl1, sl2, activation_clamp=10.0, residual=res)
    assert torch.equal(out, want)
    inplace = res.clone()
    api.fp8_fp4_mega_moe(inplace, l1, l2, buf, sl1, sl2, activation_clamp=10.0, residual=inplace)
    assert torch.equal(inplace, want)
    api.fp8_fp4_mega_moe(out, l1, l2, buf, sl1, sl2, activation_clamp=10.0)        # and none again: the plain output
    assert torch.equal(out, y)
    with pytest.raises(AssertionError):
        api.fp8_fp4_mega_moe(out, l1, l2, buf, sl1, sl2, activation_clamp=10.0, residual=res.float())


def test_outputs_do_not_depend_on_batch_composition():
    """Size-independent property: a token's output is bit-identical whatever other tokens share the call (columns of the
    tensor-core tiles are independent and the K order is fixed)."""
    layer = H.make_layer(shared=True, seed=13, **SMALL)
    m = 300
    hid = O.make_hidden(m, layer.hidden, 1)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 2)
    y, _ = H.run_layer(layer, hid, ids, w)
    perm = torch.randperm(m, generator=torch.Generator().manual_seed(0))
    y_perm, _ = H.run_layer(layer, hid[perm], ids[perm], w[perm])
    assert torch.equal(y_perm.cpu(), y.cpu()[perm])
    y_head, _ = H.run_layer(layer, hid[:17], ids[:17], w[:17])
    assert torch.equal(y_head.cpu(), y.cpu()[:17])


def test_reference_cpu_configuration():
    """The CPU-runnable configuration of the benchmark: H=5120, I=2304, E=32, top-6, one shared expert, M=128, seed 0."""
    layer = H.make_layer(5120, 2304, 32, 6, True, seed=0)
    hid = O.make_hidden(128, 5120, 0)
    ids, w = O.make_routing(128, 32, 6, 0)
    y, buf = H.run_layer(layer, hid, ids, w)
    assert buf.plan_tables()[0]["block_m"] == 32
    ref = H.oracle_layer(layer, hid, ids, w)
    H.log_parity("config 0: E=32 M=128", H.strict_metrics(y, ref))
    assert_parity(y, ref, "config 0")


def test_full_size_engines_agree_and_permutation_invariance():
    """E=384 resident experts (7.2 GB of packed weights generated on the GPU), M=256 decode-side point: the tensor-core
    kernels against the scalar validation kernels on the same pool, per-expert counts against the routing, and the
    batch-composition property at full size."""
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend.workspace import SingleRankGroup
    from vllm_plugin_b200.backend.frontend import _use_scalar_validation_kernels
    from vllm_plugin_b200.testing import SyntheticLayer, make_hidden, make_routing
    e, k, h, i, m = 384, 6, 5120, 2304, 256
    syn = SyntheticLayer(h, i, e, True, "cuda", seed=1)
    buf = api.get_symm_buffer_for_mega_moe(SingleRankGroup(), e, 3840, k, h, i, 1)
    hid = make_hidden(m, h, 1, "cuda")
    ids, w = make_routing(m, e, k, 2, "cuda")
    stats = torch.zeros(e, dtype=torch.int32, device="cuda")

    def run(hh, ii, ww, engine, st=None):
        y = torch.empty((hh.shape[0], h), dtype=torch.bfloat16, device="cuda")
        _use_scalar_validation_kernels(engine == 1)
        try:
            api.stage_inputs_for_mega_moe(buf, hh, ii, ww)
            api.fp8_fp4_mega_moe(y, syn.l1, syn.l2, buf, syn.shared_l1, syn.shared_l2,
                                 cumulative_local_expert_recv_stats=st, activation_clamp=10.0)
        finally:
            _use_scalar_validation_kernels(False)
        from vllm_plugin_b200.backend.frontend import read_status
        read_status(buf)
        return y

    y_tc = run(hid, ids, w, 0, stats)
    y_sc = run(hid, ids, w, 1)
    assert torch.equal(stats.cpu().long(), torch.bincount(ids.cpu().flatten(), minlength=e))
    assert_parity(y_tc, y_sc.cpu(), "tensor-core vs scalar engine, E=384")
    perm = torch.randperm(m, generator=torch.Generator().manual_seed(1)).cuda()
    assert torch.equal(run(hid[perm], ids[perm], w[perm], 0), y_tc[perm])


def test_layer_class_loads_a_checkpoint_and_runs(monkeypatch):
    """The plugin layer class end to end: checkpoint shards (w1 / w3 / w2 + scales) through ``weight_loader`` into the
    two-slice parameters, ``forward`` through the real backend, reload in place, output against the oracle."""
    from types import SimpleNamespace
    from vllm_plugin_b200 import _standin, api
    from vllm_plugin_b200.experts import make_experts_class

    layer_def = H.make_layer(shared=True, seed=21, **SMALL)
    h, i, e, k = layer_def.hidden, layer_def.inter, layer_def.num_experts, layer_def.num_topk
    backend = SimpleNamespace(**{name: getattr(api, name) for name in api.__all__ if name != "SymmBuffer"})
    backend.get_unsupported_reason_for_mega_moe = (
        lambda *a, **kw: api.get_unsupported_reason_for_mega_moe(*a, **{**kw, "allow_unvalidated": True}))
    cls = make_experts_class(_standin.DeepGemmMegaMoEExperts, _standin.get_ep_group, _standin.MEGA_MOE_MXFP4)
    monkeypatch.setattr(cls, "_import_backend", staticmethod(lambda: backend))
    cfg = SimpleNamespace(parallel_config=SimpleNamespace(enable_eplb=False),
                          scheduler_config=SimpleNamespace(max_num_batched_tokens=256))
    sh = layer_def.shared
    shared_mlp = SimpleNamespace(
        gate_up_proj=SimpleNamespace(weight=sh.w13.cuda(), weight_scale=sh.w13_sf.cuda()),
        down_proj=SimpleNamespace(weight=sh.w2.cuda(), weight_scale=sh.w2_sf.cuda()))
    mod = cls(cfg, prefix="model.layers.0.experts", num_experts=e, num_local_experts=e, experts_start_idx=0, top_k=k,
              hidden_size=h, intermediate_size=i, weight_format=_standin.MEGA_MOE_MXFP4,
              activation=_standin.MegaMoEActivation(clamp=10.0), shared_experts=shared_mlp, device="cuda")
    ptrs = [p.data_ptr() for p in mod.parameters()]

    def load(experts):
        for ex, ew in enumerate(experts):
            for shard, w, s in (("w1", ew.w13[:i], ew.w13_sf[:i]), ("w3", ew.w13[i:], ew.w13_sf[i:]), ("w2", ew.w2, ew.w2_sf)):
                prefix = "w2" if shard == "w2" else "w13"
                assert mod.weight_loader(getattr(mod, f"{prefix}_weight"), w.cuda(), f"experts.{prefix}_weight", shard, ex, True)
                assert mod.weight_loader(getattr(mod, f"{prefix}_weight_scale"), s.cuda(), f"experts.{prefix}_weight_scale", shard, ex, True)

    load(layer_def.experts)
    m = 50
    hid = O.make_hidden(m, h, 1)
    ids, w = O.make_routing(m, e, k, 2)
    y = mod(hid.cuda(), w.cuda(), ids.cuda())
    assert_parity(y, H.oracle_layer(layer_def, hid, ids, w), "layer class")
    # reload other weights into the same parameters: addresses unchanged, outputs follow the new weights
    layer2 = H.make_layer(shared=True, seed=22, **SMALL)
    layer2.shared = layer_def.shared
    load(layer2.experts)
    assert [p.data_ptr() for p in mod.parameters()] == ptrs
    y2 = mod(hid.cuda(), w.cuda(), ids.cuda())
    assert_parity(y2, H.oracle_layer(layer2, hid, ids, w), "layer class after reload")


def test_cuda_graph_replay_of_every_variant():
    """Every BLOCK_M variant is prepared before capture; a captured call replays bit-identically and follows new inputs
    staged into the same buffers."""
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend.workspace import SingleRankGroup
    layer = H.make_layer(shared=True, seed=31, **SMALL)
    dev = torch.device("cuda", 0)
    l1, l2, sl1, sl2 = H.kernel_weights(layer, dev)
    buf = api.get_symm_buffer_for_mega_moe(SingleRankGroup(), layer.num_experts, 1920, layer.num_topk, layer.hidden, layer.inter, 1)
    variants = api.precompile_mega_moe_variants(1, layer.num_experts, 1920, layer.num_topk, layer.hidden, layer.inter, 1)
    assert variants == (16, 32, 64, 128, 192, 240)
    for m in (1, 40, 130, 700, 1900):
        hid_a, hid_b = O.make_hidden(m, layer.hidden, m), O.make_hidden(m, layer.hidden, m + 1)
        ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, m)
        x = hid_a.cuda()
        ids_d, w_d = ids.cuda(), w.cuda()
        y = torch.empty((m, layer.hidden), dtype=torch.bfloat16, device=dev)

        def call():
            api.stage_inputs_for_mega_moe(buf, x, ids_d, w_d)
            api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, activation_clamp=10.0)

        call()
        eager = y.clone()
        side = torch.cuda.Stream(dev)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            call()
        torch.cuda.current_stream().wait_stream(side)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call()
        y.zero_()
        g.replay()
        assert torch.equal(y, eager), m
        x.copy_(hid_b.cuda())
        g.replay()
        assert_parity(y, H.oracle_layer(layer, hid_b, ids, w), f"graph replay m={m}")


@pytest.mark.parametrize("m,bm", [(1, 0), (16, 0), (17, 0), (200, 0), (160, 16)])
def test_calls_in_flight_together_on_two_streams(request, m, bm):
    """Two buffers, two streams, and a third stream whose matrix products take SMs away from both: the CTAs of a call may start
    one by one, and every call leaves bit for bit what it leaves alone.  (160, 16): with CTAs that start over with larger token slots."""
    from vllm_plugin_b200 import api
    request.addfinalizer(lambda: api.set_kernel_options(block_m=0))
    api.set_kernel_options(block_m=bm)
    layer = H.make_layer(512, 256, 32, 6, True, seed=41)
    weights = H.kernel_weights(layer, "cuda")
    lanes = []
    for lane in range(2):
        hid = O.make_hidden(m, layer.hidden, 50 + lane)
        ids, w = O.make_routing(m, 32, 6, 60 + lane, zipf_s=1.2, mask_frac=0.05)
        want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
        assert buf.plan_words[7] == 80 or bm == 0
        x, ids, w = hid.cuda(), ids.cuda(), w.cuda()
        ys = [torch.empty_like(want) for _ in range(20)]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for y in ys:
                api.stage_inputs_for_mega_moe(buf, x, ids, w)
                api.fp8_fp4_mega_moe(y, weights[0], weights[1], buf, weights[2], weights[3], activation_clamp=10.0)
        lanes.append((graph, torch.cuda.Stream(), ys, want, buf, (x, ids, w)))
    a = torch.randn(2048, 2048, device="cuda", dtype=torch.bfloat16)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        with torch.cuda.stream(other):
            for _ in range(20):
                a @ a
        for graph, stream, *_ in lanes:
            with torch.cuda.stream(stream):
                graph.replay()
    torch.cuda.synchronize()
    for _, _, ys, want, buf, _ in lanes:
        api.read_status(buf)
        for i, y in enumerate(ys):
            assert torch.equal(y, want), i


@pytest.mark.parametrize("geom", [dict(hidden=512, inter=256, num_experts=8, num_topk=6),
                                  dict(hidden=512, inter=256, num_experts=40, num_topk=31),
                                  dict(hidden=256, inter=128, num_experts=512, num_topk=6)])
@pytest.mark.parametrize("m", [1, 15, 16, 17])
def test_staged_tokens_equal_placed_rows(geom, m):
    """Calls of at most 16 tokens in pool blocks of 16 rows multiply the staged tokens as they are and order the routes inside
    GEMM1; with blocks of 32 rows the same call places its rows first.  Bit for bit the same output rows, counts and ``y``, at
    the largest numbers of routes and experts too, when all slots of a token name one expert (more than 32 rows of 16 tokens),
    and with ids past the last expert, which are counted and masked."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(shared=True, seed=71, **geom)
    e, k = layer.num_experts, layer.num_topk
    weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, layer.hidden, 3)
    ids, w = O.make_routing(m, e, k, 4, zipf_s=1.2, mask_frac=0.1)
    repeated = ids[:, :1].clamp(min=0).expand(m, k).clone()
    repeated[0] = e - 1
    beyond = ids.clone()
    beyond[0, 0], beyond[m - 1, k - 1] = e, 2 ** 40
    for case, valid in ((ids, ids), (repeated, repeated), (beyond, torch.where(beyond >= e, -1, beyond))):
        got = []
        for bm in (16, 32):
            api.set_kernel_options(block_m=bm)
            stats = torch.zeros(e, dtype=torch.int32, device="cuda")
            buf = None
            try:
                if case is beyond:
                    buf = got[0][1] if got else H.run_layer(layer, hid, valid, w, weights=weights)[1]
                    with pytest.raises(AssertionError, match="expert ids"):
                        H.run_layer(layer, hid, case, w, weights=weights, buf=buf)
                    y = torch.empty((m, layer.hidden), dtype=torch.bfloat16, device="cuda")
                    api.stage_inputs_for_mega_moe(buf, hid.cuda(), case.cuda(), w.cuda())
                    api.fp8_fp4_mega_moe(y, weights[0], weights[1], buf, weights[2], weights[3], stats, activation_clamp=10.0)
                    with pytest.raises(AssertionError, match="2 expert ids"):
                        api.read_status(buf)
                else:
                    y, buf = H.run_layer(layer, hid, case, w, weights=weights, stats=stats, buf=buf)
            finally:
                api.set_kernel_options(block_m=0)
            rows = int((valid >= 0).sum())
            assert torch.equal(stats.cpu().long(), torch.bincount(valid[valid >= 0], minlength=e))
            got.append((y, buf, buf.ret[:rows].clone(), buf.route_pos[:m].clone(), buf.sorted_route[:rows].clone(), stats))
        for a, b in zip(got[0][2:], got[1][2:]):
            assert torch.equal(a, b)
        assert torch.equal(got[0][0], got[1][0])
        if e <= 40:
            assert_parity(got[0][0], H.oracle_layer(layer, hid, valid, w), f"m {m} e {e}")


@pytest.mark.parametrize("cold", [28, 2])
def test_experts_just_past_one_pair_task(cold):
    """321, 320 and 257 rows beside experts of a few rows: with many of those the tiles have 80 rows and 321 are a second pair
    task, with few of them 112 rows and all three experts are cut into three tiles."""
    layer = H.make_layer(512, 256, 32, 6, True, seed=43)
    m = 340
    hid = O.make_hidden(m, layer.hidden, 3)
    ids = torch.full((m, 6), -1, dtype=torch.int64)
    for slot, n in enumerate((321, 320, 257)):
        ids[m - n:, slot] = slot + 1
    for t in range(3 * cold):
        ids[t, 3] = 4 + t % cold
    w = torch.rand((m, 6), generator=torch.Generator().manual_seed(1))
    y, buf = H.run_layer(layer, hid, ids, w)
    words = buf.plan_words.cpu().tolist()
    tiles, small, cap = words[0], words[6], words[7]
    assert (small, cap, tiles - small) == ((cold + 8, 80, 4) if cold == 28 else (cold + 9, 112, 0))
    assert_parity(y, H.oracle_layer(layer, hid, ids, w), f"cold {cold}")


@pytest.mark.parametrize("bm", [16, 128, 192, 240])
def test_few_tokens_that_name_an_expert_many_times(bm):
    """40 tokens, nearly all six slots of each on one expert: up to 239 rows in a call that is sized for 40 per expert."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(512, 256, 8, 6, True, seed=17)
    hid = O.make_hidden(40, layer.hidden, 4)
    _, w = O.make_routing(40, 8, 6, 5)
    for rows, expert in ((40, 2), (20, 3), (13, 3)):
        ids = torch.full((40, 6), 4, dtype=torch.int64)
        ids[:rows] = expert
        ids[39, 5] = 5
        api.set_kernel_options(block_m=bm)
        try:
            y, _ = H.run_layer(layer, hid, ids, w)
        finally:
            api.set_kernel_options(block_m=0)
        assert_parity(y, H.oracle_layer(layer, hid, ids, w), f"block_m {bm} rows {rows}")


@pytest.fixture(scope="module")
def late_write(tmp_path_factory):
    import ctypes
    import os
    import shutil
    import subprocess
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not installed")
    so = str(tmp_path_factory.mktemp("late") / "late_writer.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(os.path.dirname(__file__), "late_writer.cu")], check=True, capture_output=True)
    fn = ctypes.CDLL(so).late_write
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int64, ctypes.c_void_p]
    return fn


@pytest.mark.parametrize("what", ["shared w13", "shared w13 scales", "w13", "w2"])
@pytest.mark.parametrize("m", [1, 16, 100, 300])
def test_nothing_is_read_before_a_predecessor_that_triggers_early_has_ended(late_write, m, what):
    """Weights rewritten by a kernel in front of the call that lets the call's first kernel start at once and writes 300 us
    later: the output is that of the new weights."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(shared=True, seed=61, **SMALL)
    other = H.make_layer(shared=True, seed=62, **SMALL)
    weights, fresh = H.kernel_weights(layer, "cuda"), H.kernel_weights(other, "cuda")
    i, j = {"shared w13": (2, 0), "shared w13 scales": (2, 1), "w13": (0, 0), "w2": (1, 0)}[what]
    target = weights[i][j]
    source = fresh[i][j] if j == 0 else target + 0x01010101        # every scale doubled
    old, nbytes = target.clone(), target.numel() * target.element_size()
    assert target.stride() == source.stride()
    hid = O.make_hidden(m, layer.hidden, 1)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 2)
    y_old, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    target.copy_(source)
    want, _ = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
    assert not torch.equal(want, y_old)
    x, ids, w = hid.cuda(), ids.cuda(), w.cuda()
    y = torch.empty_like(want)
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(3):
        target.copy_(old)
        torch.cuda.synchronize()
        assert late_write(target.data_ptr(), source.data_ptr(), nbytes, 300_000, stream) == 0
        api.stage_inputs_for_mega_moe(buf, x, ids, w)
        api.fp8_fp4_mega_moe(y, weights[0], weights[1], buf, weights[2], weights[3], activation_clamp=10.0)
        api.read_status(buf)
        assert torch.equal(y, want)


@pytest.mark.parametrize("m,bm", [(7, 16), (130, 32), (300, 128), (300, 192)])
def test_shared_expert_ahead_of_the_routed_plan(m, bm):
    """The split the expert-parallel forward uses, on one GPU: shared expert planned and run first (both GEMMs), routed
    experts afterwards, leaves bit for bit what one launch over the whole plan leaves."""
    import ctypes
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.frontend import _weights_struct, check_mega_moe_arguments, read_status
    layer = H.make_layer(shared=True, seed=21, **SMALL)
    hid = O.make_hidden(m, layer.hidden, 3)
    ids, w = O.make_routing(m, layer.num_experts, layer.num_topk, 4, zipf_s=1.2, mask_frac=0.05)
    api.set_kernel_options(block_m=bm)
    try:
        y_whole, buf = H.run_layer(layer, hid, ids, w)
    finally:
        api.set_kernel_options(block_m=0)
    dev = torch.device("cuda", 0)
    l1, l2, sl1, sl2 = H.kernel_weights(layer, dev)
    y = torch.empty_like(y_whole)
    s13, s2 = check_mega_moe_arguments(y, l1, l2, buf, sl1, sl2, None, (1, 1, 32), "swiglu", 10.0, True, 1.0, 0.0)
    ws = _weights_struct(l1, l2, sl1, sl2, s13, s2)
    lib = _native.load()
    geo, base = ctypes.byref(buf.geo), buf.base_ptr
    opts = _native.MmoeOptions(10.0, 1, 0, 2000, 0)
    sp = torch.cuda.current_stream(dev).cuda_stream
    api.stage_inputs_for_mega_moe(buf, hid.to(dev), ids.to(dev), w.to(dev), block_m=bm)
    _native.check(lib.mmoe_plan_shared(geo, base, m, bm, sp))
    _native.check(lib.mmoe_experts_select(geo, base, ctypes.byref(ws), ctypes.byref(opts), m, bm, 2, sp))
    _native.check(lib.mmoe_dispatch_count(geo, base, m, sp))
    _native.check(lib.mmoe_dispatch_place(geo, base, m, bm, None, sp))
    _native.check(lib.mmoe_experts_select(geo, base, ctypes.byref(ws), ctypes.byref(opts), m, bm, 1, sp))
    _native.check(lib.mmoe_combine(geo, base, y.data_ptr(), m, sp))
    read_status(buf)
    assert torch.equal(y, y_whole)


@pytest.mark.parametrize("m,rows", [(193, (193, 192, 1)), (260, (257, 256, 129, 81, 112)), (300, (300, 160, 161, 113, 80)),
                                    (700, (700, 513, 512, 385, 225, 16)), (400, (337, 336, 258, 305, 400)), (129, (129, 100, 17))])
def test_tile_cuts_at_their_edges(m, rows):
    """Experts with exactly the row counts at which the cut changes: one, two and three tiles of the weights-as-A kernels (80 /
    112 rows each), the first pair, full and just overfull pairs, the rows past one pair that go back to three tiles, and a token that names one expert twice.  The single-GPU
    forward (routes counted, planned and placed in two launches) against the oracle, and bit for bit against the general
    sequence over receive counts."""
    import ctypes
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.frontend import _weights_struct, check_mega_moe_arguments, read_status
    layer = H.make_layer(512, 256, 8, 6, True, seed=41)
    hid = O.make_hidden(m, layer.hidden, 3)
    g = torch.Generator().manual_seed(m)
    ids = torch.full((m, 6), -1, dtype=torch.int64)
    for e, n in enumerate(rows):                               # expert e takes n of the m tokens, in slot e
        ids[torch.randperm(m, generator=g)[:n], e % 6] = e + 1
    ids[0, 5] = ids[0, 0]
    w = torch.rand((m, 6), generator=g)
    y_one, buf = H.run_layer(layer, hid, ids, w)
    pool_one, act_one = buf.l1_acts.view(torch.uint8).clone(), buf.l2_acts.view(torch.uint8).clone()
    met = O.parity_metrics(y_one.cpu(), H.oracle_layer(layer, hid, ids, w))
    assert met["rel_l2"] <= 1e-3, met
    dev = torch.device("cuda", 0)
    l1, l2, sl1, sl2 = H.kernel_weights(layer, dev)
    y = torch.empty_like(y_one)
    s13, s2 = check_mega_moe_arguments(y, l1, l2, buf, sl1, sl2, None, (1, 1, 32), "swiglu", 10.0, True, 1.0, 0.0)
    ws, opts = _weights_struct(l1, l2, sl1, sl2, s13, s2), _native.MmoeOptions(10.0, 1, 0, 2000, 0)
    lib, geo, base = _native.load(), ctypes.byref(buf.geo), buf.base_ptr
    sp = torch.cuda.current_stream(dev).cuda_stream
    bm = api.stage_inputs_for_mega_moe(buf, hid.to(dev), ids.to(dev), w.to(dev))
    _native.check(lib.mmoe_dispatch_count(geo, base, m, sp))
    _native.check(lib.mmoe_dispatch_place(geo, base, m, bm, None, sp))
    _native.check(lib.mmoe_experts(geo, base, ctypes.byref(ws), ctypes.byref(opts), m, bm, sp))
    _native.check(lib.mmoe_combine(geo, base, y.data_ptr(), m, sp))
    read_status(buf)
    assert torch.equal(buf.l1_acts.view(torch.uint8), pool_one) and torch.equal(buf.l2_acts.view(torch.uint8), act_one)
    assert torch.equal(y, y_one)


@pytest.mark.parametrize("hidden,inter,experts,shared", [(256, 128, 4, True), (256, 128, 512, False), (512, 256, 40, True), (2560, 1152, 6, True)])
@pytest.mark.parametrize("m", [1, 16, 17, 129, 193])
def test_both_gemms_in_one_launch(hidden, inter, experts, shared, m):
    """Fewer tasks than CTAs and many times more, K loops of 1, 2 and 20 stages, with and without a shared expert, no expert hit at
    all: bit for bit what a launch per GEMM leaves, call after call, with the counters of the launch back at zero."""
    import ctypes
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.frontend import _weights_struct, check_mega_moe_arguments, read_status
    layer = H.make_layer(hidden, inter, experts, min(6, experts), shared, seed=51)
    dev = torch.device("cuda", 0)
    weights = H.kernel_weights(layer, dev)
    l1, l2, sl1, sl2 = weights
    buf = None
    for call in range(4):
        hid = O.make_hidden(m, hidden, 7 + call)
        ids, w = O.make_routing(m, experts, layer.num_topk, 8 + call, zipf_s=1.2, mask_frac=0.1)
        if call == 2:
            ids = torch.full_like(ids, -1)
        y_one, buf = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
        assert buf.plan_words[9:14].cpu().tolist() == [0] * 5
        y = torch.empty_like(y_one)
        s13, s2 = check_mega_moe_arguments(y, l1, l2, buf, sl1, sl2, None, (1, 1, 32), "swiglu", 10.0, True, 1.0, 0.0)
        ws = _weights_struct(l1, l2, sl1, sl2, s13, s2)
        lib, geo, base = _native.load(), ctypes.byref(buf.geo), buf.base_ptr
        sp = torch.cuda.current_stream(dev).cuda_stream
        bm = api.stage_inputs_for_mega_moe(buf, hid.to(dev), ids.to(dev), w.to(dev))
        _native.check(lib.mmoe_dispatch_count(geo, base, m, sp))
        _native.check(lib.mmoe_dispatch_place(geo, base, m, bm, None, sp))
        for mask in (1, 2):
            opts = _native.MmoeOptions(10.0, 1, 0, 2000, mask)
            _native.check(lib.mmoe_experts(geo, base, ctypes.byref(ws), ctypes.byref(opts), m, bm, sp))
        _native.check(lib.mmoe_combine(geo, base, y.data_ptr(), m, sp))
        read_status(buf)
        assert torch.equal(y, y_one), call
        if experts <= 40 and call < 2:
            assert_parity(y_one, H.oracle_layer(layer, hid, ids, w), f"m {m} call {call}")


@pytest.mark.parametrize("hidden,k,shared", [(512, 6, True), (2560, 10, True), (256, 3, False)])
@pytest.mark.parametrize("few", [16, 64])
def test_small_kernels_of_few_tokens_against_those_of_more(hidden, k, shared, few):
    """Staging and combine have forms of their own for few tokens: what they leave for a token is bit for bit what a call with one token
    more leaves, with a residual, masked routes and more slots than are in flight at once."""
    from vllm_plugin_b200 import api
    layer = H.make_layer(hidden, 256, 12, k, shared, seed=61)
    l1, l2, sl1, sl2 = weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(few + 1, hidden, 3)
    ids, w = O.make_routing(few + 1, 12, k, 4, mask_frac=0.2)
    res = torch.randn(few + 1, hidden, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    got = []
    for m in (few, few + 1):
        y, buf = H.run_layer(layer, hid[:m], ids[:m], w[:m], weights=weights)
        plain = y.clone()
        api.fp8_fp4_mega_moe(y, l1, l2, buf, sl1, sl2, activation_clamp=10.0, residual=res[:m])
        assert torch.equal(y, plain + res[:m])
        got.append((plain[:few], y[:few].clone(), buf.x[:few].view(torch.uint8).clone(), buf.x_sf[:few].clone(), buf.topk_idx[:few].clone()))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    met = O.parity_metrics(got[0][0].cpu(), H.oracle_layer(layer, hid[:few], ids[:few], w[:few]))
    assert met["rel_l2"] <= 1e-3, met


@pytest.mark.parametrize("shared,m,skewed", [(True, 700, False), (False, 700, False), (True, 700, True), (False, 700, True), (True, 230, False)])
def test_launches_behind_the_pairs_wait_where_they_are_not_told(shared, m, skewed):
    """GEMM1 on CTA pairs counts in memory that what precedes it is complete, and what follows it waits for all of GEMM1 where it does not
    find that: here a count far below zero.  Pair tiles only, beside others, and none at all behind the shared expert's; the count
    is back at zero behind every call."""
    from vllm_plugin_b200 import api
    e, k = 16, 2
    layer = H.make_layer(512, 256, e, k, shared, seed=71)
    weights = H.kernel_weights(layer, "cuda")
    hid = O.make_hidden(m, 512, 3)
    ids, w = O.make_routing(m, e, k, 4)
    ids[:, 0] = 5
    ids[:, 1] = 7 if not skewed else torch.arange(m) % 4
    if m == 230:
        ids[:] = torch.arange(2 * m).view(m, 2) % e
    want, buf = H.run_layer(layer, hid, ids, w, weights=weights)
    assert_parity(want, H.oracle_layer(layer, hid, ids, w), f"m {m} shared {shared} skewed {skewed}")
    small, routed = int(buf.plan_words[6]), int(buf.plan_words[0])
    assert (small > 0) == (skewed or m == 230) and (small < routed) == (m == 700)
    told = buf._view(buf.layout.plan, (16 + 6 * e + 8,), torch.int32)[-1:]
    assert not told.any()
    for call in range(4):
        told.fill_(-2 ** 30 if call % 2 == 0 else 0)
        y, _ = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
        assert torch.equal(y, want) and not told.any(), call


TILE_ROWS = [(16, (160, 160, 128), 1), (16, (160, 128, 128), 1), (16, (192, 192, 192), 0), (16, (64,), 7), (32, (64, 33), 5), (32, (65, 33), 5),
             (64, (100, 65, 33), 12)]
MANY_COLD = [(16, (160, 160, 128), 49), (16, (160, 160, 128), 50)]


@pytest.mark.parametrize("hidden,inter,shared,bm,hot,cold", [(512, 256, shared, *case) for shared in (True, False) for case in TILE_ROWS + MANY_COLD] +
                         [(2560, 1152, True, *case) for case in TILE_ROWS])
def test_tile_rows_that_a_call_without_pairs_finds_in_its_plan(hidden, inter, shared, bm, hot, cold):
    """The launch of both GEMMs starts with the shared expert in stages of 32 token rows; where tiles of 80 rows would be fewer by eight, and by
    one in eight, its roles start over with larger ones.  Bit for bit what a launch per GEMM leaves, call after call, on either side of
    the lines (160, 160 and 128 rows: eight tiles fewer of 14 and one per cold expert)."""
    import ctypes
    from vllm_plugin_b200 import api
    from vllm_plugin_b200.backend import _native
    from vllm_plugin_b200.backend.frontend import _weights_struct, check_mega_moe_arguments, read_status
    e, k, m = 72 if hidden == 512 else 24, 4, max(hot)
    layer = H.make_layer(hidden, inter, e, k, shared, seed=81)
    ids = torch.full((m, k), -1, dtype=torch.int64)
    for slot, n in enumerate(hot):
        ids[m - n:, slot] = 3 * slot + 1
    for t in range(cold):
        ids[t, 3] = 8 + t
    counts = torch.bincount(ids[ids >= 0], minlength=e).tolist()
    narrow, wide = (sum(-(-n // rows) for n in counts) for rows in (32, 80))
    fewer = narrow - wide
    cap = 80 if bm == 64 or (bm == 32 and m > 64 and e < 64) or (fewer >= 8 and 8 * fewer > narrow) else 32
    w = torch.rand((m, k), generator=torch.Generator().manual_seed(2))
    dev = torch.device("cuda", 0)
    weights = H.kernel_weights(layer, dev)
    l1, l2, sl1, sl2 = weights
    lib, sp, buf = _native.load(), torch.cuda.current_stream(dev).cuda_stream, None
    api.set_kernel_options(block_m=bm)
    try:
        for call in range(3):
            hid = O.make_hidden(m, hidden, 5 + call)
            y_one, buf = H.run_layer(layer, hid, ids, w, weights=weights, buf=buf)
            words = buf.plan_words.cpu().tolist()
            assert words[6] == (wide if cap == 80 else narrow) and words[7] == cap and words[9:14] == [0] * 5
            tiles = buf.plan_tiles()
            assert torch.bincount(tiles[:words[0], 0].long(), tiles[:words[0], 2].double(), minlength=e).long().tolist() == counts
            assert tiles[words[0]:, 2].sum() == (m if shared else 0) and bool((tiles[words[0]:, 0] == -2).all())
            y = torch.empty_like(y_one)
            s13, s2 = check_mega_moe_arguments(y, l1, l2, buf, sl1, sl2, None, (1, 1, 32), "swiglu", 10.0, True, 1.0, 0.0)
            ws, geo, base = _weights_struct(l1, l2, sl1, sl2, s13, s2), ctypes.byref(buf.geo), buf.base_ptr
            api.stage_inputs_for_mega_moe(buf, hid.to(dev), ids.to(dev), w.to(dev))
            _native.check(lib.mmoe_dispatch_count(geo, base, m, sp))
            _native.check(lib.mmoe_dispatch_place(geo, base, m, bm, None, sp))
            for mask in (1, 2):
                opts = _native.MmoeOptions(10.0, 1, 0, 2000, mask)
                _native.check(lib.mmoe_experts(geo, base, ctypes.byref(ws), ctypes.byref(opts), m, bm, sp))
            _native.check(lib.mmoe_combine(geo, base, y.data_ptr(), m, sp))
            read_status(buf)
            assert torch.equal(y, y_one), call
            if call == 0:
                assert_parity(y_one, H.oracle_layer(layer, hid, ids, w), f"block_m {bm} hot {hot}")
    finally:
        api.set_kernel_options(block_m=0)


@pytest.mark.parametrize("rows,cap", [((200, 30), 32), ((200, 33), 80), ((40, 17), 80)])
def test_shared_expert_cut_as_the_routed_tiles_behind_pair_launches(rows, cap):
    """193 to 256 tokens: the shared expert's tiles have 32 rows, 80 where some routed tile has more than 32 anyway."""
    layer = H.make_layer(512, 256, 64, 6, True, seed=82)
    m = 210
    ids = torch.full((m, 6), -1, dtype=torch.int64)
    for slot, n in enumerate(rows):
        ids[m - n:, slot] = 9 * slot + 2
    w = torch.rand((m, 6), generator=torch.Generator().manual_seed(3))
    hid = O.make_hidden(m, layer.hidden, 6)
    y, buf = H.run_layer(layer, hid, ids, w)
    words = buf.plan_words.cpu().tolist()
    assert words[4] <= 32 and words[1] == -(-m // cap) and words[14] == -(-(-(-m // words[1])) // 16) * 16
    assert_parity(y, H.oracle_layer(layer, hid, ids, w), f"rows {rows}")

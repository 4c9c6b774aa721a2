"""The whole-layer call with the shared expert, at both intermediate sizes and on both sides of every rule that chooses its
route, against kernels that share nothing with it above the grouped GEMMs: the routed experts by the staged kernels (sort,
gather, GEMM1, GEMM2, a launch each) and the shared expert alone. All comparisons are bit for bit."""
import numpy as np
import pytest
import torch

from oracle import moe_oracle as orc
from tests.util import H, bits_of, dev, staged_slots

pytestmark = pytest.mark.gpu
EXPERTS = 8


@pytest.fixture(scope="module")
def C():
    from amd_kernels_b200.moe.mxfp4_h6144_i768_e128_top4 import chain
    return chain


@pytest.fixture(scope="module")
def S():
    from amd_kernels_b200.moe.mxfp4_h6144_i768_e128_top4 import shared_expert
    return shared_expert


def build_layer(inter):
    from amd_kernels_b200.moe import mxfp4_h6144_i768_e128_top4 as p768, mxfp4_h6144_i1536_e128_top4 as p1536
    pkg = p768 if inter == 768 else p1536
    raw, gen = orc.make_weights(seed=inter, experts=EXPERTS, inter=inter)
    sw = pkg.SharedWeights.from_row_major(*(dev(a) for a in orc.make_shared_weights(seed=inter + 1, inter=inter)))
    gate = torch.randn((EXPERTS, H), generator=gen) / H ** 0.5
    return pkg.MoeWeights.from_row_major(gate.cuda(), None, *(dev(a) for a in raw), shared=sw, routing_mode="softmax",
                                         routed_scaling_factor=1.0)


@pytest.fixture(scope="module", params=[768, 1536])
def layer(request):
    return build_layer(request.param)


def inputs(m, seed=0):
    gen = torch.Generator().manual_seed(10 * m + seed)
    return (torch.randn((m, H), generator=gen) * 0.7).bfloat16().cuda(), torch.randn((m, EXPERTS), generator=gen).cuda()


def separate_calls(C, S, x, w, logits):
    """(slots, shared rows, their sum) of the same layer by separate launches."""
    wt, ids = C.route(x, w, logits)
    slots = staged_slots(C, C.mxfp4_quant(x), wt, ids, w)
    # the shared expert in batches of 64: below the sizes of the CTA-pair kernels, on a stream of its own launches
    shared = torch.cat([S.shared_expert(x[a:a + 64].contiguous(), w.shared_weights) for a in range(0, len(x), 64)])
    total = orc.reduce_slots_bf16(bits_of(slots), bits_of(shared))
    return slots, shared, torch.from_numpy(total.view(np.int16)).cuda().view(torch.bfloat16)


@pytest.mark.parametrize("router", [True, False])
@pytest.mark.parametrize("m", [1, 32, 33, 127, 128, 480, 481, 512, 513, 777, 1409, 4096])
def test_layer_equals_the_separate_calls(C, S, layer, m, router):
    """One launch for both GEMMs / two, the role at 16-, 32-, 64- and 128-token blocks, above 512 tokens both quantisers in one
    pass and the shared GEMMs forked to the side stream, from 1409 on CTA pairs."""
    x, lg = inputs(m)
    lg = None if router else lg
    slots0, shared0, sum0 = separate_calls(C, S, x, layer, lg)
    slots, shared = C.mxfp4_moe(x, layer, return_partials=True, router_logits=lg)
    assert torch.equal(slots, slots0) and torch.equal(shared, shared0)
    assert torch.equal(C.mxfp4_moe(x, layer, router_logits=lg), sum0)
    torch.cuda.synchronize()
    assert C.last_status() == 0


@pytest.mark.parametrize("side", [True, False])
@pytest.mark.parametrize("m", [2176, 2177, 2305, 2432])
def test_slots_summed_by_the_shared_second_gemm(C, S, layer, m, side):
    """Around the first size (18 blocks of 128 tokens) at which nobody's shared rows stay in the second GEMM's epilogue: one block
    below, ragged, an odd count of blocks (a pair's second CTA without rows), full blocks; with and without the side stream. A caller
    that takes the slots and the shared rows gets them from the other route, with the same bits."""
    x, lg = inputs(m)
    slots0, shared0, sum0 = separate_calls(C, S, x, layer, lg)
    S.set_dbo_query(None if side else lambda: True)
    try:
        out = C.mxfp4_moe(x, layer, router_logits=lg)
        slots, shared = C.mxfp4_moe(x, layer, return_partials=True, router_logits=lg)
    finally:
        S.set_dbo_query(None)
    torch.cuda.synchronize()
    assert torch.equal(out, sum0) and torch.equal(slots, slots0) and torch.equal(shared, shared0)
    assert C.last_status() == 0


@pytest.mark.parametrize("mode", ["sigmoid_bias", "softmax"])
@pytest.mark.parametrize("m", [32, 33, 39, 481, 513])
def test_routing_beside_the_quantiser(C, S, layer, m, mode):
    """Logits given and no shared expert (with one: above), around the first size of the launch that routes and quantises, token
    counts that leave its last routing CTA part empty, a row of zeros, an infinity, a NaN, logits of NaN and ties, against the staged
    kernels. (The staged quantiser gives a NaN another code below 64 rows, so it gets 64.)"""
    from dataclasses import replace
    x, lg = inputs(m)
    x[1], x[2, 5], x[3, 40:70] = 0, float("inf"), float("nan")
    lg[4], lg[5, 1:3] = float("nan"), lg[5, 0]
    bias = torch.linspace(-0.2, 0.2, EXPERTS, device="cuda") if mode == "sigmoid_bias" else None
    w = replace(layer, shared_weights=None, correction_bias=bias, routing_mode=mode, _abi=None)
    wt, ids = C.route(x, w, lg)
    padded = torch.cat([x, torch.zeros((max(0, 64 - m), H), dtype=x.dtype, device="cuda")])
    want = staged_slots(C, tuple(t[:m].contiguous() for t in C.mxfp4_quant(padded)), wt, ids, w)
    slots, shared = C.mxfp4_moe(x, w, return_partials=True, router_logits=lg)
    torch.cuda.synchronize()
    assert shared is None and torch.equal(slots.view(torch.int16), want.view(torch.int16)) and C.last_status() == 0


@pytest.mark.parametrize("m", [1152, 1153, 2304, 2305, 5632, 5633])
def test_routing_behind_or_beside_the_quantisers_with_a_shared_expert(C, S, layer, m):
    """Around the sizes between which the routing is a launch of its own; without a side stream it never is."""
    x, lg = inputs(m)
    results = []
    for dbo in (None, lambda: True):
        S.set_dbo_query(dbo)
        try:
            results.append((C.mxfp4_moe(x, layer, router_logits=lg), *C.mxfp4_moe(x, layer, router_logits=lg, return_partials=True)))
        finally:
            S.set_dbo_query(None)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(*results)) and C.last_status() == 0


@pytest.mark.parametrize("m", [1, 40, 512, 700, 1600, 2305])
def test_layer_in_a_graph(C, S, layer, m):
    """Capture and replay, the role and (above 512 tokens) the fork to the side stream and its join included, at 2305 in front of the
    second shared GEMM that sums the slots: replayed into a poisoned result, and again with other tokens in the same buffers."""
    x, lg = inputs(m)
    C.mxfp4_moe(x, layer, router_logits=lg)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = C.mxfp4_moe(x, layer, router_logits=lg)
    for seed in (0, 1, 2):
        x2, lg2 = inputs(m, seed)
        want = separate_calls(C, S, x2, layer, lg2)[2]
        x.copy_(x2)
        lg.copy_(lg2)
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert C.last_status() == 0


@pytest.mark.parametrize("m", [40, 700])
def test_layer_inside_a_dual_batch_microbatch(C, S, layer, m):
    """Inside a microbatch no side stream is used, from bf16 rows and from a prepared input, with the same bits."""
    from amd_kernels_b200.moe.mxfp4_h6144_i768_e128_top4 import prepared_input as P
    x, lg = inputs(m)
    want = separate_calls(C, S, x, layer, lg)[2]
    routed = separate_calls(C, S, x, layer, None)[2]
    assert (C._side_stream(layer.shared_weights, m) is not None) == (m > 512)
    S.set_dbo_query(lambda: True)
    try:
        assert C._side_stream(layer.shared_weights, m) is None
        assert torch.equal(C.mxfp4_moe(x, layer, router_logits=lg), want)
        assert torch.equal(C.mxfp4_moe(P.prepare_mxfp4_moe(x, layer), layer), routed)
    finally:
        S.set_dbo_query(None)
    torch.cuda.synchronize()
    assert C.last_status() == 0


def test_workspace_has_no_shared_rows_where_the_slots_are_summed_in_the_second_gemm(layer):
    from amd_kernels_b200 import _lib
    lib = layer.lib()
    for m in (513, 2176, 2177, 16384):
        kept, own = (lib.b200moe_layer_workspace_bytes(m, EXPERTS, _lib.LAYER_SHARED | f) for f in (0, _lib.LAYER_OWN_SHARED_OUT))
        assert own - kept == (0 if m > 2176 else -(-m * 2 * H // 1024) * 1024)


def launched(calls):
    """The kernels of the library that ``calls`` launches, by name and template arguments."""
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        calls()
        torch.cuda.synchronize()
    return {e.key for e in prof.key_averages() if "b200moe" in e.key}


@pytest.mark.parametrize("partials", [False, True])
def test_warm_up_runs_every_kernel_of_the_served_calls(C, layer, partials):
    """Every rule that chooses a kernel by the token count, on both sides of its line: what a call launches, warm-up has launched."""
    sizes = [1, 16, 17, 32, 33, 64, 65, 127, 128, 200, 256, 257, 480, 481, 512, 513, 777, 1024, 1025, 1408, 1409, 2048, 2049, 2176, 2177,
             3000, 4500, 6000, 9000]

    def calls():
        for m in sizes:
            x, lg = inputs(m)
            for logits in (lg, None):
                C.mxfp4_moe(x, layer, router_logits=logits)
                if partials:
                    C.mxfp4_moe(x, layer, router_logits=logits, return_partials=True)
    warm = launched(lambda: C.warm_up_mxfp4_moe(layer, partials=partials))
    if not warm:
        pytest.skip("no kernel trace here: another program holds the profiling interface")
    assert len(warm) > 10 and launched(calls) <= warm

"""CPU-only checks: the C-ABI library loads and exports what include/b200_moe.h declares, and the host-side mirror of
the reference interface validates its arguments the way the reference does."""
import ctypes
import os
import re

import pytest
import torch

from amd_kernels_b200 import _lib
from amd_kernels_b200.moe import mxfp4_h6144_i768_e128_top4 as P
from amd_kernels_b200.moe.mxfp4_h6144_i768_e128_top4 import chain
from oracle import moe_oracle as orc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_functions():
    text = open(os.path.join(ROOT, "include", "b200_moe.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b200moe_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    names = declared_functions()
    assert len(names) >= 18
    for inter in (768, 1536):  # both builds of the sources: the i768 package's library and its i1536 sibling's
        lib = ctypes.CDLL(_lib.lib_path(inter))
        for name in names:
            assert hasattr(lib, name), (inter, name)
    assert set(_lib.SIGNATURES) == set(names), "the ctypes table and the header disagree"
    # the builds differ where the intermediate size enters: scratch for h (codes + scale atoms per sorted row)
    assert _lib.load(1536).b200moe_workspace_bytes(4096, 128) > _lib.load(768).b200moe_workspace_bytes(4096, 128)
    lib = _lib.load()
    assert lib.b200moe_arch() == b"sm_100a" and lib.b200moe_version() >= 1


def test_sizes_match_oracle_and_reference_bounds():
    lib = _lib.load()
    for tokens in (1, 2, 15, 16, 17, 300, 4097, 87381):
        for bm in (16, 32, 64, 128):
            assert lib.b200moe_max_sorted_rows(tokens, bm, 128) == orc.max_sorted_rows(tokens, bm)
        assert lib.b200moe_workspace_bytes(tokens, 128) > tokens * 3264
    assert [lib.b200moe_block_rows(t) for t in (1, 480, 481, 512, 513, 1024, 1729, 87381)] == [16, 16, 32, 32, 128, 128, 128, 128]
    assert lib.b200moe_workspace_bytes(0, 128) == 0 and lib.b200moe_workspace_bytes(87382, 128) == 0
    # the shared expert's dense blocks: the widest block the token count fills
    assert [lib.b200moe_shared_block_rows(t) for t in (1, 16, 17, 32, 33, 64, 65, 87381)] == [16, 16, 32, 32, 64, 64, 128, 128]
    assert lib.b200moe_shared_block_rows(0) == 0 and lib.b200moe_shared_workspace_bytes(0) == 0
    assert lib.b200moe_shared_workspace_bytes(100) >= 128 * (6144 + 768)
    assert lib.b200moe_permute_scratch_bytes(256, 128) == 0 and lib.b200moe_permute_scratch_bytes(257, 128) == 2 * 128 * 4


def test_workspace_holds_the_quantised_rows_where_something_writes_them():
    """(The rest of the layout is that of the call without the flag.) Up to 32 tokens with logits the rows are quantised on their
    way into sorted order; a compact input is expanded into the workspace at every size."""
    lib = _lib.load()
    for tokens in (1, 32, 33, 512, 513):
        full, compact = (lib.b200moe_layer_workspace_bytes(tokens, 128, f) for f in (0, _lib.LAYER_COMPACT))
        if tokens <= 32:
            assert tokens * 3264 <= compact - full <= tokens * 3264 + 2048
        else:
            assert compact == full


def test_dispatch_range():
    # the reference's variant_for: 1..87381, ValueError outside (tests/moe/.../test_entry.py:107-114)
    for m in (1, 8, 512, 513, 4097, 87381):
        assert chain.variant_for(m) in (16, 32, 64, 128)
    for m in (0, -1, 87382):
        with pytest.raises(ValueError):
            chain.variant_for(m)


def _weights(**override):
    m = dict(device="meta")
    w = dict(
        w13=torch.empty((P.E, 2 * P.I, P.H // 2), dtype=torch.uint8, **m),
        w13_scale=torch.empty((P.E, 2 * P.I, P.H // 32), dtype=torch.uint8, **m),
        w2=torch.empty((P.E, P.H, P.I // 2), dtype=torch.uint8, **m),
        w2_scale=torch.empty((P.E, P.H, P.I // 32), dtype=torch.uint8, **m),
        shared_w13=torch.empty((2 * P.I, P.H), dtype=torch.float8_e4m3fn, **m),
        shared_s13=torch.empty((2 * P.I, P.H // 32), dtype=torch.uint8, **m),
        shared_w2=torch.empty((P.H, P.I), dtype=torch.float8_e4m3fn, **m),
        shared_s2=torch.empty((P.H, P.I // 32), dtype=torch.uint8, **m),
    )
    w.update(override)
    return w


def test_unsupported_reason_like_the_reference():
    # tests/moe/.../test_unsupported_reason.py:29-37
    assert P.unsupported_reason(**_weights()) is None
    assert "w2:" in P.unsupported_reason(**_weights(w2=torch.empty((P.E, P.H, P.I), dtype=torch.uint8, device="meta")))
    bf16 = torch.empty((2 * P.I, P.H), dtype=torch.bfloat16, device="meta")
    assert "shared w13:" in P.unsupported_reason(**_weights(shared_w13=bf16))
    assert "SwiGLU" in P.unsupported_reason(**_weights(), swiglu=(1.0, 7.0, 1.0))
    assert "w13:" in P.unsupported_reason(**_weights(w13=None))
    assert P.SWIGLU_OAI == (1.702, 7.0, 1.0) and (P.H, P.I, P.E, P.TOPK) == (6144, 768, 128, 4)


def test_entry_rejects_bad_inputs_without_a_gpu():
    w = object()
    with pytest.raises(ValueError):
        P.mxfp4_moe(torch.zeros((0, 6144), dtype=torch.bfloat16), w)
    with pytest.raises(ValueError):
        P.mxfp4_moe(torch.zeros((4, 6144), dtype=torch.float32), w)
    with pytest.raises(ValueError):
        P.mxfp4_moe(torch.zeros((4, 6000), dtype=torch.bfloat16), w)
    with pytest.raises(ValueError):
        P.mxfp4_moe(torch.zeros((8, 6144), dtype=torch.bfloat16)[::2], w)
    with pytest.raises(ValueError):
        P.MoeWeights.from_row_major(None, None, *(_weights()[k] for k in ("w13", "w13_scale", "w2")), None)


def test_c_abi_rejects_null_and_bad_sizes():
    lib = _lib.load()
    assert lib.b200moe_quant_mxfp4(None, 4, 6144, None, None, None) == _lib.E_ARG
    assert lib.b200moe_permute(None, None, 4, 128, 16, None, None, None, None, None, None) == _lib.E_ARG
    assert lib.b200moe_reduce_slots(None, None, 4, None, None) == _lib.E_ARG
    one = ctypes.c_void_p(16)
    assert lib.b200moe_permute(one, one, 4, 128, 24, one, one, one, one, one, None) == _lib.E_ARG  # bm not 16/32/64/128
    assert lib.b200moe_permute(one, one, 87382, 128, 16, one, one, one, one, one, None) == _lib.E_ARG
    assert lib.b200moe_quant_mxfp4(ctypes.c_void_p(8), 4, 6144, one, one, None) == _lib.E_ALIGN
    with pytest.raises(ValueError):
        _lib.check(_lib.E_ARG, "x")
    with pytest.raises(RuntimeError):
        _lib.check(700, "x")


class _NoLaunch:
    """Stands in for the library handle: the functions that only compute sizes answer as the library does, every other one is
    a launch and fails the test."""
    HOST = ("b200moe_block_rows", "b200moe_max_sorted_rows", "b200moe_permute_scratch_bytes", "b200moe_router_splits",
            "b200moe_layer_workspace_bytes", "b200moe_shared_block_rows", "b200moe_shared_workspace_bytes")

    def __init__(self, real):
        self.real = real

    def __getattr__(self, name):
        if name in self.HOST:
            return getattr(self.real, name)

        def launch(*_):
            raise AssertionError(f"{name} was called with host pointers")
        return launch


def _host_layer(monkeypatch):
    """A layer and its operands on the CPU, with the library replaced and the CUDA queries answered as on a machine with one
    GPU, so that only the entry's own checks stand between the host tensors and a launch."""
    real = _lib.load()
    monkeypatch.setattr(_lib, "load", lambda *a: _NoLaunch(real))
    monkeypatch.setattr(chain, "status_word", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 0, raising=False)
    u8 = lambda *shape: torch.zeros(shape, dtype=torch.uint8)  # noqa: E731
    w = chain.MoeWeights(torch.zeros((8, 6144)), None, u8(8, 12, 1), None, u8(8, 1), None, 1.0, "softmax",
                         router_split=torch.zeros((3, 128, 6144), dtype=torch.bfloat16))
    x = torch.zeros((5, 6144), dtype=torch.bfloat16)
    sort = chain.SortBuffers(torch.zeros(160, dtype=torch.int32), torch.zeros(160), torch.zeros(10, dtype=torch.int32),
                             torch.zeros(2, dtype=torch.int32), 16, 5)
    return w, x, sort, u8


HOST_CALLS = {
    "mxfp4_moe": lambda w, x, sort, u8: P.mxfp4_moe(x, w),
    "mxfp4_moe_logits": lambda w, x, sort, u8: P.mxfp4_moe(x, w, router_logits=torch.zeros((5, 8))),
    "prepare_mxfp4_moe": lambda w, x, sort, u8: P.prepare_mxfp4_moe(x, w),
    "mxfp4_moe_experts": lambda w, x, sort, u8: chain.mxfp4_moe_experts(
        (u8(5, 3072), u8(5, 192)), torch.zeros((5, 4)), torch.zeros((5, 4), dtype=torch.int32), w),
    "mxfp4_quant": lambda w, x, sort, u8: chain.mxfp4_quant(x),
    "topk_route": lambda w, x, sort, u8: chain.topk_route(torch.zeros((5, 8)), None, 1.0, "softmax"),
    "route": lambda w, x, sort, u8: chain.route(x, w),
    "moe_sort": lambda w, x, sort, u8: chain.moe_sort(torch.zeros((5, 4), dtype=torch.int32), torch.zeros((5, 4)), 16, 8),
    "route_sort": lambda w, x, sort, u8: chain.route_sort(torch.zeros((5, 8)), w),
    "dispatch_rows": lambda w, x, sort, u8: chain.dispatch_rows((u8(5, 3072), u8(5, 192)), sort),
    "quant_dispatch": lambda w, x, sort, u8: chain.quant_dispatch(x, sort),
    "grouped_gemm1": lambda w, x, sort, u8: chain.grouped_gemm1(u8(160, 3072), u8(10, 48, 512), sort, w),
    "grouped_gemm2": lambda w, x, sort, u8: chain.grouped_gemm2(u8(160, 384), u8(10, 6, 512), sort, w),
    "grouped_gemm12": lambda w, x, sort, u8: chain.grouped_gemm12(u8(160, 3072), u8(10, 48, 512), sort, w),
    "router_gemm_partials": lambda w, x, sort, u8: chain.router_gemm_partials(x, w.router_weight),
    "router_gemm_quant": lambda w, x, sort, u8: chain.router_gemm_quant(x, w.router_weight, shared=True),
    "split_gate": lambda w, x, sort, u8: chain.split_gate(w.router_weight),
    "reduce_slots": lambda w, x, sort, u8: chain.reduce_slots(torch.zeros((5, 4, 6144), dtype=torch.bfloat16)),
    "reduce_rows": lambda w, x, sort, u8: chain.reduce_rows(torch.zeros((20, 6144), dtype=torch.bfloat16),
                                                            torch.zeros((5, 4), dtype=torch.int32), 5),
}


@pytest.mark.parametrize("call", sorted(HOST_CALLS))
def test_host_tensors_are_refused_before_any_launch(monkeypatch, call):
    layer = _host_layer(monkeypatch)
    with pytest.raises(ValueError):
        HOST_CALLS[call](*layer)


def test_operands_on_another_device_than_the_weights_are_refused(monkeypatch):
    """(The meta device stands in for the other one.)"""
    w, x, sort, u8 = _host_layer(monkeypatch)
    w.w13 = w.w13.to("meta")
    for call in ("mxfp4_moe", "mxfp4_moe_logits", "prepare_mxfp4_moe", "mxfp4_moe_experts"):
        with pytest.raises(ValueError, match="weights"):
            HOST_CALLS[call](w, x, sort, u8)
    w.w13, x = w.w13.to("meta"), x.to("meta")
    with pytest.raises(ValueError, match="router_logits are on cpu"):
        P.mxfp4_moe(x, w, router_logits=torch.zeros((5, 8)))


@pytest.mark.parametrize("inter", [768, 1536])
def test_c_abi_refuses_shared_weights_of_another_intermediate_size(inter):
    """The kernels take the tile counts from the size the library was built for, so the struct says which size its weights
    have. (The misaligned workspace ends the accepted calls before anything is launched.)"""
    lib = _lib.load(inter)
    one = ctypes.c_void_p(256)
    w = _lib.Weights(256, 256, None, 128, _lib.ROUTE_SOFTMAX, 1.0, None, None)
    prep = _lib.Prepared(256, 256, 256, 256, 256, 256, None)
    for size, want in ((inter, _lib.E_ALIGN), (0, _lib.E_ALIGN), (2304 - inter, _lib.E_ARG)):
        sw = _lib.SharedWeights(256, 256, size)
        bad = ctypes.c_void_p(8)
        assert lib.b200moe_layer(ctypes.byref(w), ctypes.byref(sw), one, one, 4, bad, 1 << 40, one, one, one, one, None, None) == want
        assert lib.b200moe_layer_prepared(ctypes.byref(w), ctypes.byref(sw), ctypes.byref(prep), 4, bad, 1 << 40, one, one, one,
                                          one, None, None) == want


@pytest.mark.parametrize("tokens", [1, 512, 513, 2176, 2177, 16384])
def test_c_abi_refuses_misaligned_results_at_every_size(tokens):
    """Whichever kernel ends the call: the same answer on both sides of 18 blocks of 128 tokens, and before anything is launched.
    (A workspace of 0 bytes ends the accepted calls there.)"""
    lib = _lib.load()
    at = ctypes.c_void_p
    w = _lib.Weights(256, 256, None, 128, _lib.ROUTE_SOFTMAX, 1.0, None, None)
    sw = _lib.SharedWeights(256, 256, 768)
    prep = _lib.Prepared(256, 256, 256, 256, 256, 256, None)

    def calls(slots, shared_out, out, shared=True):
        s = ctypes.byref(sw) if shared else None
        p = [None if a is None else at(a) for a in (slots, shared_out, out)]
        yield lib.b200moe_layer(ctypes.byref(w), s, at(256), at(256), tokens, at(256), 0, *p, at(256), None, None)
        yield lib.b200moe_layer_prepared(ctypes.byref(w), s, ctypes.byref(prep), tokens, at(256), 0, *p, at(256), None, None)

    for off in (2, 4, 8):
        for refused in ((None, None, 256 + off), (256, None, 256 + off), (256 + off, None, 256), (256, 256, 256 + off)):
            assert all(r == _lib.E_ALIGN for r in calls(*refused)), refused
            assert all(r == _lib.E_ALIGN for r in calls(refused[0], None, refused[2], shared=False)), refused
        # slots alone: 8 bytes are enough in blocks of up to 32 rows
        want = _lib.E_ARG if off == 8 and tokens <= 512 else _lib.E_ALIGN
        assert all(r == want for r in calls(256 + off, 256, None))
    assert all(r == _lib.E_ARG for r in calls(256, 256, 256))


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("tokens", [1, 32, 33, 513])
def test_c_abi_refuses_misaligned_rows_with_logits(tokens, shared):
    """The quantisers read 16 bytes at a time in every form; up to 32 tokens without a shared expert nobody looked."""
    lib = _lib.load()
    at = ctypes.c_void_p
    w = _lib.Weights(256, 256, None, 128, _lib.ROUTE_SOFTMAX, 1.0, None, None)
    sw = ctypes.byref(_lib.SharedWeights(256, 256, 768)) if shared else None
    for off, want in ((2, _lib.E_ALIGN), (8, _lib.E_ALIGN), (16, _lib.E_ARG)):  # (0 bytes of workspace end the accepted call)
        assert lib.b200moe_layer(ctypes.byref(w), sw, at(256 + off), at(256), tokens, at(256), 0, at(256), at(256), at(256), at(256),
                                 None, None) == want


class _Recorder(_NoLaunch):
    """The library handle's stand-in that accepts the whole-layer calls and keeps the weights struct they were given."""
    def __init__(self, real):
        super().__init__(real)
        self.weights = []

    def __getattr__(self, name):
        if name in ("b200moe_prepare", "b200moe_layer_prepared"):
            def call(w, *_):
                s = w._obj
                self.weights.append((s.w13t, s.bias, s.route_mode, s.route_scale, s.gate, s.gate_split))
                return 0
            return call
        return super().__getattr__(name)


def test_prepared_calls_take_the_weights_as_they_are(monkeypatch):
    """prepare_mxfp4_moe reads the bias, the scale, the mode and the gate that the weights hold at the call, and the calls on
    routed tokens neither need nor make the gate's bf16 terms."""
    w, x, sort, u8 = _host_layer(monkeypatch)
    rec = _Recorder(_lib.load().real)
    monkeypatch.setattr(_lib, "load", lambda *a: rec)
    monkeypatch.setattr(chain, "_raw_stream", lambda device: 0)
    monkeypatch.setattr(chain, "split_gate", lambda gate: pytest.fail("the gate's terms were made"))
    w.abi()
    w.correction_bias, w.routed_scaling_factor, w.routing_mode = torch.ones(8), 2.5, "sigmoid_bias"
    w.router_weight = torch.ones((8, 6144))
    P.prepare_mxfp4_moe(x, w)
    got = rec.weights.pop()
    assert got[1:5] == (w.correction_bias.data_ptr(), _lib.ROUTE_SIGMOID_BIAS, 2.5, w.router_weight.data_ptr())
    w.router_split = w._abi = None
    w.w13 = w.w13.clone()
    HOST_CALLS["mxfp4_moe_experts"](w, x, sort, u8)
    got = rec.weights.pop()
    assert got[0] == w.w13.data_ptr() and got[4] is None and got[5] is None and w.router_split is None


def test_routed_experts_on_a_padded_input(monkeypatch):
    """The routing says how many rows there are; the quantised input may have more rows, never fewer."""
    w, _, _, u8 = _host_layer(monkeypatch)
    monkeypatch.setattr(chain, "layer_prepared", lambda prep, n, *_: None)
    routing = torch.zeros((5, 4)), torch.zeros((5, 4), dtype=torch.int32)
    for rows in (5, 8, 300):
        assert chain.mxfp4_moe_experts((u8(rows, 3072), u8(rows, 192)), *routing, w).shape == (5, 4, 6144)
    for rows in (0, 4):
        with pytest.raises(ValueError):
            chain.mxfp4_moe_experts((u8(rows, 3072), u8(rows, 192)), *routing, w)


def _kernels():
    """(file, name, body) of every __global__ function of the sources, comments removed."""
    csrc = os.path.join(ROOT, "amd_kernels_b200", "csrc")
    for f in sorted(os.listdir(csrc)):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read())
        for m in re.finditer(r"__global__", text):
            body = text[m.start():]
            end = body.find("\n}\n")
            yield f, re.search(r"(\w+)\s*\(const|(\w+_kernel)\s*\(", body).group(0), body[:end]


def test_no_kernel_reads_global_memory_before_its_wait():
    """A kernel that is launched early may ask L2 for data before griddepcontrol.wait, never load it: what the launch before
    it wrote (weights among them) is only certain to be seen behind the wait, and only through L2."""
    seen = 0
    for f, name, body in _kernels():
        at = re.search(r"\bpdl_(enter|wait)\s*\(", body)
        if at is None:
            continue  # ordinary stream order
        seen += 1
        early = re.findall(r"__ldg\(|__ldcg\(|\bld\.|cp\.async\.c[ag]\b|\bload_\w+\(|\*\s*reinterpret_cast<const", body[:at.start()])
        assert not early, (f, name, early)
    assert seen >= 15


def _function(file, start):
    """The source of the function that begins at ``start``, comments removed."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "amd_kernels_b200", "csrc", file)).read())
    body = text[text.index(start):]
    return body[:body.index("\n}\n")]


@pytest.mark.parametrize("file,start,claim", [("gemm_tc.cu", "gemm12_kernel(const", "claim_unit12(done"),
                                              ("shared_role.cuh", "void shared_role(", "atomicAdd(a.ticket, 1)")])
def test_units_that_others_wait_for_belong_to_running_ctas(file, start, claim):
    """Where work of one CTA waits for work of another, a unit is claimed by a CTA that runs. A fixed deal by block index gives
    GEMM1 units to CTAs that may not be resident while waiting ones hold the SMs (two launches on two streams), and then the
    waits run out. So the block index chooses a role here, never a unit."""
    body = _function(file, start)
    assert body.count(claim) == 2  # the first unit, and the next one
    assert "wait_count(" in body and "ring.put(0, u)" in body and body.count("ring.get(") >= 3
    for line in body.splitlines():
        if "blockIdx" in line:
            assert re.search(r"blockIdx\.x\) (>= n_ctas|- \(static_cast<int>\(gridDim\.x\) - ctas\))", line), line
    assert not re.search(r"u \+= (n_ctas|ctas|gridDim)", body)

"""The work that a server of this framework has it do, as cases that can be timed: one MoE layer call on the tokens of one
scheduler step, through the package's public entry points.

Sizes: decode steps of 1 to 256 tokens (the benchmark's decode sweep; a step is rarely a round number, and a CUDA-graph bucket
is padded with zero rows), mixed steps of several hundred tokens, and prefill steps up to the 16384 tokens of the benchmark's
headline. Shapes: hidden 6144, 128 experts, top-4 and intermediate 768, and the sibling package's intermediate 1536. Both
routing rules, the router inside the call or logits from the caller, with and without the MXFP8 shared expert, and the three
forms a caller takes the result in: reduced, the four slots handed to the fused residual + norm + MXFP8 tail, and the
prepared (sequence-parallel) input. ``draw`` gives more calls of the same ranges.
"""
import math

import torch

from amd_kernels_b200.moe import mxfp4_h6144_i768_e128_top4 as moe768
from amd_kernels_b200.moe import mxfp4_h6144_i1536_e128_top4 as moe1536

H, E, TOPK = 6144, 128, 4
SKEW = 2.2  # logit bias -2.2 ln(rank): the benchmark's Zipf-like routing, the top experts get about ten times the mean load


def _case(name, tokens, *, inter=768, router=True, shared=True, mode="sigmoid_bias", form="reduced", skew=False, pad=0):
    case = {} if name is None else {"name": name}
    return {**case, "tokens": tokens, "inter": inter, "router": router, "shared": shared, "mode": mode, "form": form,
            "skew": skew, "pad": pad}


def listed():
    return [
        # one sequence is being generated: the whole layer (router, routed experts, shared expert) on one token
        _case("decode_1_layer", 1),
        # a few sequences, an engine that has its own router and no shared expert
        _case("decode_7_logits", 7, router=False, shared=False, mode="softmax"),
        # the decode step of a small batch, and of a medium one whose result goes into the fused tail
        _case("decode_32_layer", 32),
        _case("decode_100_tail", 100, form="tail"),
        # a CUDA-graph bucket of 256 with 27 padding rows (zero tokens that are routed all the same)
        _case("decode_256_logits_padded", 256, router=False, shared=False, mode="softmax", pad=27),
        # decode and a piece of prefill in one step: ragged, between the decode and the prefill kernels
        _case("mixed_777_layer", 777),
        # the sequence-parallel hand-over: quantise and route the rows, compact them, run the layer on the compact input
        _case("prefill_2048_prepared", 2048, form="prepared"),
        # prefill with skewed routing (the benchmark's stress configuration): a few long experts, some empty ones
        _case("prefill_4096_skewed", 4096, router=False, shared=False, mode="softmax", skew=True),
        # a prefill chunk whose slots go into the fused tail
        _case("prefill_8191_tail", 8191, form="tail"),
        # the largest step: the benchmark's headline token count, whole layer
        _case("prefill_16384_layer", 16384),
        # the sibling shape: a decode step and a prefill chunk
        _case("i1536_decode_64_layer", 64, inter=1536),
        _case("i1536_prefill_4096_layer", 4096, inter=1536),
    ]


def draw(rng):
    """One more call: token count spread over the logarithm of its range, every option drawn."""
    inter = 1536 if rng.random() < 0.2 else 768
    tokens = int(round(math.exp(rng.uniform(0.0, math.log(6144 if inter == 1536 else 16384)))))
    router = rng.random() < 0.6
    form = rng.choice(["reduced", "reduced", "tail", "prepared"] if router else ["reduced", "reduced", "tail"])
    shared = form == "prepared" or rng.random() < 0.6
    return _case(None, tokens, inter=inter, router=router, shared=shared, mode=rng.choice(["sigmoid_bias", "softmax"]),
                 form=form, skew=not router and rng.random() < 0.3,
                 pad=tokens // 8 if tokens <= 256 and rng.random() < 0.3 else 0)


def _bytes(shape, lo, hi, dev, gen):
    return torch.randint(lo, hi, shape, dtype=torch.uint8, device=dev, generator=gen)


def prepare(case, seed):
    """Weights in the kernels' layout (a server keeps them) and the step's inputs, all drawn on the GPU from the seed. Routed
    weights: E2M1 codes uniform, E8M0 scales 2^-7..2^-3 (the benchmark's recipe). Shared weights: E4M3 codes of 20 N(0,1) with
    scales that give outputs of the routed experts' size. Tokens are normed rows, N(0,1) in bf16."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    inter, t = case["inter"], case["tokens"]
    pkg = moe1536 if inter == 1536 else moe768

    def randn(*shape):
        return torch.randn(shape, device=dev, generator=gen)

    shared = None
    if case["shared"]:
        def weight(n, k, lo, hi):
            return (randn(n, k) * 20).to(torch.float8_e4m3fn), _bytes((n, k // 32), lo, hi, dev, gen)
        shared = pkg.SharedWeights.from_row_major(*weight(2 * inter, H, 114, 120), *weight(H, inter, 116, 122))
    gate = randn(E, H) / math.sqrt(H) if case["router"] else None
    bias = randn(E) * 0.05 if case["mode"] == "sigmoid_bias" else None
    weights = pkg.MoeWeights.from_row_major(
        gate, bias, _bytes((E, 2 * inter, H // 2), 0, 256, dev, gen), _bytes((E, 2 * inter, H // 32), 120, 125, dev, gen),
        _bytes((E, H, inter // 2), 0, 256, dev, gen), _bytes((E, H, inter // 32), 120, 125, dev, gen), shared=shared,
        routed_scaling_factor=2.0 if case["mode"] == "sigmoid_bias" else 1.0, routing_mode=case["mode"])
    state = {"case": case, "pkg": pkg, "w": weights, "x": randn(t, H).bfloat16()}
    if case["pad"]:
        state["x"][t - case["pad"]:] = 0
    if not case["router"]:
        state["logits"] = randn(t, E)
        if case["skew"]:
            state["logits"] -= SKEW * torch.log(torch.arange(1, E + 1, device=dev, dtype=torch.float32))
    if case["form"] == "tail":
        state["residual"] = (randn(t, H) * 3).bfloat16()
        state["norm"] = (randn(H) * 0.2).bfloat16()
    return state


def run(state):
    case, pkg, w = state["case"], state["pkg"], state["w"]
    with torch.inference_mode():
        if case["form"] == "prepared":
            return pkg.mxfp4_moe(pkg.prepare_mxfp4_moe(state["x"], w).compact(), w)
        logits = state.get("logits")
        if case["form"] == "reduced":
            return pkg.mxfp4_moe(state["x"], w, router_logits=logits)
        slots, shared = pkg.mxfp4_moe(state["x"], w, return_partials=True, router_logits=logits)
        tail = pkg.slots4_add_rmsnorm_mxfp8(slots, shared, state["residual"], state["norm"])
        return [tail.residual, tail.codes.view(torch.float8_e4m3fn), tail.scales]


def work(case):
    """Bytes: the codes and scales of every expert that is expected to be chosen, the gate, the shared expert's weights, each
    token's row and logits in and its result out. Flops: the routed and shared GEMMs and the router's product."""
    t, inter = case["tokens"], case["inter"]
    if case["skew"]:  # the chance of an expert to be among a token's four, to first order four draws by its softmax weight
        p = [(e + 1) ** -SKEW for e in range(E)]
        active = sum(1.0 - (1.0 - q / sum(p)) ** (TOPK * t) for q in p)
    else:
        active = E * (1.0 - (1.0 - TOPK / E) ** t)
    rows = 2 * inter * H + H * inter  # weights of one expert
    nbytes = active * rows * (1 / 2 + 1 / 32) + t * 2 * H + (4 * E * H if case["router"] else 4 * E * t)
    flops = 2.0 * t * TOPK * rows + (2.0 * t * E * H if case["router"] else 0.0)
    if case["shared"]:
        nbytes += rows * (1 + 1 / 32)
        flops += 2.0 * t * rows
    nbytes += t * (2 * H + 2 * H + H + H // 32 if case["form"] == "tail" else 2 * H)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """A sum in another order moves a few of the intermediate's FP4 and FP8 codes and of the bf16 roundings. Measured: routed
    experts against the CUDA-core kernels (another summation order) rel 3e-5, the tail's E4M3 codes 1.4e-4, no scale byte
    different; the shared expert's bf16 output against the fp32 oracle rel 1.7e-3. Four times the largest."""
    return {"rel": 7e-3, "differ": 1e-3} if case["form"] == "tail" else {"rel": 7e-3}

"""The work a program has this library do: one expert layer (or one dense feed-forward) per call, over the
layer shapes of `oco_b200.synth.CONFIGS`, from one token to the largest prefill batch.

A case names a layer shape, a number of rows and the way of calling:

  forward    the layer on device rows, launched kernel by kernel (`Bindings.experts` and its siblings)
  graph      the same call replayed from the library's recorded step (`_Plan.capture`), as decode loops do
  add_norm   the residual add, the norm and the layer in one call (`_Plan.add_norm_forward`)
  host       the layer on pinned host rows, copies in and out included (`_Plan.forward_host`)
  dense      a projection or feed-forward beside the layer (`dense.DensePlan`)

`interleaved` stages gate and up as one tensor; `offset` starts the packed tensors that many bytes past an
allocation's start, as they lie in a file.
"""
import numpy as np
import torch

from oco_b200 import dense, moe, synth

MAX_ROWS = 8192
DENSE = {"projection": dense.PROJECTION, "relu2": dense.FFN_RELU2, "silu_gate": dense.FFN_SILU_GATE}
# the dense shapes beside the layers: kind, weight format, input features, output or intermediate features
DENSE_SHAPES = {
    "nemotron-shared-ffn": ("relu2", synth.FMT_Q4_0, 2688, 3712),
    "qwen3-dense-ffn": ("silu_gate", synth.FMT_Q4_K, 2048, 6144),
    "mxfp4-projection": ("projection", synth.FMT_MXFP4, 2880, 2880),
    "q4_0-projection": ("projection", synth.FMT_Q4_0, 2688, 2688),
    "q4_k-projection": ("projection", synth.FMT_Q4_K, 2048, 2048),
}


def listed():
    def case(name, config, rows, call, interleaved=False, offset=0):
        return dict(name=name, config=config, rows=rows, call=call, interleaved=interleaved, offset=offset)

    return [
        # decode of one sequence: a token per step through the recorded step
        case("20b-token-graph", "gpt-oss-20b", 1, "graph"),
        # the same without a recorded step: many small kernels, host work and launch gaps count
        case("qwen-token", "qwen3-30b-a3b", 1, "forward"),
        case("nemotron-token", "nemotron-h", 1, "forward"),
        # a few sequences (or the tokens of one speculative step), norm included
        case("20b-7-tokens-norm", "gpt-oss-20b", 7, "add_norm"),
        # a serving batch in decode: most experts are touched by a few tokens each
        case("120b-decode-64", "gpt-oss-120b", 64, "forward"),
        # the ragged last chunk of a prompt
        case("20b-chunk-333", "gpt-oss-20b", 333, "forward"),
        # prefill batches of each family
        case("qwen-prefill-512", "qwen3-30b-a3b", 512, "forward"),
        case("nemotron-prefill-1000", "nemotron-h", 1000, "forward"),
        case("20b-prefill-2048", "gpt-oss-20b", 2048, "forward"),
        # a chunk whose rows live in host memory
        case("20b-host-512", "gpt-oss-20b", 512, "host"),
        # the feed-forward of a dense layer over a chunk
        case("dense-silu-512", "qwen3-dense-ffn", 512, "dense"),
        # the largest batch, from a checkpoint with gate and up in one tensor
        case("120b-prefill-8192", "gpt-oss-120b", 8192, "forward", interleaved=True),
    ]


def draw(rng):
    rows = int(round(2 ** rng.uniform(0, 13)))
    if rng.random() < 0.15:
        return dict(config=rng.choice(sorted(DENSE_SHAPES)), rows=rows, call="dense", interleaved=False, offset=0)
    calls = ["forward", "forward", "add_norm", "host"] + (["graph", "graph"] if rows <= 64 else [])
    config = rng.choice(sorted(synth.CONFIGS))
    return dict(config=config, rows=rows, call=rng.choice(calls),
                interleaved=config != "nemotron-h" and rng.random() < 0.25,
                offset=rng.choice([0, 0, 32, 4]))


# ---- inputs ----------------------------------------------------------------------------------------------
def _packed(gen, fmt, rows, k):
    """Random packed rows, uint8 [rows, row bytes], with the distributions of `synth`."""
    elems, size = synth.BLOCK[fmt]
    w = torch.randint(0, 256, (rows, k // elems, size), dtype=torch.uint8, device="cuda", generator=gen)

    def f16(lo, hi):
        v = torch.rand((rows, k // elems, 1), device="cuda", generator=gen) * (hi - lo) + lo
        return v.to(torch.float16).view(torch.uint8)

    if fmt == synth.FMT_MXFP4:
        w[:, :, 0] = torch.randint(127 - 8, 127 - 2, (rows, k // elems), dtype=torch.uint8, device="cuda", generator=gen)
    else:
        w[:, :, 0:2] = f16(1e-3, 1e-2)
        if fmt == synth.FMT_Q4_K:
            w[:, :, 2:4] = f16(1e-3, 1e-2)
    return w.reshape(rows, -1)


def _placed(w, offset):
    """The bytes of `w`, `offset` bytes past the start of an allocation."""
    if w is None:
        return None
    w = w.reshape(-1)
    if not offset:
        return w
    room = torch.zeros(w.numel() + offset + 64, dtype=torch.uint8, device="cuda")
    room[offset:offset + w.numel()] = w
    return room[offset:offset + w.numel()]


def _normal(gen, shape, scale):
    return torch.randn(shape, device="cuda", generator=gen) * scale


def _rows(gen, rows, width):
    return _normal(gen, (rows, width), 1.0).to(torch.bfloat16)


def _layer(case, gen):
    c = dict(shared_ffn=0, normalize=False, scale=1.0)
    c.update(synth.CONFIGS[case["config"]])
    E, H, F, fmt, arch = c["experts"], c["hidden"], c["ffn"], c["fmt"], c["arch"]
    gated, offset = arch != synth.ARCH_NEMOTRON, case["offset"]
    w = dict(router_w=_normal(gen, (E, H), 0.02), down_w=_placed(_packed(gen, fmt, E * H, F), offset))
    if case["interleaved"]:
        w["gate_up_w"] = _placed(_packed(gen, fmt, E * 2 * F, H), offset)
    else:
        w["up_w"] = _placed(_packed(gen, fmt, E * F, H), offset)
        if gated:
            w["gate_w"] = _placed(_packed(gen, fmt, E * F, H), offset)
    if arch == synth.ARCH_GPT_OSS:
        w["router_b"] = _normal(gen, (E,), 0.01)
        if case["interleaved"]:
            w["gate_up_b"] = _normal(gen, (E, 2 * F), 0.01)
        else:
            w["gate_b"], w["up_b"] = _normal(gen, (E, F), 0.01), _normal(gen, (E, F), 0.01)
        w["down_b"] = _normal(gen, (E, H), 0.01)
        return moe.ExpertPlan.new(H, F, E, c["top_k"]), moe.Experts(**w), moe.Bindings.experts, H
    if arch == synth.ARCH_NEMOTRON:
        w["router_b"] = _normal(gen, (E,), 0.1)
        w["shared_up_w"] = _placed(_packed(gen, fmt, c["shared_ffn"], H), offset)
        w["shared_down_w"] = _placed(_packed(gen, fmt, H, c["shared_ffn"]), offset)
        plan = moe.ReluExpertPlan.new(H, F, c["shared_ffn"], E, c["top_k"], c["normalize"], c["scale"])
        return plan, moe.ReluExperts(**w), moe.Bindings.relu_experts, H
    return moe.GatedExpertPlan.new(H, F, E, c["top_k"]), moe.Experts(**w), moe.Bindings.gated_experts, H


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rows = case["rows"]
    if case["call"] == "dense":
        kind, fmt, H, F = DENSE_SHAPES[case["config"]]
        plan = dense.DensePlan(DENSE[kind], fmt, H, F)
        plan.reserve(rows)
        plan.bind(_packed(gen, fmt, F, H).cpu().numpy(),
                  _packed(gen, fmt, F, H).cpu().numpy() if kind == "silu_gate" else None,
                  _packed(gen, fmt, H, F).cpu().numpy() if kind != "projection" else None)
        y = torch.empty((rows, F if kind == "projection" else H), dtype=torch.bfloat16, device="cuda")
        return dict(call="dense", plan=plan, x=_rows(gen, rows, H), y=y, rows=rows)
    plan, weights, operator, H = _layer(case, gen)
    plan.reserve(rows)
    plan.bind(weights)
    s = dict(call=case["call"], plan=plan, weights=weights, operator=operator, rows=rows)
    if case["call"] == "host":
        for name in ("x", "residual"):
            s[name + "_pinned"] = _rows(gen, rows, H).cpu().pin_memory()
            s[name] = s[name + "_pinned"].view(torch.int16).numpy()
        return s
    s["x"], s["residual"] = _rows(gen, rows, H), _rows(gen, rows, H)
    if case["call"] == "forward":
        s["bindings"] = moe.Bindings(moe.Scratch(norm=s["x"]))
    elif case["call"] == "graph":
        s["graph"] = plan.capture(s["x"], s["residual"], rows)
    elif case["call"] == "add_norm":
        s["norm"] = 1.0 + _normal(gen, (H,), 0.1)
        s["hidden"] = torch.empty_like(s["residual"])
    torch.cuda.synchronize()
    return s


def run(s):
    call = s["call"]
    if call == "forward":
        s["operator"](s["bindings"], s["weights"], s["plan"], None, s["residual"], s["rows"])
    elif call == "graph":
        s["graph"].replay()
    elif call == "add_norm":
        # the hidden rows are both input and output: every step starts from rows that came from elsewhere
        s["hidden"].copy_(s["residual"])
        s["plan"].add_norm_forward(s["hidden"], s["x"], s["norm"], 1e-5, True, s["rows"])
        return s["hidden"]
    elif call == "host":
        s["plan"].forward_host(s["x"], s["residual"], s["rows"])
        return s["residual_pinned"]
    else:
        s["plan"].forward(s["x"], s["y"], s["rows"])
        return s["y"]
    return s["residual"]


# ---- what a pass cannot do without -------------------------------------------------------------------------
def work(case):
    rows = case["rows"]
    if case["call"] == "dense":
        kind, fmt, H, F = DENSE_SHAPES[case["config"]]
        mats = {"projection": 1, "relu2": 2, "silu_gate": 3}[kind]
        weights = (F * synth.row_bytes(fmt, H)) * (2 if kind == "silu_gate" else 1)
        weights += 0 if kind == "projection" else H * synth.row_bytes(fmt, F)
        out = F if kind == "projection" else H
        return dict(bytes=weights + 2 * rows * (H + out), flops=2.0 * rows * mats * H * F)
    layer = synth.Layer(**synth.CONFIGS[case["config"]])
    E, H = layer.experts, layer.hidden
    touched = E * (1.0 - (1.0 - layer.top_k / E) ** rows)          # experts that some token of the batch chooses
    bias = 4 * E if layer.arch != synth.ARCH_QWEN else 0
    moved = touched * layer.expert_bytes() + layer.shared_bytes() + 4 * E * H + bias
    moved += rows * H * 2 * (4 if case["call"] == "add_norm" else 3)  # rows in, residual in and out
    return dict(bytes=moved, flops=layer.flops(rows))


def tolerance(case):
    # the outputs are bf16 (unit roundoff 2^-8): an expert's rows, their sum and the residual are each rounded
    # to bf16, with half operands before that
    return {"rel": 5e-3}

"""What is timed of the Qwen4 MoE layer: the calls that an engine makes on it, over the sizes that it makes them at.

An engine keeps, for every layer of its stack, one handle (the weights resident in HBM) and one workspace, and calls the
layer once per decode step, verify step, serving step or prompt chunk.  A case is such a call: on device pointers
(qw4cu_moe_forward_device), on device pointers with the hyper-connection add behind the layer
(qw4cu_moe_forward_hc_add_device), or on host views, the drop-in call of the forward graph (qwen4_moe_forward).

Cases of up to 64 tokens go through `layers` layers of a stack, each with its own weights and its own input (in the
engine a layer's input comes from its mixer, not from the previous MoE layer): the stack's weights are then larger than
L2, as they are in use.  Larger ones run one layer.

Shapes: "config", the layer that the benchmark's configurations name (hidden 2048, 512 experts, top 10, intermediate
512, the routed experts all Q4_K, IQ2_XXS or Q2_K, the shared expert Q4_K); "checkpoint", the layer of the Qwen3.8
checkpoint (hidden 2560, intermediate 640, IQ2_XXS gate and up, Q2_K down stored in 768 columns, Q8_0 shared expert).
Weights are random valid blocks with super-scales for a spread of about 0.02 (as picoforge_b200.synth makes its
"fabricated" ones, made on the GPU here), the router N(0, 0.02), activations N(0, 1).  "zipf": expert popularity follows
Zipf(1.1), carried by one router column against a constant input column, because the router has no bias.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from picoforge_b200 import abi
from picoforge_b200.layer import LayerSpec, MoeLayer

EXPERTS, TOP_K = 512, 10
STREAMS = 4                                     # residual streams of the hyper-connection add
TYPES = {"F32": abi.F32, "Q8_0": abi.Q8_0, "Q2_K": abi.Q2_K, "Q4_K": abi.Q4_K, "IQ2_XXS": abi.IQ2_XXS}


def case(name, entry, tokens, layers, shape, routed, zipf=False, routes=False):
    c = {"entry": entry, "tokens": tokens, "layers": layers, "shape": shape, "routed": routed, "zipf": zipf, "routes": routes}
    return dict(c, name=name) if name else c


def listed():
    return [
        # single-stream decode: the call whose latency a user waits for at every token
        case("decode-1 Q4_K", "device", 1, 4, "config", "Q4_K"),
        # the same step made through host views, as the engine's forward graph calls it
        case("decode-1 IQ2_XXS host", "host", 1, 4, "config", "IQ2_XXS"),
        # speculative verify: one confirmed token and three drafts, with the ids for the route log
        case("verify-4 IQ2_XXS", "device", 4, 4, "config", "IQ2_XXS", routes=True),
        # serving a few, some and many streams at one token each
        case("serve-7 Q2_K hc", "hc", 7, 4, "config", "Q2_K"),
        case("serve-23 IQ2_XXS", "device", 23, 4, "config", "IQ2_XXS"),
        case("serve-64 Q4_K zipf", "device", 64, 4, "config", "Q4_K", zipf=True),
        # prompts: a short one of odd length through host views, one chunk of 1024 in each of two formats, a long one
        case("prefill-333 IQ2_XXS host", "host", 333, 1, "config", "IQ2_XXS", routes=True),
        case("prefill-1024 Q4_K zipf", "device", 1024, 1, "config", "Q4_K", zipf=True),
        case("prefill-1024 Q2_K hc", "hc", 1024, 1, "config", "Q2_K"),
        case("prefill-8192 Q2_K", "device", 8192, 1, "config", "Q2_K"),
        # the real checkpoint's layer: a verify step, and a prompt of odd length
        case("checkpoint verify-4", "device", 4, 4, "checkpoint", "IQ2_XXS", routes=True),
        case("checkpoint prefill-777", "device", 777, 1, "checkpoint", "IQ2_XXS"),
    ]


def draw(rng):
    """Any batch from one token to the longest listed prompt, in every format, by every entry; the checkpoint's layer up
    to its longest listed prompt."""
    shape = rng.choice(["config", "config", "config", "checkpoint"])
    most = 8192 if shape == "config" else 777
    tokens = min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1)))))
    entry = rng.choice(["device", "device", "host", "hc"])
    if entry == "hc":
        tokens = min(tokens, 2048)              # the most that this entry takes
    routed = rng.choice(["Q4_K", "IQ2_XXS", "Q2_K"]) if shape == "config" else "IQ2_XXS"
    return case(None, entry, tokens, rng.choice([3, 4]) if tokens <= 64 else 1, shape, routed, rng.random() < 0.5,
                entry != "hc" and rng.random() < 0.5)


def dims(c):
    """(hidden, intermediate, shared intermediate, stored K of the routed down projection, tensor types)"""
    if c["shape"] == "config":
        r, s = TYPES[c["routed"]], abi.Q4_K
        return 2048, 512, 512, 512, (abi.F32, r, r, r, s, s, s, abi.F32)
    return 2560, 640, 640, 768, (abi.F32, abi.IQ2_XXS, abi.IQ2_XXS, abi.Q2_K, abi.Q8_0, abi.Q8_0, abi.Q8_0, abi.F32)


def blank_spec(c):
    h, i, s, dp, types = dims(c)
    return LayerSpec(h, EXPERTS, TOP_K, i, s, dp, True, types)


# where the fp16 scales of a block lie, their base value, and dmin / d (so that decoded weights centre on zero)
SCALES = {abi.Q4_K: (0, 1.1e-4, 2, 7.5), abi.Q2_K: (80, 2.0e-3, 82, 1.5), abi.IQ2_XXS: (0, 3.0e-4, None, 0.0), abi.Q8_0: (0, 2.7e-4, None, 0.0)}
_staging = []                                   # one pinned buffer for the packed bytes on their way into handles


def packed(gguf_type, rows, k, gen):
    """`rows` rows of k weights as packed bytes on the GPU."""
    if gguf_type == abi.F32:
        return (torch.randn(rows * k, generator=gen, device="cuda") * 0.02).view(torch.uint8)
    size = abi.FORMATS[gguf_type][2]
    blocks = rows * abi.row_bytes(gguf_type, k) // size
    out = torch.randint(0, 256, (blocks, size), generator=gen, device="cuda", dtype=torch.uint8)
    at, base, at_min, ratio = SCALES[gguf_type]
    d = base * (0.75 + 0.5 * torch.rand(blocks, 1, generator=gen, device="cuda"))
    out[:, at:at + 2] = d.half().view(torch.uint8)
    if at_min is not None:
        out[:, at_min:at_min + 2] = (d * ratio).half().view(torch.uint8)
    return out.view(-1)


def zipf_column(gen):
    ranks = (torch.randperm(EXPERTS, generator=gen, device="cuda") + 1).double()
    pmf = ranks ** -1.1
    return (pmf / pmf.sum()).log().float()


def make_layers(c, gen):
    """The handles and workspaces of `layers` layers.  Their routed experts are windows, one expert apart, of one run of
    experts, so no two layers hold the same weights in the same places; routers and shared experts are drawn per layer."""
    n = c["layers"]
    spec = blank_spec(c)
    layouts = spec.layouts()
    parts = []                                  # (tensor, layer or None, bytes on the GPU)
    for index, layout in enumerate(layouts):
        if 1 <= index <= 3:
            parts.append((index, None, packed(layout.gguf_type, layout.n_out * (EXPERTS + n - 1), layout.k_storage, gen)))
            continue
        for l in range(n):
            data = packed(layout.gguf_type, layout.n_out, layout.k_storage, gen)
            if index == 0 and c["zipf"]:
                data.view(torch.float32).view(EXPERTS, spec.hidden)[:, 0] = zipf_column(gen)
            parts.append((index, l, data))
    total = sum(p[2].numel() + 256 for p in parts)
    if not _staging or _staging[0].numel() < total:
        _staging[:] = [torch.empty(total, dtype=torch.uint8, pin_memory=True)]
    host, at, views = _staging[0].numpy(), 0, {}
    for index, l, data in parts:
        _staging[0][at:at + data.numel()].copy_(data)
        views[index, l] = host[at:at + data.numel()]
        at += (data.numel() + 255) // 256 * 256
    del parts
    torch.cuda.synchronize()
    torch.cuda.empty_cache()                    # the library allocates with cudaMalloc, beside torch's pool
    made = []
    for l in range(n):
        spec = blank_spec(c)
        for index, layout in enumerate(layouts):
            if 1 <= index <= 3:
                spec.tensors.append(views[index, None][l * layout.expert_bytes:(l + EXPERTS) * layout.expert_bytes])
            else:
                spec.tensors.append(views[index, l])
        made.append(MoeLayer(abi.product(), spec, c["tokens"]))
        spec.tensors = []                       # the handle has its own copy
    return made


class State:
    """Handles, workspaces and buffers of one case, and the argument lists of its calls."""


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = State()
    s.layers = make_layers(case, gen)
    lib = abi.product().lib
    tokens, hidden = case["tokens"], s.layers[0].spec.hidden
    s.error = abi.Qwen4Error()
    s.calls, s.out, s.keep = [], [], []
    for layer in s.layers:
        x = torch.randn(tokens, hidden, generator=gen, device="cuda")
        if case["zipf"]:
            x[:, 0] = 1.0
        if case["entry"] == "host":
            x, y = x.cpu().numpy(), np.empty((tokens, hidden), np.float32)
            out, routes = {"y": y}, None
            if case["routes"]:
                out["ids"], out["weights"] = np.empty((tokens, TOP_K), np.uint32), np.empty((tokens, TOP_K), np.float32)
                routes = abi.Qwen4MoeRoutes(abi.u32_view(out["ids"]), abi.f32_view(out["weights"]))
                s.keep.append(routes)
            s.calls.append((lib.qwen4_moe_forward, (layer.moe, abi.f32_view(x), abi.f32_view(y), C.byref(routes) if routes else None,
                                                    layer.work, C.byref(s.error))))
        elif case["entry"] == "hc":
            out = {"y": torch.empty(tokens, hidden, device="cuda"),
                   "residual": torch.randn(tokens, STREAMS, hidden, generator=gen, device="cuda")}
            inject = torch.randn(tokens, STREAMS, generator=gen, device="cuda")
            s.keep.append(inject)
            s.calls.append((lib.qw4cu_moe_forward_hc_add_device, (layer.moe, x.data_ptr(), out["y"].data_ptr(), tokens, out["residual"].data_ptr(),
                                                                  inject.data_ptr(), STREAMS, layer.work, C.byref(s.error))))
        else:
            out = {"y": torch.empty(tokens, hidden, device="cuda")}
            if case["routes"]:
                out["ids"] = torch.empty(tokens, TOP_K, device="cuda", dtype=torch.int32)
                out["weights"] = torch.empty(tokens, TOP_K, device="cuda")
            s.calls.append((lib.qw4cu_moe_forward_device, (layer.moe, x.data_ptr(), out["y"].data_ptr(), tokens,
                                                           out["ids"].data_ptr() if case["routes"] else None,
                                                           out["weights"].data_ptr() if case["routes"] else None, layer.work, C.byref(s.error))))
        s.keep.append(x)
        s.out.append(out)
    torch.cuda.synchronize()                    # the library runs on a stream of its own
    return s


def run(state):
    for call, args in state.calls:
        status = call(*args)
        if status:
            raise abi.MoeError(status, state.error)
    return state.out


def distinct_experts(c, hidden):
    """Experts that the batch's tokens choose, on a sample of the same distribution (logits N(0, 0.02^2 hidden) plus the popularity)."""
    rng = np.random.default_rng(c["tokens"])
    bias = np.log(np.arange(1, EXPERTS + 1) ** -1.1) if c["zipf"] else np.zeros(EXPERTS)
    logits = rng.standard_normal((c["tokens"], EXPERTS), np.float32) * (0.02 * hidden ** 0.5) + bias.astype(np.float32)
    return len(np.unique(np.argpartition(logits, EXPERTS - TOP_K, axis=1)[:, EXPERTS - TOP_K:]))


def work(case):
    spec = blank_spec(case)
    h, i, s, t = spec.hidden, spec.inter, spec.shared_inter, case["tokens"]
    layouts = spec.layouts()
    weights = sum(l.tensor_bytes for n, l in enumerate(layouts) if not 1 <= n <= 3)
    weights += distinct_experts(case, h) * sum(l.expert_bytes for l in layouts[1:4])
    values = 2 * t * h * 4                                                          # x and y
    if case["entry"] == "hc":
        values += t * STREAMS * (2 * h + 1) * 4                                     # the residual read and written, inject
    if case["routes"]:
        values += t * TOP_K * 8
    flops = 2.0 * t * (3 * TOP_K * h * i + 3 * h * s + h * (EXPERTS + 1))
    return {"bytes": case["layers"] * (weights + values), "flops": case["layers"] * flops}


def tolerance(case):
    """The layer's own bar on y is an RMS error of 1e-4 of RMS(y).  Paths that carry activations as two int8 digits (15 bits
    of the row's largest value) sit at up to about 7e-5 from the FP32 result, so two right ones may be this far apart; ids are
    the same, bit for bit.  The checkpoint's layer and Q4_K prompts are computed from FP32 or 22-bit activations."""
    if case["shape"] == "checkpoint" or (case["routed"] == "Q4_K" and case["tokens"] > 64):
        return {"rel": 1e-5}
    return {"rel": 1.5e-4}

"""The layer at the sizes where its kernels' tiles end: the exact router's chain tiles (8, 16, 32, 64, 128 tokens) and GEMM
tiles (256, 512), groups of 32 rows, the two ways of building the lists (64 tokens), short K rings and the widened formats, on
device pointers and host views, against the CPU oracle: ids and weights bit for bit, y within 1e-3."""
import numpy as np
import pytest

from picoforge_b200 import abi, synth
from picoforge_b200.layer import MoeLayer

pytestmark = pytest.mark.gpu

Q4, Q2, IQ2, F32 = abi.Q4_K, abi.Q2_K, abi.IQ2_XXS, abi.F32


@pytest.mark.parametrize("routed,down,shared,hidden,inter,physical,experts,top_k,tokens", [
    (Q4, Q4, Q4, 256, 256, 256, 4, 2, 5),            # K of one block: rings shorter than their slots
    (Q2, Q2, Q2, 512, 256, 256, 3, 2, 8),
    (IQ2, IQ2, Q4, 1536, 512, 512, 40, 10, 9),       # 41 router rows: a ragged last tile
    (IQ2, Q2, F32, 1536, 384, 512, 16, 4, 16),        # the checkpoint's mixture: stored padding, a widened shared expert
    (IQ2, Q2, F32, 512, 640, 768, 33, 6, 17),
    (Q2, Q2, Q4, 2560, 256, 256, 24, 8, 32),         # K beyond one pass of the chain ring
    (Q4, Q4, F32, 512, 256, 256, 5, 1, 33),           # top-1; groups of 32 and 1 rows in the shared expert
    (Q4, Q4, Q4, 512, 256, 256, 2, 2, 64),           # every expert takes every token: two full groups each
    (Q4, Q4, Q4, 512, 256, 256, 2, 2, 65),           # the first size with a launch of its own for the lists
    (Q2, Q2, Q2, 512, 512, 512, 7, 3, 128),
    (IQ2, IQ2, Q4, 512, 512, 512, 96, 10, 129),     # the first size of the router GEMM
    (Q4, Q4, Q4, 512, 256, 256, 512, 10, 257),
    (IQ2, Q2, F32, 512, 384, 512, 130, 8, 513),
])
def test_layer_at_tile_edges(gpu, routed, down, shared, hidden, inter, physical, experts, top_k, tokens):
    import oracle
    spec = synth.make_layer(7000 + tokens, routed_type=routed, down_type=down, shared_type=shared, hidden=hidden, inter=inter, shared_inter=256,
                            down_physical=physical, experts=experts, top_k=top_k)
    x = synth.activations(7000 + tokens, tokens, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, tokens) as layer:
        y, ids, weights = layer.forward(x)
        y2, ids2, weights2 = layer.forward(x)
        bad = x.copy()
        bad[tokens - 1, hidden - 1] = np.inf
        with pytest.raises(abi.MoeError):
            layer.forward(bad)                       # found while the rows are staged: nothing is written, the workspace stays usable
        y3, _, _ = layer.forward(x)
    np.testing.assert_array_equal(ids, want["ids"])
    np.testing.assert_array_equal(weights, want["weights"])
    assert np.abs(y - want["y"]).max() <= 1e-3
    np.testing.assert_array_equal(y2, y)             # deterministic
    np.testing.assert_array_equal(y3, y)
    np.testing.assert_array_equal(ids2, ids)
    np.testing.assert_array_equal(weights2, weights)


@pytest.mark.parametrize("hidden,inter", [(256, 768), (768, 256), (1280, 512)])
def test_iq2_rows_of_an_odd_number_of_blocks(gpu, hidden, inter):
    """The resident image of IQ2_XXS rows of three and five blocks decodes to the oracle's bits, and the layer computes with it."""
    import oracle
    spec = synth.make_layer(7800 + hidden, routed_type=IQ2, shared_type=Q4, hidden=hidden, inter=inter, shared_inter=256, experts=8, top_k=3)
    x = synth.activations(7800 + hidden, 6, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, 6) as layer:
        for tensor in (1, 2, 3):
            k, _, rows, experts = spec.shapes()[tensor]
            raw = oracle.decode_rows(IQ2, spec.tensors[tensor], rows * experts, k).reshape(experts, rows, k)
            for expert in (0, experts - 1):
                np.testing.assert_array_equal(layer.decode_rows(tensor, expert, 0, rows).view(np.uint32), raw[expert].view(np.uint32))
        y, ids, _ = layer.forward(x)
    np.testing.assert_array_equal(ids, want["ids"])
    assert np.abs(y - want["y"]).max() <= 1e-3


@pytest.mark.parametrize("routed,hidden,inter,kernel", [
    (IQ2, 1024, 1024, "grouped_mma_kernel"),         # the most down columns of the four-row kernels
    (IQ2, 512, 1280, "gate_up_kernel"),               # one more block: no pair of blocks for the tcgen05 products either
    (IQ2, 512, 1536, "expert_tile_kernel"),
    (IQ2, 3328, 256, "gate_up_kernel"),               # beyond their gate and up columns
    (Q4, 2304, 256, "expert_tile_kernel"),
])
def test_layers_around_the_four_row_kernels_largest_rows(gpu, routed, hidden, inter, kernel):
    """A layer whose rows do not fit the four-row kernels' shared memory twice goes elsewhere, whatever path is preferred."""
    import oracle
    spec = synth.make_layer(7700 + inter, routed_type=routed, shared_type=Q4, hidden=hidden, inter=inter, shared_inter=256, experts=6, top_k=2)
    x = synth.activations(7700 + inter, 6, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    try:
        with MoeLayer(gpu, spec, 6) as layer:
            for path in (-1, 1):
                gpu.lib.qw4cu_set_expert_path(path)
                gpu.lib.qw4cu_launch_log_begin()
                y, ids, _ = layer.forward(x)
                assert kernel in gpu.launch_names()
                np.testing.assert_array_equal(ids, want["ids"])
                assert np.abs(y - want["y"]).max() <= 1e-3
    finally:
        gpu.lib.qw4cu_set_expert_path(-1)


@pytest.mark.parametrize("routed,shared,inter,physical,shared_inter", [
    (Q2, F32, 5, 256, 7),                # experts that start four bytes off an 8-byte boundary; logical columns that end inside a run of eight
    (IQ2, F32, 5, 256, 7),               # two bytes off
    (IQ2, F32, 6, 256, 7),
    (Q2, IQ2, 12, 256, 256),             # experts on the boundary, a last run of four
    (F32, Q4, 5, 5, 256),                # rows of five activations ahead of one that is read 128 bits at a time
    (F32, Q2, 7, 7, 256),
])
def test_packed_layers_off_the_units(gpu, routed, shared, inter, physical, shared_inter):
    import oracle
    spec = synth.make_layer(7600 + inter, routed_type=routed, shared_type=shared, hidden=256, inter=inter, shared_inter=shared_inter, down_physical=physical,
                            experts=5, top_k=2)
    x = synth.activations(7600 + inter, 6, 256)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, 6) as layer:
        for tensor in (1, 3):
            k, _, rows, experts = spec.shapes()[tensor]
            raw = oracle.decode_rows(spec.types[tensor], spec.tensors[tensor], rows * experts, k).reshape(experts, rows, k)
            for expert in range(experts):
                np.testing.assert_array_equal(layer.decode_rows(tensor, expert, 0, rows).view(np.uint32), raw[expert].view(np.uint32))
        for tokens in (1, 6):
            y, ids, weights = layer.forward(x[:tokens])
            np.testing.assert_array_equal(ids, want["ids"][:tokens])
            np.testing.assert_array_equal(weights, want["weights"][:tokens])
            assert np.abs(y - want["y"][:tokens]).max() <= 1e-3


@pytest.mark.parametrize("routed,shared,tokens", [(IQ2, Q4, 40), (Q4, Q4, 96), (Q4, Q4, 7)])
def test_one_workspace_through_every_path_in_turn(gpu, routed, shared, tokens):
    """The four-row kernels' digits and the tcgen05 products' halves lie in the same rows of the workspace: each path gives the same
    bits before and after the others have used it."""
    spec = synth.make_layer(7900 + tokens, routed_type=routed, shared_type=shared, hidden=512, inter=512, shared_inter=256, experts=24, top_k=6)
    x = synth.activations(7900 + tokens, tokens, 512)
    paths = {"expert_tile_kernel": (-1, 1), "grouped_mma_kernel": (1, 0), "gate_up_kernel": (0, -1)}      # expert path, tile path
    seen = {}
    try:
        with MoeLayer(gpu, spec, tokens) as layer:
            for turn in range(2):
                for kernel, (expert, tile) in paths.items():
                    gpu.lib.qw4cu_set_expert_path(expert)
                    gpu.lib.qw4cu_set_tile_path(tile)
                    gpu.lib.qw4cu_set_prefill_path(0)
                    gpu.lib.qw4cu_launch_log_begin()
                    y, ids, _ = layer.forward(x)
                    assert kernel in gpu.launch_names()
                    if turn:
                        np.testing.assert_array_equal(y, seen[kernel])
                    seen[kernel] = y
    finally:
        gpu.lib.qw4cu_set_expert_path(-1)
        gpu.lib.qw4cu_set_tile_path(-1)
        gpu.lib.qw4cu_set_prefill_path(-1)
    for kernel in paths:
        assert np.abs(seen[kernel] - seen["gate_up_kernel"]).max() <= 1e-3


def _in_64_bits(spec, x, ids, weights):
    """y of the layer from the decoded weights, everything behind the routes in float64."""
    import oracle
    x = x.astype(np.float64)

    def matrix(tensor, expert):
        k, logical, rows, experts = spec.shapes()[tensor]
        raw = spec.tensors[tensor].reshape(experts, -1)[expert]
        return oracle.decode_rows(spec.types[tensor], np.ascontiguousarray(raw), rows, k)[:, :logical].astype(np.float64)

    def expert(first, e, rows):
        g, u = rows @ matrix(first, e).T, rows @ matrix(first + 1, e).T
        return (g / (1.0 + np.exp(-g)) * u) @ matrix(first + 2, e).T

    gate = 1.0 / (1.0 + np.exp(-(x @ spec.tensors[7].view(np.float32).astype(np.float64))))
    y = expert(4, 0, x) * gate[:, None]
    for e in np.unique(ids):
        token, slot = np.nonzero(ids == e)
        y[token] += expert(1, e, x[token]) * weights[token, slot].astype(np.float64)[:, None]
    return y


@pytest.mark.parametrize("routed,down,shared,hidden,inter,physical,tokens", [
    (Q4, Q4, Q4, 2048, 512, 512, 40),
    (Q4, Q4, Q4, 2048, 512, 512, 96),
    (Q2, Q2, Q2, 2048, 512, 512, 7),
    (Q2, Q2, Q4, 512, 256, 256, 96),
    (IQ2, IQ2, IQ2, 2048, 512, 512, 96),
    (IQ2, Q2, F32, 2560, 640, 768, 4),               # the checkpoint's mixture, its shared expert widened
    (IQ2, Q2, F32, 2560, 640, 768, 96),
])
def test_tcgen05_products_keep_fp32_accuracy(gpu, routed, down, shared, hidden, inter, physical, tokens):
    """Exact integer codes against activations in fp16 hi + lo: RMS error within 3e-6 of RMS(y), against 64 bits, in every format.

    A chain of K <= 2560 FP32 additions is off by about sqrt(K / 3) roundings of 2^-24, 1.7e-6, in each of gate, up and down: 3e-6
    together.  The products add in blocks and stay below that although the tensor core truncates (1.5e-6 to 2.4e-6 measured over
    formats and sizes); the halves add 2^-22 per value.  Activations without their low half would be off by 2^-12, int8 digits by 2^-16
    (5e-5 of RMS(y)); a bit lost from a code or a scale by far more."""
    import oracle
    spec = synth.make_layer(7500 + tokens, routed_type=routed, down_type=down, shared_type=shared, hidden=hidden, inter=inter, shared_inter=inter,
                            down_physical=physical, experts=32, top_k=6)
    x = synth.activations(7500 + tokens, tokens, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, tokens) as layer:
        gpu.lib.qw4cu_launch_log_begin()
        y, ids, weights = layer.forward(x)
        assert {"expert_tile_kernel", "prefill_tc_kernel"} & set(gpu.launch_names())
    np.testing.assert_array_equal(ids, want["ids"])
    exact = _in_64_bits(spec, x, ids, weights)
    error = np.sqrt(np.mean((y - exact) ** 2)) / np.sqrt(np.mean(exact ** 2))
    print(f"RMS error {error:.3e}")
    assert error <= 3e-6


@pytest.mark.parametrize("routed,down,hidden,inter,physical", [
    (Q4, Q4, 256, 128, 256),              # one unit an item, more than eight items a CTA: the rings of groups, pairs and scales at their tightest
    (Q2, Q2, 256, 128, 256),
    (IQ2, IQ2, 512, 128, 512),
    (Q2, Q2, 256, 128, 2304),             # scales of two items held, an item one stage of four
    (Q2, Q2, 256, 384, 4096),             # two stages
    (IQ2, Q2, 512, 640, 2560),            # three: the first that cannot run ahead of its scales
])
def test_many_short_items_a_cta(gpu, routed, down, hidden, inter, physical):
    """64 experts with 640 rows each: 1280 groups, and as many or twice as many items of the down product on 148 CTAs."""
    import oracle
    tokens = 4096
    spec = synth.make_layer(7550 + physical, routed_type=routed, down_type=down, shared_type=Q4, hidden=hidden, inter=inter, shared_inter=256,
                            down_physical=physical, experts=64, top_k=10, fabricated=True)
    x = synth.activations(7550, tokens, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, tokens) as layer:
        gpu.lib.qw4cu_launch_log_begin()
        y, ids, _ = layer.forward(x)
        assert {"expert_tile_kernel", "prefill_tc_kernel"} & set(gpu.launch_names())
        y2, _, _ = layer.forward(x)
    np.testing.assert_array_equal(ids, want["ids"])
    np.testing.assert_array_equal(y2, y)
    exact = want["y"].astype(np.float64)
    assert np.sqrt(np.mean((y - exact) ** 2)) <= 1e-5 * np.sqrt(np.mean(exact ** 2))


def _with_scales(blocks, gguf_type, doubled):
    """Copies of Q4_K / Q2_K blocks whose integer scales fit one bit less than the format has; plain: with twice
    the super-scale; `doubled`: with those scales times two, the same weights bit for bit."""
    out = blocks.copy()
    at = 0 if gguf_type == Q4 else 80
    if gguf_type == Q2:
        low = out[:, :16] & 7
        out[:, :16] = (out[:, :16] & 0xF0) | (low << 1 if doubled else low)
    else:                                            # scales of runs 0-3 in six bits of one byte each, of 4-7 in a nibble and the two bits above
        first, last = out[:, 4:8] & 0x1F, out[:, 12:16] & 0x0F
        out[:, 4:8] = (first << 1) | (last >> 3 << 6) if doubled else first
        if doubled:
            out[:, 12:16] = (out[:, 12:16] & 0xF0) | (last << 1 & 0x0F)
    d = out[:, at:at + 2].copy().view(np.float16)
    out[:, at:at + 2] = (d if doubled else d * np.float16(2)).view(np.uint8)
    return out


@pytest.mark.parametrize("routed,tokens", [(Q4, 7), (Q4, 96), (Q2, 7), (Q2, 96)])
def test_tcgen05_products_do_not_depend_on_where_a_power_of_two_lies(gpu, routed, tokens):
    """A factor of two in the integer scales or in the super-scales makes the same weights, so y is the same bits, as long as the operands that codes and
    scales are folded into are normal halves (the tensor core aligns products of subnormal ones as if they were larger: 1e-7 of y)."""
    import oracle
    seen = []
    for doubled in (False, True):
        spec = synth.make_layer(7450, routed_type=routed, shared_type=routed, hidden=1024, inter=512, shared_inter=512, experts=24, top_k=6, fabricated=True)
        for tensor in range(1, 7):
            blocks = spec.tensors[tensor].reshape(-1, abi.FORMATS[routed][2])
            spec.tensors[tensor] = np.ascontiguousarray(_with_scales(blocks, routed, doubled)).reshape(-1)
        x = synth.activations(7450 + tokens, tokens, 1024)
        decoded = oracle.decode_rows(routed, spec.tensors[1], 512, 1024)
        with MoeLayer(gpu, spec, tokens) as layer:
            gpu.lib.qw4cu_launch_log_begin()
            y, ids, _ = layer.forward(x)
            assert {"expert_tile_kernel", "prefill_tc_kernel"} & set(gpu.launch_names())
        seen.append((decoded, ids, y))
    for plain, twice in zip(*seen):
        np.testing.assert_array_equal(plain, twice)


@pytest.mark.parametrize("routed,tokens", [(Q4, 2048), (Q2, 2049), (Q4, 4096), (Q2, 4097), (Q4, 4500)])
def test_long_prompts(gpu, routed, tokens):
    """Lists of more than 64 words of 32 tokens an expert, the last word full or of one token, and a second launch sequence of one
    token or of 404."""
    import oracle
    spec = synth.make_layer(7400 + tokens, routed_type=routed, shared_type=routed, hidden=256, inter=256, shared_inter=256, experts=40, top_k=3)
    x = synth.activations(7400 + tokens, tokens, 256)
    want = oracle.forward(spec, x, threads=synth.threads())
    with MoeLayer(gpu, spec, tokens) as layer:
        y, ids, weights = layer.forward(x)
    np.testing.assert_array_equal(ids, want["ids"])
    np.testing.assert_array_equal(weights, want["weights"])
    exact = want["y"].astype(np.float64)
    assert np.sqrt(np.mean((y - exact) ** 2)) <= 1e-5 * np.sqrt(np.mean(exact ** 2))


@pytest.mark.parametrize("top_k,inter,shared_inter", [(16, 640, 512), (16, 640, 256), (33, 256, 256)])
def test_down_rows_around_48_kb_of_shared_memory(gpu, top_k, inter, shared_inter):
    """The CUDA-core down kernel holds a token's activations: (16, 640, 512) are 48,656 bytes, which with its table are more than
    the 48 KB that a launch gets unasked."""
    import oracle
    spec = synth.make_layer(7300 + inter, routed_type=Q4, down_type=IQ2, shared_type=Q4, hidden=768, inter=inter, shared_inter=shared_inter,
                            down_physical=(inter + 255) // 256 * 256, experts=40, top_k=top_k)
    x = synth.activations(7300 + inter, 9, 768)
    want = oracle.forward(spec, x, threads=synth.threads())
    gpu.lib.qw4cu_set_expert_path(0)
    try:
        with MoeLayer(gpu, spec, 9) as layer:
            y, ids, _ = layer.forward(x)
    finally:
        gpu.lib.qw4cu_set_expert_path(-1)
    np.testing.assert_array_equal(ids, want["ids"])
    assert np.abs(y - want["y"]).max() <= 1e-3


def test_an_upload_has_arrived_when_the_call_returns(gpu):
    """A megabyte and a row from pageable memory: the row travels as a piece of its own, and the library's stream does not wait for the
    stream that it travels on."""
    import ctypes as C
    lib, err = gpu.lib, abi.Qwen4Error()
    spec = synth.make_layer(7200, routed_type=Q4, shared_type=Q4, hidden=512, inter=256, shared_inter=256, experts=16, top_k=4)
    tokens, k = 513, spec.top_k
    d_x, d_ids = lib.qw4cu_malloc(tokens * 2048), lib.qw4cu_malloc(tokens * k * 4)
    try:
        with MoeLayer(gpu, spec, tokens) as layer:
            for turn in range(40):
                x = synth.activations(7200 + turn, tokens, 512)
                assert lib.qw4cu_upload(d_x, x.ctypes.data, x.nbytes) == 0
                assert lib.qw4cu_moe_route_device(layer.moe, d_x, tokens, d_ids, None, layer.work, C.byref(err)) == abi.OK
                assert lib.qw4cu_moe_work_sync(layer.work, C.byref(err)) == abi.OK
                ids = np.empty((tokens, k), np.uint32)
                assert lib.qw4cu_download(ids.ctypes.data, d_ids, ids.nbytes) == 0
                _, want, _ = layer.forward(x)
                np.testing.assert_array_equal(ids, want, err_msg=f"turn {turn}")
    finally:
        lib.qw4cu_free(d_x)
        lib.qw4cu_free(d_ids)

"""The four-row grouped kernels on the expanded image of an IQ2_XXS layer against the same kernels on its packed image: the same
integers, scales and order of sums, so the same bits; and against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,inter,tokens,shared", [
    (2048, 512, 5, 12),                  # one block of 512 columns down, four gate/up; a row or two to an expert
    (2048, 512, 64, 12),                 # whole groups of four, and their remainders
    (512, 512, 7, 12),                   # one block each: k-slices without a half block
    (1536, 512, 23, 16),                 # an odd number of blocks; the shared expert on its image as well
    (2560, 512, 9, 16),                  # the most gate/up columns of which two units fit
    (3072, 512, 6, 16),                  # one more block: the packed image
    (1024, 1024, 6, 12),                 # two blocks down: the packed image there
])
def test_expanded_and_packed_images_give_the_same_bits(gpu, hidden, inter, tokens, shared):
    import oracle
    from picoforge_b200 import abi, synth
    from picoforge_b200.layer import MoeLayer
    spec = synth.make_layer(9100 + hidden + tokens, routed_type=abi.IQ2_XXS, shared_type=shared, hidden=hidden, inter=inter, shared_inter=512, experts=24, top_k=5)
    x = synth.activations(9100 + tokens, tokens, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    results = []
    for fused in (-1, 0):                                    # 0 before create: a layer without expanded images
        try:
            gpu.lib.qw4cu_set_fused_decode(fused)
            with MoeLayer(gpu, spec, tokens) as layer:
                gpu.lib.qw4cu_set_expert_path(1)
                gpu.lib.qw4cu_launch_log_begin()
                results.append(layer.forward(x))
                assert "grouped_mma_kernel" in gpu.launch_names()
        finally:
            gpu.lib.qw4cu_set_expert_path(-1)
            gpu.lib.qw4cu_set_fused_decode(-1)
    (y, ids, weights), (y_packed, ids_packed, weights_packed) = results
    np.testing.assert_array_equal(ids, want["ids"])
    np.testing.assert_array_equal(ids, ids_packed)
    np.testing.assert_array_equal(weights, weights_packed)
    np.testing.assert_array_equal(y, y_packed)
    assert np.sqrt(np.mean((y - want["y"]) ** 2)) <= 1e-4 * np.sqrt(np.mean(want["y"] ** 2))

"""Device pointers that are aligned to a float and no more.

x_dev and y_dev of qw4cu_moe_forward_device are dense FP32 (include/qwen4_moe_b200.h); nothing asks for a 16-byte boundary, and a
row of a larger activation buffer need not start on one.  Every path that such a call can take reads x through kernels whose
128-bit loads have a scalar twin: the result is the aligned call's, bit for bit, where both take the same products."""
import ctypes as C

import numpy as np
import pytest

from picoforge_b200 import abi, synth
from picoforge_b200.layer import MoeLayer

pytestmark = pytest.mark.gpu

Q4, Q2, IQ2, F32 = abi.Q4_K, abi.Q2_K, abi.IQ2_XXS, abi.F32


def device_call(api, layer, x, shift):
    """(y, ids, weights, kernels) of one call whose x and y start `shift` bytes into their allocations."""
    lib, err = api.lib, abi.Qwen4Error()
    tokens, k = x.shape[0], layer.spec.top_k
    bases = [lib.qw4cu_malloc(x.nbytes + 64) for _ in range(2)] + [lib.qw4cu_malloc(tokens * k * 4) for _ in range(2)]
    try:
        assert all(b and b % 256 == 0 for b in bases)
        dx, dy = bases[0] + shift, bases[1] + shift
        assert lib.qw4cu_upload(dx, x.ctypes.data, x.nbytes) == 0
        lib.qw4cu_launch_log_begin()
        assert lib.qw4cu_moe_forward_device(layer.moe, dx, dy, tokens, bases[2], bases[3], layer.work, C.byref(err)) == abi.OK, err.detail
        names = api.launch_names()
        assert lib.qw4cu_moe_work_sync(layer.work, C.byref(err)) == abi.OK, err.detail
        y, ids, weights = np.empty_like(x), np.empty((tokens, k), np.uint32), np.empty((tokens, k), np.float32)
        for host, device in ((y, dy), (ids, bases[2]), (weights, bases[3])):
            assert lib.qw4cu_download(host.ctypes.data, device, host.nbytes) == 0
        return y, ids, weights, names
    finally:
        for b in bases:
            lib.qw4cu_free(b)


@pytest.mark.parametrize("routed,shared,hidden,inter,tokens,expert_path,kernel", [
    (IQ2, Q4, 1024, 512, 4, -1, "quantize_rows_kernel"),       # the one-kernel decode path refuses such an x: the four-row kernels take it
    (IQ2, Q4, 512, 256, 23, -1, "quantize_rows_kernel"),
    (Q2, Q2, 512, 256, 7, -1, "split_rows_kernel"),
    (Q4, Q4, 512, 256, 65, -1, "split_rows_kernel"),
    (IQ2, F32, 1536, 512, 130, -1, "split_rows_kernel"),       # beyond the chain router's tokens: the GEMM does not take it either
    (Q4, Q4, 512, 256, 9, 0, "gate_up_kernel"),
    (Q2, IQ2, 512, 256, 66, 0, "gate_up_kernel"),
])
def test_rows_off_the_16_byte_grid(gpu, routed, shared, hidden, inter, tokens, expert_path, kernel):
    import oracle
    spec = synth.make_layer(8100 + tokens, routed_type=routed, shared_type=shared, hidden=hidden, inter=inter, shared_inter=inter, experts=24, top_k=5)
    x = synth.activations(8100 + tokens, tokens, hidden)
    want = oracle.forward(spec, x, threads=synth.threads())
    gpu.lib.qw4cu_set_expert_path(expert_path)
    try:
        with MoeLayer(gpu, spec, tokens) as layer:
            aligned = device_call(gpu, layer, x, 0)
            for shift in (4, 8, 12):
                y, ids, weights, names = device_call(gpu, layer, x, shift)
                assert kernel in names and "fused_decode_kernel" not in names, names
                np.testing.assert_array_equal(ids, want["ids"])
                np.testing.assert_array_equal(weights, want["weights"])
                assert np.abs(y - want["y"]).max() <= 1e-3
                if kernel in aligned[3]:                       # the same products: the same bits
                    np.testing.assert_array_equal(y, aligned[0])
    finally:
        gpu.lib.qw4cu_set_expert_path(-1)


def test_fast_router_off_the_16_byte_grid(gpu):
    """The tree-summed router reads x 128 bits at a time too; its sums do not depend on how they were loaded."""
    spec = synth.make_layer(8200, routed_type=Q4, shared_type=Q4, hidden=512, inter=256, shared_inter=256, experts=24, top_k=5)
    x = synth.activations(8200, 9, 512)
    gpu.lib.qw4cu_set_router_mode(1)
    try:
        with MoeLayer(gpu, spec, 9) as layer:
            aligned = device_call(gpu, layer, x, 0)
            for shift in (4, 8, 12):
                moved = device_call(gpu, layer, x, shift)
                assert "router_fast_kernel" in moved[3]
                for a, b in zip(moved[:3], aligned[:3]):
                    np.testing.assert_array_equal(a, b)
    finally:
        gpu.lib.qw4cu_set_router_mode(0)


def test_expert_parallel_rows_off_the_16_byte_grid(gpu):
    """x and y of the expert-parallel step may start anywhere a float may; the exchange rows and partial sums, which kernels of this
    library write for kernels of this library, are refused off a 16-byte boundary, and a layer that the step has no kernel for
    before anything is launched."""
    import sys
    from pathlib import Path
    sys.path.insert(0, str(Path(__file__).resolve().parent))
    import cases
    from picoforge_b200.expert_parallel import Communicator, EpLayer
    lib, err = gpu.lib, abi.Qwen4Error()
    spec = synth.make_layer(8300, routed_type=Q2, shared_type=Q4, hidden=512, inter=256, shared_inter=256, experts=16, top_k=4)
    x = synth.activations(8300, 9, 512)
    layer, comm = EpLayer(gpu, spec, 9, 1, 0), Communicator(gpu, 0, 1)
    pitch = lib.qw4cu_ep_row_floats(layer.layer.moe)
    d_x, d_y, d_rows = lib.qw4cu_malloc(x.nbytes + 16), lib.qw4cu_malloc(x.nbytes + 16), lib.qw4cu_malloc(9 * pitch * 4 + 16)
    try:
        got = []
        for shift in (0, 4, 12):
            assert lib.qw4cu_upload(d_x + shift, x.ctypes.data, x.nbytes) == 0
            layer.forward(comm, d_x + shift, d_y + shift)
            layer.sync()
            y = np.empty_like(x)
            assert lib.qw4cu_download(y.ctypes.data, d_y + shift, y.nbytes) == 0
            got.append((y, *layer.routes()))
        for moved in got[1:]:
            for a, b in zip(moved, got[0]):
                np.testing.assert_array_equal(a, b)
        moe, work = layer.layer.moe, layer.layer.work
        assert lib.qw4cu_moe_ep_begin_device(moe, d_x, 9, d_rows + 4, None, None, work, C.byref(err)) == abi.STRIDE
        assert lib.qw4cu_moe_ep_experts_device(moe, d_rows + 8, 9, 0, d_y, work, C.byref(err)) == abi.STRIDE
        assert lib.qw4cu_moe_ep_experts_device(moe, d_rows, 9, 0, d_y + 4, work, C.byref(err)) == abi.STRIDE
        odd = cases.float_layer(8301, hidden=10)              # rows of 40 bytes: every other one lies off the grid
        with MoeLayer(gpu, odd, 6) as generic:
            launches = lib.qw4cu_launch_count()
            assert lib.qw4cu_moe_ep_begin_device(generic.moe, d_x, 3, d_rows, None, None, generic.work, C.byref(err)) == abi.GPU_ERROR
        assert lib.qw4cu_launch_count() == launches
    finally:
        layer.close()
        comm.close()
        for p in (d_x, d_y, d_rows):
            lib.qw4cu_free(p)

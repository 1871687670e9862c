"""Threads with a workspace each, on one layer each, all at once in a fresh process: what the library makes on first use (streams,
events, tables) is made once, and every call gives the bits of a call made alone."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np
from picoforge_b200 import abi, synth
from picoforge_b200.layer import MoeLayer
gpu = abi.product()
assert gpu.lib.qw4cu_set_device(0) == 0
made = []
for n, (routed, shared, tokens) in enumerate([(12, 12, 1), (16, 12, 4), (16, 12, 23), (16, 16, 24), (10, 12, 9), (12, 12, 70), (10, 10, 300), (0, 0, 5)]):
    hidden = 2048 if n == 3 else 1024               # the two layers on the four-row kernels differ in the shared memory they ask for
    spec = synth.make_layer(50 + n, routed_type=routed, shared_type=shared, hidden=hidden, inter=512, shared_inter=512, experts=24 if routed else 8, top_k=6)
    made.append((synth.activations(60 + n, tokens, hidden), MoeLayer(gpu, spec, tokens)))
seen, failed = [[] for _ in made], []
together = threading.Barrier(len(made))
def calls(i):
    x, layer = made[i]
    gpu.lib.qw4cu_set_device(0)
    together.wait()
    try:
        for _ in range(40):
            seen[i].append(layer.forward(x))
    except abi.MoeError as e:
        failed.append((i, len(seen[i]), str(e)))
threads = [threading.Thread(target=calls, args=(i,)) for i in range(len(made))]
for t in threads: t.start()
for t in threads: t.join()
assert not failed, failed
for i, (x, layer) in enumerate(made):
    alone = layer.forward(x)
    for turn, got in enumerate(seen[i]):
        for a, b in zip(got, alone):
            np.testing.assert_array_equal(a, b, err_msg=f"layer {i}, call {turn}")
print("same bits")
"""


def test_first_calls_of_many_threads(gpu):
    done = subprocess.run([sys.executable, "-c", PROGRAM], cwd=Path(__file__).parent.parent, capture_output=True, text=True, timeout=180)
    assert done.returncode == 0 and "same bits" in done.stdout, done.stdout + done.stderr[-3000:]

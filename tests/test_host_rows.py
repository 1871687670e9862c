"""The host calls' memory, threads and row ring (picoforge_b200/csrc/moe_host.c) on a stand-in for the CUDA shim whose copies
are carried out as late as their events allow (tests/host_rows_harness.c): no GPU is needed, and none is used."""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_rows") / "host_rows"
    subprocess.run([shutil.which("gcc") or "gcc", "-std=c11", "-O2", "-Wall", "-Wextra", "-D_DEFAULT_SOURCE", f"-I{HERE.parent / 'include'}",
                    str(HERE / "host_rows_harness.c"), "-o", str(out), "-lm", "-lpthread", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return out


def run(harness, *args, cores=None):
    pin = (lambda: os.sched_setaffinity(0, cores)) if cores else None
    done = subprocess.run([str(harness), *map(str, args)], capture_output=True, text=True, timeout=120, preexec_fn=pin)
    assert done.returncode == 0, (done.returncode, done.stderr)
    return [int(v) for v in done.stdout.split()]


@pytest.mark.parametrize("tokens,hidden,xpad,ypad", [
    (40, 2048, 0, 0),                  # the ring, without helpers
    (333, 2048, 3, 17),                # slices of four rows, pitches larger than a row: the ring turns once and a third
    (4096, 2048, 5, 1),                # sixteen turns
    (5000, 512, 1, 5),                 # a second launch sequence of 904 tokens
    (9000, 64, 7, 1),                  # rows far smaller than a slice; a last sequence that fits the pinned block
    (333, 8191, 0, 2),                 # one odd row to a slice
    (3, 200000, 1, 0),                 # rows larger than a slice: a ring of eight rows
    (100, 200000, 0, 1),
])
def test_rows_come_and_go_through_the_ring(harness, tokens, hidden, xpad, ypad):
    """Twice, with other values: y = 2 x + 1 of every row, the bytes between the rows untouched, ids and weights of every token."""
    wrong, _, _, _ = run(harness, "rows", tokens, hidden, xpad, ypad, 2)
    assert wrong == 0


def test_no_signal_of_the_process_reaches_a_helper_thread(harness):
    """Helpers are there, none of them would handle a signal that is sent to the process, and the caller's own mask is as it was."""
    cores = os.sched_getaffinity(0)
    wrong, threads, open_to_signals, mask_changed = run(harness, "rows", 333, 2048, 0, 0, 20)
    assert wrong == 0 and threads == 1 + min(5, len(cores) - 1)
    assert open_to_signals == 0 and mask_changed == 0


@pytest.mark.parametrize("cores", [1, 2, 3])
def test_no_more_threads_than_the_caller_has_cores(harness, cores):
    mine = sorted(os.sched_getaffinity(0))
    if len(mine) < cores:
        pytest.skip("fewer cores here")
    wrong, threads, _, _ = run(harness, "rows", 333, 2048, 0, 0, 10, cores=mine[:cores])
    assert wrong == 0 and threads == cores


@pytest.mark.parametrize("cap,hidden", [(1, 2048), (15, 2048), (16, 2048), (8192, 2048), (2**62, 2048), (64, 8), (2, 200000)])
def test_a_workspace_stays_within_the_host_bytes_it_asks_for(harness, cap, hidden):
    asked, held, refused = run(harness, "budget", cap, hidden)
    assert held <= asked
    assert asked - held <= 64                                  # and asks for little more than that
    assert refused == 10                                       # QW4_CAPACITY with one byte less


def test_digits_and_halves_of_a_row_share_their_room(harness):
    """4096 tokens of the benchmark's layer: x, act and shared act as halves (4 bytes a value) and not as digits beside them."""
    cap, h, e, k, i = 4096, 2048, 512, 10, 512
    bytes_, = run(harness, "device", cap, h, e, k, i)
    values = cap * h + cap * k * i + cap * i                   # x, routed and shared activations
    # staging, logits, outputs and the like; the halves; their sums and scales (an eighth to a quarter of the values' count, in words)
    rest = 4 * (2 * cap * h + 2 * cap * e + cap * k * h + cap * h + cap * k * i + cap * i)
    assert rest + 4 * values < bytes_ < rest + 4 * values + values + (8 << 20)

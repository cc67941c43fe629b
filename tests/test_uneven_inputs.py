"""What an uneven batch's call sees of its inputs, and holds of them: each array
as it was at one time, although other Python threads may write to it, and no
more than a bounded amount of converted copies."""

from __future__ import annotations

import sys
import threading
import tracemalloc

import numpy as np
import pytest

N, COUNT = 256, 200  # 0.5 MB an array in FP64, 105 MB together


def peak_of_call(forcing) -> int:
    import darcy_cpp_gb300 as darcy

    fields = [np.full((N, N), 2.0)] * COUNT
    tracemalloc.start()
    try:
        darcy.solve_batch_uneven(fields, forcing, max_iter=1, x0=forcing)
    except RuntimeError:  # no GPU here: the inputs have been packed by then
        pass
    peak = tracemalloc.get_traced_memory()[1]
    tracemalloc.stop()
    return peak


def test_converted_forcings_and_starts_are_not_all_held_at_once() -> None:
    """FP32 forcings and starts need FP64 copies, 210 MB of them. Beyond what
    the call with FP64 arrays (no copies) traces, the solutions included, at
    most two bounded sets of 32 MB and an array each may be alive."""
    plain = peak_of_call([np.ones((N, N))] * COUNT)
    converted = peak_of_call([np.ones((N, N), dtype=np.float32)] * COUNT)
    assert converted - plain < (72 << 20)


@pytest.mark.gpu
def test_fields_written_by_another_thread_are_seen_whole() -> None:
    """A thread rewrites every field, one assignment each (under the GIL), with
    ones and twos in turn: every problem is the one of ones or the one of twos,
    whose iterates are half as large (exactly: a power of two), and nothing in
    between. Tolerance: launch shapes differ, so sums round differently."""
    import darcy_cpp_gb300 as darcy

    n, count = 256, 150  # 79 MB, packed by several threads; too few problems for the shape tuner
    ones = np.ones((n, n))
    u1 = darcy.solve_batch_uneven([ones], max_iter=1).u[0]
    fields = [ones.copy() for _ in range(count)]
    views = [memoryview(a).cast("B") for a in fields]
    values = [ones.tobytes(), (2 * ones).tobytes()]
    stop = threading.Event()

    def write() -> None:
        k = 0
        while not stop.is_set():
            k += 1
            for v in views:
                v[:] = values[k & 1]

    writer = threading.Thread(target=write)
    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-4)
    writer.start()
    try:
        for _ in range(6):
            got = darcy.solve_batch_uneven(fields, max_iter=1)
            for u in got.u:
                error = min(np.abs(u - u1).max(), np.abs(u - 0.5 * u1).max())
                assert error < 1e-10 * np.abs(u1).max()
    finally:
        stop.set()
        writer.join()
        sys.setswitchinterval(interval)

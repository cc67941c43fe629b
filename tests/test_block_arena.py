"""Scratch of the batched engine's CTAs in batches of several sides. A CTA takes
problems of all of them in turn and lays its arena out anew for each, so the
arenas are as far apart as the neediest side wants: a side just below 8 * 2^k
(whose dense tail has 64 columns) can want more than one just above (36).

Tolerance of the solutions: both batches stop at a relative residual of 1e-12
and differ in launch shape only; as in test_block_engine.py, 1e-9.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from conftest import ROOT, two_phase

LIMIT = 383  # the largest side that batches solve by one CTA
BUDGETS = [kb << 10 for kb in (0, 32, 48, 96, 100, 180)]  # every shared-memory budget the tuner tries


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("budget", BUDGETS)
def test_arenas_hold_every_pair_of_sides(budget, mixed) -> None:
    import __graft_entry__

    builder = __graft_entry__._builder()
    if not builder.LIB.exists():
        builder.build()
    lib = ctypes.CDLL(str(builder.LIB))
    need = lib["_ZN4dgpu17block_arena_bytesEibm"]  # dgpu::block_arena_bytes(int, bool, size_t)
    need.argtypes, need.restype = [ctypes.c_int, ctypes.c_bool, ctypes.c_size_t], ctypes.c_size_t
    stride = lib["_ZN4dgpu18block_arena_strideEPKilbm"]  # dgpu::block_arena_stride(const int*, int64_t, bool, size_t)
    stride.argtypes = [ctypes.POINTER(ctypes.c_int), ctypes.c_int64, ctypes.c_bool, ctypes.c_size_t]
    stride.restype = ctypes.c_size_t
    want = [0] + [need(n, mixed, budget) for n in range(1, LIMIT + 1)]
    beyond = 0
    for small in range(1, LIMIT):
        for large in range(small + 1, LIMIT + 1):
            got = stride((ctypes.c_int * 2)(small, large), 2, mixed, budget)
            assert got % 256 == 0 and got >= max(want[small], want[large])
            beyond += want[small] > want[large]
    assert beyond  # pairs whose smaller side wants more


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("sides", [range(13, 25), range(25, 45), (64, 65, 63, 70, 128, 129)])
def test_batches_of_such_sides_solve_every_problem(monkeypatch, tmp_path, sides, form) -> None:
    from darcy_cpp_gb300 import capi

    # (launch shapes tuned for these batches are not for others of the same size bucket)
    monkeypatch.setenv("DARCY_GPU_TUNE_FILE", str(tmp_path / "tune.json"))
    ctx = capi.Context()
    sides = list(sides)
    fields = {n: np.stack([two_phase(n, seed=s) for s in range(3)]) for n in sides}
    want = {n: ctx.solve_batch(a, tol=1e-12, form=form)["u"] for n, a in fields.items()}
    order = [(n, q) for q in range(3) for n in sides]
    count = 3000 if max(sides) < 60 else 1400  # more problems than CTAs are resident
    batch = [order[q % len(order)] for q in range(count)]
    got = ctx.solve_uneven([fields[n][q] for n, q in batch], f_scalar=1.0, tol=1e-12, form=form)
    assert got["converged"].all()
    for u, (n, q) in zip(got["u"], batch):
        w = want[n][q]
        assert np.linalg.norm(u - w) < 1e-9 * np.linalg.norm(w)

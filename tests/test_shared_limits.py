"""The dynamic shared-memory limit of a kernel belongs to the function, not to
a context, network or thread: callers that need different amounts must not
take it from one another."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["tensor", "simt"])
def test_a_smaller_network_leaves_a_larger_one_usable(engine) -> None:
    from darcy_cpp_gb300 import learn

    def step(net, side):
        a = np.stack([two_phase(side, seed=s) for s in range(2)])
        net.set_scaling([float(np.log(a).mean()), 1.0, 1e-2, 1.0])
        grads, _ = net.handle.gradients(a, np.full_like(a, 1e-2))
        return net.predict(a), grads

    def made(side):
        net = learn.WarmStartNet(side, seed=1)
        net.handle.set_engine(engine)
        return net

    alone = {side: step(made(side), side) for side in (16, 256)}
    nets = {side: made(side) for side in (256, 16)}  # the larger one first
    for side in (16, 256, 16):
        for got, want in zip(step(nets[side], side), alone[side]):
            assert np.array_equal(got, want)


def test_fields_of_two_sides_from_two_threads() -> None:
    from darcy_cpp_gb300 import capi

    want = {n: capi.random_fields(n, 3, seed=4) for n in (128, 8)}
    errors: list[Exception] = []

    def work(n: int) -> None:
        try:
            for _ in range(300):
                assert np.array_equal(capi.random_fields(n, 3, seed=4), want[n])
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    run_together(work, (128, 8))
    assert not errors, errors[0]


def test_solves_of_two_sides_from_two_contexts() -> None:
    """New plans all the time (the sweep counts are part of a plan's key), so
    that the kernel that builds the dense coarse operator is launched with the
    largest and the smallest need by both threads at once."""
    from darcy_cpp_gb300 import capi

    a = {n: two_phase(n, seed=1) for n in (32, 3)}
    errors: list[Exception] = []

    def work(n: int) -> None:
        try:
            ctx = capi.Context()
            for k in range(600):
                r = ctx.solve(a[n], pre_sweeps=1 + k % 5, post_sweeps=1 + k % 7)
                assert r["converged"]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    run_together(work, (32, 3, 3, 3))
    assert not errors, errors[0]


def test_batches_of_two_shapes_from_two_contexts() -> None:
    """The batched kernel's default shapes below and above side 256."""
    from darcy_cpp_gb300 import capi

    a = {n: two_phase(n, seed=1)[None] for n in (256, 8)}
    errors: list[Exception] = []

    def work(n: int) -> None:
        try:
            ctx = capi.Context()
            for _ in range(400 if n == 256 else 4000):
                assert ctx.solve_batch(a[n], form="mixed", max_iter=2)["iterations"][0] == 2
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    run_together(work, (256, 8, 8))
    assert not errors, errors[0]


def run_together(work, args) -> None:
    threads = [threading.Thread(target=work, args=(n,)) for n in args]
    for t in threads:
        t.start()
    for t in threads:
        t.join()

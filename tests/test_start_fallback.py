"""Predicted starts that are unusable: not finite, or beyond what the FP32 cycle
holds. The batched engine's passes multiply the neighbours of boundary cells by
zero faces instead of skipping them, so nothing that such a start's cycle left
behind may reach the zero start's.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def darcy():
    import darcy_cpp_gb300

    return darcy_cpp_gb300


def rel_l2(x, y) -> float:
    return float(np.linalg.norm(np.asarray(x) - np.asarray(y)) / max(np.linalg.norm(y), 1e-300))


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("start", ["not finite", "overflows FP32"])
@pytest.mark.parametrize("side", [8, 32, 34, 66])
def test_learned_start_that_is_not_usable_falls_back_to_zero(darcy, side, start, form) -> None:
    """As test_learn.py's fallback, with predictions that are not finite (the
    weights' activations overflow) or finite beyond what the FP32 cycle holds:
    every problem takes the zero start's iterations and ends at its solution
    (the same arithmetic from the fallback on, so to rounding of the sums)."""
    from darcy_cpp_gb300 import learn

    a = np.stack([two_phase(side, seed=s) for s in range(6)])
    net = learn.WarmStartNet(side, seed=5)
    scale = 1e38 if start == "overflows FP32" else 1.0
    net.set_scaling([float(np.log(a).mean()), float(np.log(a).std()) or 1.0, scale, 1.0])
    w = np.random.default_rng(2).standard_normal(net.num_params).astype(np.float32) * 0.2
    net.set_params(w * np.float32(1e30) if start == "not finite" else w)
    u0 = net.predict(a)
    assert np.isfinite(u0).all() == (start == "overflows FP32") and not (np.abs(u0) < 1e30).all()
    warm = learn.solve_batch_learned(net, a, tol=1e-10, form=form)
    zero = darcy.solve_batch(a, tol=1e-10, form=form)
    assert warm.all_converged
    assert np.array_equal(warm.iterations, zero.iterations)
    for q in range(len(a)):
        assert rel_l2(warm.u[q], zero.u[q]) < 1e-12

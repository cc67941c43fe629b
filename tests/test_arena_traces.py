"""Problems that leave non-finite values in their CTA's arena and end with a
finite residual all the same: the next problem of the same side, which takes
the arena over as it is laid out, must not see them (its passes multiply the
neighbours of boundary cells by zero faces, and 0 * NaN is NaN).
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx(monkeypatch, tmp_path):
    """A context of its own: launch shapes tuned for these batches are not for
    others of the same size bucket."""
    from darcy_cpp_gb300 import capi

    monkeypatch.setenv("DARCY_GPU_TUNE_FILE", str(tmp_path / "tune.json"))
    return capi.Context()


def rel_l2(x, y) -> float:
    return float(np.linalg.norm(np.asarray(x) - np.asarray(y)) / max(np.linalg.norm(y), 1e-300))


def overflowing_later(ctx):
    """A field, a forcing and a number of iterations after which the FP32 cycle
    overflows for the first time: permeabilities a factor of up to 1e10 apart
    from cell to cell and a point source, so that the residual grows in the
    first iterations, at a magnitude just below where the first cycle does."""
    n, rng = 24, np.random.default_rng(14)
    a = 1e3 * 10.0 ** rng.uniform(-5, 5, (n, n))
    source = np.zeros((n, n))
    source.flat[rng.integers(n * n)] = 1.0
    forcings = [10.0**m * source for m in np.arange(39.6, 40.9, 0.1)]
    got = ctx.solve_uneven([a] * len(forcings), forcings, max_iter=100, form="mixed")
    later = [(f, int(it)) for f, it, c in zip(forcings, got["iterations"], got["converged"]) if not c and 0 < it < 100]
    assert later, "no magnitude overflows later"
    return a, *later[len(later) // 2]


def test_cycle_that_overflows_after_the_last_iteration_leaves_no_trace(ctx) -> None:
    bad, source, last = overflowing_later(ctx)
    n, count = len(bad), 4200
    sound, ones = two_phase(n, seed=1), np.ones((n, n))
    want = ctx.solve_batch(sound[None], max_iter=last, form="mixed")
    got = ctx.solve_uneven([sound if q % 2 else bad for q in range(count)],
                           [ones if q % 2 else source for q in range(count)], max_iter=last, form="mixed")
    assert np.isfinite(got["residuals"]).all()
    for q in range(1, count, 2):
        assert got["iterations"][q] == last and rel_l2(got["u"][q], want["u"][0]) < 1e-12


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_zero_forcing_on_overflowing_coefficients_leaves_no_trace(ctx, form) -> None:
    """Coefficients below FP32's range overflow the dense tail's reciprocals;
    with a zero forcing such a problem is solved (u = 0) without a cycle."""
    n, count = 24, 4200
    tiny, sound = np.full((n, n), 1e-44), two_phase(n, seed=1)
    fields = [tiny if q % 2 == 0 else sound for q in range(count)]
    forcing = [np.full((n, n), float(q % 2)) for q in range(count)]
    got = ctx.solve_uneven(fields, forcing, form=form)
    want = ctx.solve_batch(sound[None], form=form)
    assert got["converged"].all()
    for q in range(count):
        if q % 2:
            assert rel_l2(got["u"][q], want["u"][0]) < 1e-9
        else:
            assert got["iterations"][q] == 0 and not got["u"][q].any()

"""The unfused level kernels of even sides (a thread per 2 x 2 aggregate) where
their tiles can go wrong: one aggregate, sides at and beside whole tiles of 64
x 16 cells, odd coarse levels under even ones (those keep the other kernels).
Two sweeps a side take no fused visit, so every level above the dense tail runs
them. One preconditioner application against the oracle; the FP32 cycle against
the FP64 one.

Tolerances: those of tests/test_fused_visits.py, derived for the same cycle;
twice the sweeps are twice the roundings, and the smoother damps their errors.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [34, 36, 62, 64, 66, 126, 128, 130, 144, 254, 258, 322])
def test_even_levels_at_tile_edges(orc, n) -> None:
    import darcy_cpp_gb300 as darcy

    a = two_phase(n, seed=n)
    r = np.random.default_rng(n).standard_normal((n, n))
    sweeps = {"pre_sweeps": 2, "post_sweeps": 2}
    want = orc.apply_preconditioner(a, r, **sweeps)
    got = darcy.apply_preconditioner(a, r, **sweeps)
    assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want)
    mixed = darcy.apply_preconditioner(a, r, form="mixed", **sweeps)
    assert np.linalg.norm(mixed - want) < 1e-5 * np.linalg.norm(want)

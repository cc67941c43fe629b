"""The fused level visits where their tiles can go wrong: sides just below, at
and above whole 8 x 16 and 16 x 32 tiles, odd sides (aggregates with cells
outside the domain, whose staged neighbours are inside), on the finest level
and, through the hierarchy, on coarser ones. One preconditioner application
against the oracle; the FP32 cycle against the FP64 one.

Tolerances: FP64 1e-12 as in tests/test_gpu_parity.py. FP32: smoothing and
transfers round at 6e-8, restricted residuals are double-float, a contrast-4
operator's cycle has ~1e2 such roundings in a row: 1e-5.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cycle", [1, 2])
@pytest.mark.parametrize("n", [33, 39, 40, 41, 47, 49, 63, 65, 127, 129, 255, 257, 271, 289, 514])
def test_visits_at_tile_edges(orc, n, cycle) -> None:
    import darcy_cpp_gb300 as darcy

    a = two_phase(n, seed=n)
    r = np.random.default_rng(n).standard_normal((n, n))
    want = orc.apply_preconditioner(a, r, cycle_index=cycle)
    got = darcy.apply_preconditioner(a, r, cycle_index=cycle)
    assert np.linalg.norm(got - want) < 1e-12 * np.linalg.norm(want)
    mixed = darcy.apply_preconditioner(a, r, cycle_index=cycle, form="mixed")
    assert np.linalg.norm(mixed - want) < 1e-5 * np.linalg.norm(want)

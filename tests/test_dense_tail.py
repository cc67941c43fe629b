"""The dense coarse-tail operator's columns kernel at the sides where its
column blocks, padded levels and bottom can go wrong: the whole hierarchy in
the tail (side <= 32, M is that one matrix), odd and even tail sides, column
counts that do not fill the last block, more sweeps, V and W cycles. One
preconditioner application against the oracle.

Tolerance: as tests/test_gpu_parity.py's (1e-12): a cycle is ~1e3 dependent
FP64 operations on terms of a contrast-4 operator, ~1e3 eps relative.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu

REL = 1e-12


@pytest.mark.parametrize("options", [{}, {"cycle_index": 1}, {"pre_sweeps": 3, "post_sweeps": 2}])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 9, 13, 25, 31, 32, 34, 49, 63])
def test_tail_operator_matches_the_oracle(orc, n, options) -> None:
    import darcy_cpp_gb300 as darcy

    a = two_phase(n, seed=n) if n > 1 else np.full((1, 1), 2.5)
    r = np.random.default_rng(n).standard_normal((n, n))
    want = orc.apply_preconditioner(a, r, **options)
    got = darcy.apply_preconditioner(a, r, **options)
    assert np.linalg.norm(got - want) < REL * np.linalg.norm(want)

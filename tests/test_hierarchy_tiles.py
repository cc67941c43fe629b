"""The hierarchy where its kernels' splits can go wrong: fine levels just
below, at and above whole tiles of 32 x 8 cells, chains of coarse levels that
begin at, above and below the level one CTA takes over (side 32). Bit for bit
against the oracle: faces and their sums are rounded in one order only.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 7, 8, 9, 31, 32, 33, 39, 63, 127, 128, 129, 161])
def test_hierarchy_at_tile_edges(orc, n) -> None:
    import darcy_cpp_gb300 as darcy

    a = np.exp(np.random.default_rng(n).normal(0.0, 2.0, (n, n)))
    got = darcy._core.hierarchy(a)
    off = 0
    for level in orc.hierarchy(a):
        m = level["e"].size
        for q, k in enumerate(("e", "w", "n", "s", "diag", "inv_diag")):
            part = got[off + q * m: off + (q + 1) * m].reshape(level[k].shape)
            assert np.array_equal(part, level[k]), (n, k)
        off += 6 * m
    assert off == got.size


@pytest.mark.parametrize("n", [9, 33, 65])
def test_first_invalid_cell_is_named(n) -> None:
    import darcy_cpp_gb300 as darcy

    for pos in (0, n * n // 2, n * n - 1):
        a = np.ones((n, n))
        a.flat[[pos, n * n - 1]] = np.nan, -1.0
        with pytest.raises(ValueError, match=rf"flat index {pos}$"):
            darcy.solve(a)

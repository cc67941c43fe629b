"""The batched engine's padded level layout (csrc/patch.cuh) where it can go
wrong: sides whose levels are odd, even or below the dense tail, every option
that takes its own path through the cycle, a CTA that moves between layouts,
and a problem whose non-finite values stay behind in a CTA's arena.

Tolerance: both solvers stop at a relative residual of 1e-12; the operator's
conditioning (~n^2 contrast / pi^2 below 1e5 here) bounds the relative
difference of the two solutions by ~2e-12 sqrt(1e5) in the energy norm, so
1e-9 in the L2 norm leaves room for the norm's own factor.
"""

from __future__ import annotations

import numpy as np
import pytest

from conftest import two_phase

pytestmark = pytest.mark.gpu

REL_L2 = 1e-9


def rel_l2(x, y) -> float:
    return float(np.linalg.norm(np.asarray(x) - np.asarray(y)) / max(np.linalg.norm(y), 1e-300))


@pytest.fixture(scope="module")
def darcy():
    import darcy_cpp_gb300

    return darcy_cpp_gb300


def field(n: int, seed: int) -> np.ndarray:
    return two_phase(n, seed=seed) if n > 1 else np.full((1, 1), 3.0 + seed)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 10, 17, 31, 34, 57, 66, 97])
def test_padded_levels_match_the_oracle(darcy, orc, n, form) -> None:
    a = np.stack([field(n, s) for s in range(2)])
    got = darcy.solve_batch(a, tol=1e-12, form=form)
    assert got.all_converged
    for q in range(2):
        assert rel_l2(got.u[q], orc.solve(a[q], tol=1e-12)["u"]) < REL_L2


@pytest.mark.parametrize("options", [{"cycle_index": 1}, {"pre_sweeps": 2, "post_sweeps": 3},
                                     {"preconditioner": "jacobi"}, {"preconditioner": "none"}])
@pytest.mark.parametrize("n", [6, 33])
def test_options_match_the_oracle(darcy, orc, n, options) -> None:
    a = field(n, 5)
    got = darcy.solve_batch(a[None], tol=1e-12, **options)
    want = orc.solve(a, tol=1e-12, **options)
    assert got.all_converged and abs(int(got.iterations[0]) - want["iterations"]) <= 2
    assert rel_l2(got.u[0], want["u"]) < REL_L2


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("options", [{}, {"cycle_index": 1}, {"pre_sweeps": 3, "post_sweeps": 2}])
@pytest.mark.parametrize("n", [4, 5, 12, 16])
def test_dense_tails_match_the_oracle(darcy, orc, n, options, form) -> None:
    """The dense tail from its first level down to side 2, which one thread
    solves for a column: directly below it, and one or two levels below."""
    a = field(n, 7)
    got = darcy.solve_batch(a[None], tol=1e-12, form=form, **options)
    assert got.all_converged
    assert rel_l2(got.u[0], orc.solve(a, tol=1e-12, **options)["u"]) < REL_L2


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_layout_changes_and_broken_neighbours_leave_no_trace(darcy, form) -> None:
    """Thousands of small problems of two sides, a third of them with a
    non-finite forcing: every CTA meets both sides and broken problems, and
    each sound problem must come out as it does in a batch of its own."""
    sides = [12, 9]
    fields = [field(n, s) for n in sides for s in range(3)]
    count = 4200
    batch = [fields[q % len(fields)] for q in range(count)]
    forcing = [np.ones_like(a) for a in batch]
    for q in range(0, count, 3):
        forcing[q] = forcing[q].copy()
        forcing[q][q % 5, 1] = np.inf if q % 2 else np.nan
    got = darcy.solve_batch_uneven(batch, forcing, form=form)
    for q, a in enumerate(batch):
        if q % 3 == 0:
            assert not got.converged[q] and got.iterations[q] == 0 and not got.u[q].any()
        else:
            assert got.converged[q]
    want = [darcy.solve(a).u for a in fields]
    for q in (1, 2, 500, 1999, count - 1):
        if q % 3:
            assert rel_l2(got.u[q], want[q % len(fields)]) < REL_L2


def test_packed_inputs_reach_their_problems(darcy) -> None:
    """Fields, forcings and starts of an uneven batch large enough to be packed
    by several threads (blocks end inside problems): each problem comes out as
    in a batch of its own, packed by one."""
    sides = [97, 33, 130, 64, 181, 1, 150, 77] * 6
    a = [field(n, s) for s, n in enumerate(sides)]
    rng = np.random.default_rng(3)
    f = [rng.standard_normal((n, n)) if s % 3 else 2.0 + s for s, n in enumerate(sides)]
    x0 = [rng.standard_normal((n, n)) * 1e-3 for n in sides]
    assert sum(x.nbytes for x in a) > 4 << 20
    got = darcy.solve_batch_uneven(a, f, tol=1e-12, x0=x0)
    for q in range(0, len(sides), 5):
        want = darcy.solve_batch_uneven([a[q]], [f[q]], tol=1e-12, x0=[x0[q]])
        assert rel_l2(got.u[q], want.u[0]) < REL_L2

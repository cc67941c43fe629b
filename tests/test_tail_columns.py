"""Columns of the dense tail operator that a CTA builds (host rule): one wave of
CTAs where up to eight columns each allow it, and never more than its shared
memory holds, whatever the number of SMs."""

from __future__ import annotations

import ctypes

import pytest

LEVELS = {n: [n] for n in range(1, 33)}
for n, sides in LEVELS.items():
    while sides[-1] > 1:
        sides.append((sides[-1] + 1) // 2)


@pytest.fixture(scope="module")
def columns():
    import __graft_entry__

    builder = __graft_entry__._builder()
    if not builder.LIB.exists():
        builder.build()
    # dgpu::tail_columns_per_cta(const int* sides, int l0, int nlev, int N, int sms)
    f = ctypes.CDLL(str(builder.LIB))["_ZN4dgpu20tail_columns_per_ctaEPKiiiii"]
    f.argtypes = [ctypes.POINTER(ctypes.c_int)] + [ctypes.c_int] * 4
    return lambda n, sms: f((ctypes.c_int * len(LEVELS[n]))(*LEVELS[n]), 0, len(LEVELS[n]), n * n, sms)


def shared_bytes(n: int, per: int) -> int:
    """Per level of padded side p: e, nf, d, 1/d (p^2 doubles each, guards of 2
    and p) and, a column, x and b (p^2 + 2 p, a guard of p each)."""
    total = 0
    for side in LEVELS[n]:
        p = 2 * ((side + 1) // 2)
        total += 4 * p * p + 2 + p + 2 * (p + per * (p * p + 2 * p))
    return 8 * total


@pytest.mark.parametrize("n", LEVELS)
def test_columns_fill_a_wave_and_fit(columns, n) -> None:
    for sms in (1, 16, 76, 108, 132, 148, 152, 160, 192, 304, 1024):
        per = columns(n, sms)
        wave = -(-n * n // sms)
        assert 1 <= per <= 8 and shared_bytes(n, per) <= 224 << 10
        assert per == min(8, wave) or shared_bytes(n, per + 1) > 224 << 10
    assert columns(32, 152) == 7

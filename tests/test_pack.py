"""Packing an uneven batch's arrays (csrc/pack.h), compiled on its own: every
number in its place at the sizes where one or several threads pack, and no
abort when memory runs out while the threads are started (the ones there are
pack everything) or before (an exception the caller can catch)."""

from __future__ import annotations

import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <new>

#include "pack.h"

static std::atomic<int> left{1 << 30};  // allocations until they fail
void* operator new(std::size_t n) {
    if (left.fetch_sub(1) <= 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

using namespace dgpu;

// pieces of odd lengths, every third a constant
static bool packed_right(std::size_t total, int allocations, bool& thrown) {
    std::vector<double> src(total), dst(total, -1.0);
    for (std::size_t k = 0; k < total; ++k) src[k] = (double)k;
    std::vector<Piece> pieces;
    for (std::size_t at = 0, q = 0; at < total; ++q) {
        const std::size_t len = std::min(total - at, 1 + q * 977 % 70001);
        pieces.push_back(q % 3 == 2 ? Piece{nullptr, 0.5, len} : Piece{src.data() + at, 0.0, len});
        at += len;
    }
    thrown = false;
    left = allocations;
    try {
        pack(pieces, dst.data());
    } catch (const std::bad_alloc&) {
        thrown = true;
    }
    left = 1 << 30;
    if (thrown) return true;
    std::size_t at = 0;
    for (const Piece& p : pieces)
        for (std::size_t k = 0; k < p.len; ++k, ++at)
            if (dst[at] != (p.src ? (double)at : p.value)) return false;
    return at == total;
}

int main() {
    bool thrown;
    const std::size_t alone = kPackAlone / sizeof(double);  // from here on several threads
    for (std::size_t total : {std::size_t(1), kPackBlock - 1, kPackBlock + 1, alone - 1, alone, 3 * alone + 5})
        if (!packed_right(total, 1 << 30, thrown) || thrown) return 1;
    for (int allocations = 0; allocations < 24; ++allocations) {
        if (!packed_right(2 * alone + 3, allocations, thrown)) return 2;
        if (thrown && allocations >= 2) return 3;  // (its own two tables; threads are not worth an exception)
    }
    return 0;
}
"""


def test_packing_is_right_and_survives_a_lack_of_memory(tmp_path) -> None:
    source, program = tmp_path / "pack.cpp", tmp_path / "pack"
    source.write_text(PROGRAM)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-pthread", "-I",
                    str(ROOT / "darcy_cpp_gb300" / "csrc"), str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0

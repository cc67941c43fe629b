// Several arrays laid out one after another, by several host threads.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <thread>
#include <vector>

namespace dgpu {

// One stretch of a packed array: `len` numbers copied from src, or `value` where src is null.
struct Piece {
    const double* src;
    double value;
    size_t len;
};

// Lay the pieces one after another into dst. By one thread this is a core's
// memory bandwidth and the first touch of dst's pages, ~14 GB/s, while the GPU
// waits: on GB300's Arm host a call with 640 fields of 78 MB took 20.5 ms with
// one thread, 17.7 with 2, 16.4 with 4, 15.9 with 8 and with 16. Below
// kPackAlone bytes one thread packs: starting the others costs ~50 us (0.77 MB:
// 1.24 ms a call alone, 1.28 with 8), what they save at ~1 MB.
constexpr size_t kPackThreads = 8, kPackAlone = size_t(4) << 20, kPackBlock = size_t(1) << 15;
inline void pack(const std::vector<Piece>& pieces, double* dst) {
    std::vector<size_t> at(pieces.size() + 1, 0);  // where each piece begins
    for (size_t q = 0; q < pieces.size(); ++q) at[q + 1] = at[q] + pieces[q].len;
    const size_t total = at.back(), blocks = (total + kPackBlock - 1) / kPackBlock;
    std::atomic<size_t> next{0};
    auto work = [&]() noexcept {
        for (size_t b; (b = next.fetch_add(1)) < blocks;) {
            size_t k = b * kPackBlock;
            const size_t end = std::min(total, k + kPackBlock);
            size_t q = (size_t)(std::upper_bound(at.begin(), at.end(), k) - at.begin()) - 1;
            for (; k < end; ++q) {
                const size_t n = std::min(at[q + 1], end) - k;
                if (pieces[q].src)
                    std::memcpy(dst + k, pieces[q].src + (k - at[q]), n * sizeof(double));
                else
                    std::fill_n(dst + k, n, pieces[q].value);
                k += n;
            }
        }
    };
    const size_t cores = std::max<size_t>(1, std::thread::hardware_concurrency());
    const size_t threads = total * sizeof(double) < kPackAlone ? 1 : std::min({kPackThreads, cores, blocks});
    std::vector<std::thread> helpers;
    helpers.reserve(threads);
    try {
        while (helpers.size() + 1 < threads) helpers.emplace_back(work);
    } catch (...) {  // no more threads, or no memory for one, to be had: those there are do the rest
    }
    work();
    for (std::thread& t : helpers) t.join();
}

}  // namespace dgpu

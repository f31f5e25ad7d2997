// bw_staging.h -- host copies between a batch's caller buffers and its pinned
// staging arenas, in chunks that overlap the DMA.  Host code only.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstddef>
#include <thread>
#include <vector>

namespace bw {

constexpr size_t kStageChunks = 8;  // most chunks
constexpr size_t kStageThreads = 16;

// Chunks of a copy: one per 256 KiB.  Each costs a copy, an event and a wait
// (16 products of 64 words: 97 us with eight chunks whatever the size, 50 in
// one; 16 of 1000 words 113, 68).
inline size_t stage_chunks(size_t bytes) {
    return std::min(kStageChunks, std::max<size_t>(1, bytes >> 18));
}

// A thread's part of every chunk: part t of T, by words (off(i): word offset of
// product i, off(count) the end).
template <class Off>
size_t part_begin(size_t lo, size_t hi, size_t t, size_t T, Off off) {
    const size_t w = off(lo) + (off(hi) - off(lo)) * t / T;
    while (lo < hi) {
        const size_t mid = (lo + hi) / 2;
        if (off(mid) < w) {
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    return lo;
}

// copy(i) for every product, chunk by chunk (chunk c of stage_chunks(bytes):
// products [chunk(c), chunk(c + 1))), on T threads: one set of them works through the chunks
// (started anew for each of four chunks, at most eight, the upload of 137 MB
// took 5.6-7.3 ms where its DMA takes 2.6).  before(c) runs on the caller's
// thread before chunk c may be copied, after(c) once it has been; a non-zero
// result of either ends the walk and is returned.  Threads that cannot be
// started are done without.
// A thread that waits for a chunk spins for kStageSpin, then naps for a
// sixteenth of its wait so far, at most kStageNap: on the way down it is there
// before the products are computed, and other processes' threads need the
// cores.  4096 products, 137 MB each way: 10.2 ms and 10.6 cores busy, where
// spinning throughout took 10.3 and 14.8.  (Blocked on a condition variable
// until a chunk is ready: 11.0 ms and 8.6; 256 products of 8000 words 1.2 -> 1.7
// ms, an idle core takes that long to come back.)
constexpr std::chrono::microseconds kStageSpin{250}, kStageNap{1000};

template <class Chunk, class Off, class Copy, class Before, class After>
int staged_copy(size_t bytes, Chunk chunk, Off off, Copy copy, Before before, After after) {
    using Clock = std::chrono::steady_clock;
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t chunks = stage_chunks(bytes);
    const size_t T = std::min<size_t>({kStageThreads, hw, std::max<size_t>(1, bytes >> 21)});
    std::atomic<size_t> ready{0}, parts[kStageChunks];
    for (auto& p : parts) p.store(0);
    std::atomic<bool> stop{false};
    auto part = [&](size_t c, size_t t) {
        const size_t lo = chunk(c), hi = chunk(c + 1);
        const size_t end = t + 1 == T ? hi : part_begin(lo, hi, t + 1, T, off);
        for (size_t i = part_begin(lo, hi, t, T, off); i < end; ++i) copy(i);
        parts[c].fetch_add(1, std::memory_order_release);
    };
    std::vector<std::thread> th;
    size_t started = 1;  // the caller's thread takes part 0 and those not started
    try {
        th.reserve(T);
        for (; started < T; ++started)
            th.emplace_back([&, t = started] {
                for (size_t c = 0; c < chunks; ++c) {
                    const auto t0 = Clock::now();
                    while (ready.load(std::memory_order_acquire) <= c) {
                        if (stop.load(std::memory_order_relaxed)) return;
                        const auto waited = Clock::now() - t0;
                        if (waited < kStageSpin) {
                            std::this_thread::yield();
                        } else {
                            std::this_thread::sleep_for(std::min<Clock::duration>(
                                kStageNap, waited / 16));
                        }
                    }
                    part(c, t);
                }
            });
    } catch (...) {
    }
    int rc = 0;
    for (size_t c = 0; c < chunks && !rc; ++c) {
        rc = before(c);
        if (rc) break;
        ready.store(c + 1, std::memory_order_release);
        part(c, 0);
        for (size_t t = started; t < T; ++t) part(c, t);
        // (the others finish about when this thread does)
        while (parts[c].load(std::memory_order_acquire) < T) std::this_thread::yield();
        rc = after(c);
    }
    stop.store(true);
    for (auto& x : th) x.join();
    return rc;
}

}  // namespace bw

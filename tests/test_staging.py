"""The batch's host staging copies (csrc/bw_staging.h), compiled for the host:
every product copied exactly once whatever the sizes, in chunks that follow the
bytes, errors end the walk, and threads that wait sleep -- a caller that waits 0.4 s for its DMA costs next to
no processor time."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <sys/resource.h>
#include <unistd.h>
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "bw_staging.h"

static double cpu() {
    rusage u;
    getrusage(RUSAGE_SELF, &u);
    return u.ru_utime.tv_sec + u.ru_stime.tv_sec + 1e-6 * (u.ru_utime.tv_usec + u.ru_stime.tv_usec);
}

// argv: products, bytes to claim, wait per chunk (us), failing chunk (-1: none),
// 0: in before, 1: in after
int main(int, char** v) {
    const size_t np = atoi(v[1]), bytes = strtoull(v[2], 0, 10);
    const int wait = atoi(v[3]), bad = atoi(v[4]), mode = atoi(v[5]);
    std::vector<size_t> off(np + 1, 0);
    for (size_t i = 0; i < np; ++i) off[i + 1] = off[i] + 1 + (i * 2654435761u >> 20) % 997;
    std::vector<std::atomic<int>> seen(np);
    for (auto& x : seen) x = 0;
    const double c0 = cpu();
    auto chunk = [&](size_t c) { return c * np / bw::stage_chunks(bytes); };
    auto offs = [&](size_t i) { return off[i]; };
    auto copy = [&](size_t i) { ++seen[i]; };
    int befores = 0, afters = 0;
    bool early = false, late = false;
    auto before = [&](size_t c) {
        ++befores;
        for (size_t i = chunk(c); i < np; ++i) early |= seen[i] != 0;
        if (wait) usleep(wait);
        return mode == 0 && (int)c == bad ? 7 : 0;
    };
    auto after = [&](size_t c) {
        ++afters;
        for (size_t i = 0; i < chunk(c + 1); ++i) late |= seen[i] != 1;
        return mode != 0 && (int)c == bad ? 9 : 0;
    };
    const int rc = bw::staged_copy(bytes, chunk, offs, copy, before, after);
    size_t once = 0;
    for (auto& x : seen) once += x == 1;
    printf("%d %zu %d %d %d %d %.4f\n", rc, once, befores, afters, early, late, cpu() - c0);
}
"""


@pytest.fixture(scope="module")
def staging(tmp_path_factory):
    d = tmp_path_factory.mktemp("staging")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "birdwing_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)

    def run(*args):
        p = subprocess.run([str(exe)] + [str(a) for a in args], capture_output=True, text=True,
                           timeout=60, check=True)
        f = p.stdout.split()
        return [int(x) for x in f[:6]] + [float(f[6])]

    return run


@pytest.mark.parametrize("nbytes", [0, 1 << 21, 5 << 21, 1 << 30])
@pytest.mark.parametrize("products", [1, 2, 7, 8, 9, 100, 4096])
def test_every_product_once(staging, products, nbytes):
    rc, once, befores, afters, early, late, _ = staging(products, nbytes, 0, -1, 0)
    assert (rc, once, early, late) == (0, products, 0, 0) and befores == afters


@pytest.mark.parametrize("nbytes,chunks", [(0, 1), (8192, 1), ((1 << 18) - 4, 1), (3 << 18, 3),
                                           (1 << 21, 8), (1 << 30, 8)])
def test_chunks_follow_bytes(staging, nbytes, chunks):
    # a chunk costs a copy, an event and a wait: small batches take one
    assert staging(64, nbytes, 0, -1, 0)[2:4] == [chunks, chunks]


@pytest.mark.parametrize("mode,rc", [(0, 7), (1, 9)])
@pytest.mark.parametrize("bad", [0, 3])
def test_errors_end_the_walk(staging, bad, mode, rc):
    got, _, befores, afters, _, _, _ = staging(64, 1 << 30, 0, bad, mode)
    assert (got, befores, afters) == (rc, bad + 1, bad + mode)


def test_waiting_threads_sleep(staging):
    # eight chunks of 50 ms each, 0.4 s in which nothing is to be copied: up to
    # 15 threads may spin for 0.25 ms a chunk (0.03 s) and wake some 65 times
    # (below 0.1 s at 0.1 ms each)
    assert staging(64, 1 << 30, 50000, -1, 0)[6] < 0.13

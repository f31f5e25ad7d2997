"""bw_server_prewarm leaves nothing for the first request of a length to do: it
builds the tables and loads the kernels, which are one per length."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# in a process of its own: kernels are loaded once per process
SCRIPT = """
import json, time
import numpy as np
import birdwing_b200 as bw
from birdwing_b200 import workloads
rng = np.random.default_rng(1)
extra = []
with bw.Server() as srv:
    srv.prewarm(18)

    def request_us(words, path):
        a, b = (workloads.rand_operand(rng, words) for _ in range(2))
        out = np.zeros(2 * words, np.uint32)
        t = time.perf_counter()
        srv.wait(srv.submit(a, b, out, path=path))
        return 1e6 * (time.perf_counter() - t)

    for path in (32, 64):
        for _ in range(5):
            request_us(1 << 16, path)  # the pools and the module
        for words in (10, 20, 40, 100, 200, 400, 900, 1800, 3600, 7000, 14000):
            us = [request_us(words, path) for _ in range(9)]
            extra.append(us[0] - np.median(us[1:]))
print(json.dumps(float(np.median(extra))))
"""


def test_first_request_of_a_length():
    # loading a length's kernels takes 50 us and more; without it first requests
    # measured 9 to 17 us above the ones that follow
    seen = []
    for _ in range(3):  # the host is shared: one undisturbed run is enough
        p = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True,
                           text=True, timeout=300)
        assert p.returncode == 0, p.stderr[-2000:]
        seen.append(json.loads(p.stdout.splitlines()[-1]))
        if seen[-1] < 30.0:
            return
    assert False, seen

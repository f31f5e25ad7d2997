"""The server's kernel_launches counts the kernels its groups launch: one for
single-pass lengths, four with the look-back carry (groups of at most three
tiles of 2048 words per SM), five with the words pass and its fix."""
import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import workloads

pytestmark = pytest.mark.gpu


def kernels_of(words, group_size):
    if words <= 900:
        return 1
    tiles = -(-2 * words // 2048)
    return 4 if group_size * tiles <= 3 * 148 else 5


@pytest.mark.parametrize("path", [32, 64])
@pytest.mark.parametrize("words,count", [(900, 1), (16384, 1), (32768, 1), (32768, 60), (900, 40)])
def test_kernel_launches(words, count, path):
    rng = np.random.default_rng(words + count)
    a = workloads.rand_operand(rng, words)
    b = workloads.rand_operand(rng, words)
    with bw.Server(path=path, lanes=1, max_groups=1) as srv:
        tickets = [srv.submit(a, b) for _ in range(count)]
        infos = [srv.wait(t)[1] for t in tickets]
        st = srv.stats()
    # the requests of a group all report its size
    want = sum(kernels_of(words, i["group_size"]) / i["group_size"] for i in infos)
    assert st["kernel_launches"] == round(want)
    assert count == 1 or st["max_group_size"] > 1

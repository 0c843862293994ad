"""A prepared layout is kept for the next request of the same sizes, also where
the node limit was cut to fit the kernels' shared memory.  No GPU needed: a
layout of this mesh takes tens of milliseconds to build, a kept one none."""
import time

import pytest

from femorph_b200 import api, mesh


def seconds(f):
    t = time.perf_counter()
    f()
    return time.perf_counter() - t


@pytest.mark.parametrize("threads", [128, 256])  # limits of 3,882 and 2,943 nodes
def test_repeated_prepare_builds_nothing(threads):
    g = api.GpuProblem(mesh.channel(60, 30, 30, seed=1))
    first = seconds(lambda: g.prepare(2600, 3100, threads))
    again = min(seconds(lambda: g.prepare(2600, 3100, threads)) for _ in range(5))
    assert again < first / 10
    g.check_layout(2600, 3100, threads)
    g.close()

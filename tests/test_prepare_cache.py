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


@pytest.mark.parametrize("n,tile_elems", [(32, 32), (33, 0), (40, 0)])
def test_static_solve_builds_its_layout_once(n, tile_elems):
    """196,608 tets prepared in tiles of 32, whose partials do not fit the
    static scratch; 215,622, which fit in no tiles; 384,000, whose nodes and
    elements alone do not (no layout built at all)."""
    p = mesh.cavity(n, seed=1, steps=2)
    g = api.GpuProblem(p)
    built = seconds(lambda: g.prepare(tile_elems=tile_elems))
    code = []
    call = lambda: code.append(api.lib().fm_vms_solve_static(g.h, 0, 0, None, None, None))
    first = seconds(call)
    again = min(seconds(call) for _ in range(5))
    if n == 32:
        assert code[0] in (api.FM_OK, api.FM_ERR_NODEVICE)
        assert code[0] == api.FM_OK or again < built / 10
    else:
        assert code[0] == api.FM_ERR_INVALID and again < built / 10
        assert n != 40 or first < built / 10
    g.close()

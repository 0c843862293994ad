"""A problem prepared for CTAs of 128 threads in a batch of 256: its tiles are
cut to the node limit of 256 threads, as a problem's that was not prepared."""
import numpy as np
import pytest

from femorph_b200 import api, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,then", [(128, 256), (256, 128)])
def test_prepared_for_other_threads(first, then):
    p = mesh.channel(30, 20, 12, seed=3, noise=1e-2)
    shape = dict(tile_elems=2600, tile_nodes=3100)  # 128 threads hold 3,882 nodes, 256 2,943
    out = []
    for prepared in (False, True):
        g = api.GpuProblem(p)
        if prepared:
            g.prepare(**shape, threads=first)
        b = api.Batch([g], **shape, threads=then)
        b.step(3)
        b.sync()
        out.append(g.state())
        b.close()
        g.close()
    for x, y in zip(*out):
        assert (x is None and y is None) or np.array_equal(x, y)

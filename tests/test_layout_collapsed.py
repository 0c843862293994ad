"""The layout check on hexas whose corners repeat a node (wedges written as
hexas): valid, and marked for the kernel, which adds their corners one by one.
No GPU needed."""
import numpy as np
import pytest

from femorph_b200 import api, mesh


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("tile_elems", [0, 32])
def test_collapsed_hexas_pass_the_check(tile_elems, precision):
    p = mesh.channel(9, 5, 3, seed=6)
    conn = []
    for i, c in enumerate(np.asarray(p.conn).reshape(-1, 8)):
        if i % 3:
            conn.append(c)
        else:
            conn += [c[[0, 1, 2, 2, 4, 5, 6, 6]], c[[0, 2, 3, 3, 4, 6, 7, 7]]]
    p.conn = np.ascontiguousarray(conn, dtype=p.conn.dtype)
    g = api.GpuProblem(p, precision)
    g.check_layout(tile_elems=tile_elems)
    g.close()

"""Tiles around nodes of a hundred tets each, which need most of the 128
colours: the layout spreads elements over colours, but may not run out of them
where the smallest colour that fits would do.  No GPU needed."""
import numpy as np
import pytest

from femorph_b200 import api, mesh

spatial = pytest.importorskip("scipy.spatial")


def hubs(seed):
    """Delaunay tets of a few nodes inside a sphere of points, and points
    outside it; all tets positive, fluid at rest."""
    rng = np.random.default_rng(seed)
    h, n = int(rng.integers(2, 6)), int(rng.integers(60, 150))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    near = 0.15 * rng.normal(size=(h, 3))
    far = rng.normal(size=(int(rng.choice([200, 500, 900])), 3))
    far *= (rng.uniform(1.5, 4, size=len(far)) / np.linalg.norm(far, axis=1))[:, None]
    X = np.concatenate([d, near, far])
    conn = spatial.Delaunay(X).simplices.astype(np.int32)
    a, b, c, e = (X[conn[:, i]] for i in range(4))
    flip = np.einsum("ei,ei->e", np.cross(b - a, c - a), e - a) < 0
    conn[flip] = conn[flip][:, [1, 0, 2, 3]]
    p = mesh.cavity(2, seed=1, solver=mesh.SUPG, cfl=0.05)
    p.coords, p.conn, p.init_state = X, np.ascontiguousarray(conn), np.zeros((len(X), 4))
    return p


@pytest.mark.parametrize("tile_elems,tile_nodes", [(1024, 512), (3500, 1200), (9000, 2200)])
@pytest.mark.parametrize("seed", [0, 1, 9, 13])  # the last two have three nodes of 94 to 116 tets
def test_tiles_of_high_valence_are_taken(seed, tile_elems, tile_nodes):
    p = hubs(seed)
    valence = np.bincount(p.conn.ravel())
    assert valence.max() <= 128  # more of them in one tile cannot be coloured
    g = api.GpuProblem(p)
    g.check_layout(tile_elems=tile_elems, tile_nodes=tile_nodes)
    g.close()

"""The resident CG kernel at the edges of its blocks: one CTA and several,
ragged slices, matrices that stay in shared memory and ones that stream, the
forms with two and no vectors in shared memory, and a system that it does
not take (the three-kernel iteration then).  Bar: the solution within 1e-10
of a direct solve, as test_gpu_poisson.py; systems too large for one are held
to a residual of 1e-10 in the oracle's element matrices at a CG tolerance of
1e-12 (the recursive residual drifts from the true one by rounding only)."""
import numpy as np
import pytest

from femorph_b200 import api, mesh
from oracle import oracle_b

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def box(nx, ny, nz, elem_type, seed):
    """poisson_box on nx x ny x nz cells."""
    rng = np.random.default_rng(seed)
    p = mesh.channel(nx, ny, nz, seed=seed, jitter=0.1, steps=1)
    X, conn = p.coords / np.array([4.0, 1.0, 1.0]), p.conn
    if elem_type == mesh.TET4:  # six tets a hexa around its 0-6 diagonal
        ring = (1, 2, 3, 7, 4, 5)
        conn = np.concatenate([conn[:, [0, ring[i], ring[(i + 1) % 6], 6]] for i in range(6)])
    E = conn.shape[0]
    dn = np.nonzero(X[:, 0] < 1e-12)[0].astype(np.int32)
    return mesh.PoissonProblem(X, np.ascontiguousarray(conn, np.int32), rng.uniform(0.5, 2.0, (E, 3)),
                               np.arange(0, E, 3, dtype=np.int32), rng.uniform(-1.0, 1.0, (E + 2) // 3),
                               np.zeros(1, np.int32), np.zeros(0, np.int32), np.zeros(0), dn,
                               np.sin(np.pi * X[dn, 1]))


@pytest.mark.parametrize("elem_type", [mesh.TET4, mesh.HEXA8])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 4), (15, 7, 7), (4, 4, 40), (11, 10, 9), (23, 17, 13)])
def test_against_direct_solve(dims, elem_type):
    p = box(*dims, elem_type, seed=sum(dims))
    s = api.GpuPoisson(p)
    it, rr, _ = s.solve(1e-14)
    x, _ = s.solution()
    it2, rr2, _ = s.solve(1e-14)
    x2, _ = s.solution()
    s.close()
    assert it == it2 and rr == rr2 and np.array_equal(x, x2)
    assert np.array_equal(x[p.dir_node], p.dir_value)
    xo, _ = oracle_b.poisson_solve(p)
    assert rr <= 1e-14 and rel(x, xo) <= 1e-10


def test_hub_row():
    """A fan of tets around one apex: its row has 46,226 columns, and the halo
    of the block that owns it does not fit shared memory."""
    m = 215
    g = np.linspace(-1.0, 1.0, m)
    top = np.stack(np.meshgrid(g, g, indexing="ij"), -1).reshape(-1, 2)
    X = np.concatenate([np.concatenate([top, np.ones((m * m, 1))], 1), np.zeros((1, 3))])
    i, j = np.meshgrid(np.arange(m - 1), np.arange(m - 1), indexing="ij")
    a = (i * m + j).ravel()
    tri = np.concatenate([np.stack([a, a + 1, a + m], 1), np.stack([a + m + 1, a + m, a + 1], 1)])
    conn = np.concatenate([tri, np.full((tri.shape[0], 1), m * m)], 1).astype(np.int32)
    dn = np.nonzero(np.abs(X[:, 0]) > 1.0 - 1e-12)[0].astype(np.int32)
    p = mesh.PoissonProblem(X, conn, np.ones((conn.shape[0], 3)), np.arange(0, conn.shape[0], 7, dtype=np.int32),
                            np.full((conn.shape[0] + 6) // 7, 2.0), np.zeros(1, np.int32), np.zeros(0, np.int32),
                            np.zeros(0), dn, X[dn, 1].copy())
    s = api.GpuPoisson(p)
    _, rr, _ = s.solve(1e-14)
    x, _ = s.solution()
    s.close()
    xo, _ = oracle_b.poisson_solve(p)
    assert rr <= 1e-14 and rel(x, xo) <= 1e-10


@pytest.mark.parametrize("n", [95, 110])
def test_large_systems(n):
    """884,736 and 1,367,631 rows: two vectors and none beside the direction
    in shared memory on 148 SMs."""
    p = box(n, n, n, mesh.HEXA8, seed=n)
    s = api.GpuPoisson(p)
    _, rr, _ = s.solve(1e-12)
    x, _ = s.solution()
    s.close()
    conn = oracle_b.poisson_fix(p)
    y = np.einsum("eab,eb->ea", oracle_b.poisson_elements(p, conn), x[conn])
    r = -np.bincount(conn.ravel(), y.ravel(), p.n_nodes)
    r += np.bincount(conn[p.source_elem].ravel(), oracle_b.poisson_sources(p, conn).ravel(), p.n_nodes)
    r[p.dir_node] = 0.0
    # the system's right-hand side holds the Dirichlet values too
    b = np.linalg.norm(p.dir_value)
    assert rr <= 1e-12 and np.linalg.norm(r) <= 1e-10 * b

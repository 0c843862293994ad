"""The SUPG tile kernels at the edges of their chunks (128 elements) and over
their option combinations, against the FP64 oracle.  Bars: those of
test_gpu_parity.py, velocity 1e-12 and element pressure / lambda 1e-11
relative L2 after a few steps in FP64; 1e-6 velocity in the mixed form."""
import numpy as np
import pytest

from femorph_b200 import api, mesh
from oracle import oracle_b

pytestmark = pytest.mark.gpu

STEPS = 4


def rel(a, b):
    nb = np.linalg.norm(b)
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / (nb if nb > 0 else 1.0))


def compare(p, precision, **tuning):
    g = api.GpuProblem(p, precision)
    b = api.Batch([g], **tuning)
    b.step(STEPS)
    b.sync()
    u, pr, el, _ = g.state()
    o = oracle_b.OracleSolve(p)
    o.step(STEPS)
    st, oel, _, _ = o.state()
    b.close()
    g.close()
    eu, ep, ew = rel(u, st[:, :3]), rel(pr, oel[:, 0]), rel(el[:, 0], oel[:, 1])
    if precision == api.FM_FP64:
        assert eu <= 1e-12 and ep <= 1e-11 and ew <= 1e-11, (eu, ep, ew)
    else:
        assert eu <= 1e-6, (eu, ep, ew)


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("ab2,bbar", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("dims,threads", [((1, 1, 1), 128), ((7, 5, 3), 128), ((16, 4, 2), 128), ((9, 5, 3), 256),
                                          ((13, 9, 7), 128)])
def test_hexa(dims, threads, ab2, bbar, precision):
    p = mesh.channel(*dims, seed=sum(dims), noise=1e-2, ex_opts=(1 - ab2, bbar, 1, 1, 1, 1))
    compare(p, precision, threads=threads)


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("ab2", [0, 1])
@pytest.mark.parametrize("n,threads", [(1, 128), (3, 128), (4, 256), (5, 128)])
def test_tet(n, threads, ab2, precision):
    p = mesh.cavity(n, seed=n, solver=mesh.SUPG, cfl=0.05, noise=1e-2)
    p.ex_opts = (1 - ab2, 0, 1, 1, 1, 1)
    compare(p, precision, threads=threads)


@pytest.mark.parametrize("npe", [4, 8])
@pytest.mark.parametrize("opts", [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1), (0, 1, 1, 1)])
def test_single_terms(npe, opts):
    """Each of K1..K4 alone, and all but K1."""
    p = mesh.channel(5, 4, 3, seed=2, noise=1e-2) if npe == 8 else mesh.cavity(3, seed=2, solver=mesh.SUPG, cfl=0.05,
                                                                              noise=1e-2)
    p.ex_opts = (1, 0) + opts
    compare(p, api.FM_FP64)


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("npe", [4, 8])
def test_both_integrators_in_one_batch(npe, precision):
    """Euler and AB2 problems share a batch (one launch serves both): each
    bitwise as alone in a batch of its own, where an Euler problem runs the
    kernel without the history."""
    def make(seed, euler, bbar):
        p = mesh.channel(9, 7, 6, seed=seed, noise=1e-2) if npe == 8 else mesh.cavity(5, seed=seed, solver=mesh.SUPG,
                                                                                     cfl=0.05, noise=1e-2)
        p.ex_opts = (euler, bbar, 1, 1, 1, 1)
        return p
    ps = [make(1, 1, 0), make(2, 0, 0), make(3, 1, int(npe == 8))]
    gs = [api.GpuProblem(p, precision) for p in ps]
    b = api.Batch(gs)
    b.step(20)
    b.sync()
    for p, g in zip(ps, gs):
        h = api.GpuProblem(p, precision)
        c = api.Batch([h])
        c.step(20)
        c.sync()
        for x, y in zip(g.state()[:3], h.state()[:3]):
            assert np.array_equal(x, y)
        c.close()
        h.close()


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("ab2,bbar", [(0, 0), (1, 1)])
@pytest.mark.parametrize("threads", [128, 256])
def test_collapsed_hexa(threads, ab2, bbar, precision):
    """Every third cell split into two wedges, written as hexas whose corners
    repeat a node: those are added into their nodes corner by corner."""
    p = mesh.channel(9, 5, 3, seed=6, noise=1e-2, ex_opts=(1 - ab2, bbar, 1, 1, 1, 1))
    conn = []
    for i, c in enumerate(np.asarray(p.conn).reshape(-1, 8)):
        if i % 3:
            conn.append(c)
        else:
            conn += [c[[0, 1, 2, 2, 4, 5, 6, 6]], c[[0, 2, 3, 3, 4, 6, 7, 7]]]
    p.conn = np.ascontiguousarray(conn, dtype=p.conn.dtype)
    compare(p, precision, threads=threads)


@pytest.mark.parametrize("npe,tile_elems,tile_nodes", [(4, 14000, 2700), (8, 2600, 3100)])
def test_node_limit_above_shared_memory(npe, tile_elems, tile_nodes):
    """A node limit whose tiles the kernel's shared memory does not hold
    gives smaller tiles, not an error."""
    p = mesh.channel(25, 13, 8, seed=3, noise=1e-2) if npe == 8 else mesh.cavity(14, seed=3, solver=mesh.SUPG,
                                                                                 cfl=0.05, noise=1e-2)
    compare(p, api.FM_FP64, tile_elems=tile_elems, tile_nodes=tile_nodes, threads=256)

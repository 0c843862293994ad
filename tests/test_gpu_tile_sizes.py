"""Default tiles follow the problem's size (one to four waves of CTAs, then full
tiles): solves at sizes on both sides of each line against the oracle (bars of
test_gpu_parity.py), and the same problem's bits alone, in a batch with others
and in a pool."""
import numpy as np
import pytest

from femorph_b200 import api, mesh
from oracle import oracle_b

pytestmark = pytest.mark.gpu


def rel(a, b):
    nb = np.linalg.norm(b)
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / (nb if nb > 0 else 1.0))


# 26^3 cells: 105,456 tets (256 a tile), 27^3: 118,098 (384), 33^3: 215,622 (512),
# 36^3: 279,936 (640), 37^3: 303,918 (two waves)
@pytest.mark.parametrize("n", [2, 26, 27, 33, 36, 37])
def test_vms_against_oracle(n):
    p = mesh.cavity(n, seed=n, noise=1e-2)
    g = api.GpuProblem(p)
    b = api.Batch([g])
    b.step(3)
    b.sync()
    u, pr, _, _ = g.state(elements=False)
    o = oracle_b.OracleSolve(p)
    o.step(3)
    st = o.state()[0]
    assert rel(u, st[:, :3]) <= 1e-12 and rel(pr, st[:, 3]) <= 1e-12
    b.close()
    g.close()


@pytest.mark.parametrize("dims", [(35, 37, 33), (61, 31, 31)])
def test_hexa_against_oracle(dims):
    """42,735 hexa (256 a tile) and 58,621."""
    p = mesh.channel(*dims, seed=3, noise=1e-2)
    g = api.GpuProblem(p)
    b = api.Batch([g])
    b.step(2)
    b.sync()
    u, pr, _, _ = g.state(elements=False)
    o = oracle_b.OracleSolve(p)
    o.step(2)
    st, oel, _, _ = o.state()
    assert rel(u, st[:, :3]) <= 1e-12 and rel(pr, oel[:, 0]) <= 1e-11
    b.close()
    g.close()


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
def test_alone_in_a_batch_and_in_a_pool(precision):
    ps = [mesh.cavity(n, seed=n, noise=1e-2) for n in (4, 27, 13)]
    alone = []
    for p in ps:
        g = api.GpuProblem(p, precision)
        b = api.Batch([g])
        b.step(5)
        b.sync()
        alone.append(g.state())
        b.close()
        g.close()
    gs = [api.GpuProblem(p, precision) for p in ps]
    b = api.Batch(gs)
    b.step(5)
    b.sync()
    got = [g.state() for g in gs]
    b.close()
    E, N = sum(p.n_elems for p in ps), sum(p.n_nodes for p in ps)
    pool = api.Pool(mesh.VMS, 4, max_problems=3, max_elems=E, max_nodes=N, precision=precision)
    for g in gs:
        assert pool.add(g)  # the stated maxima are room enough
    pool.step(gs, [5] * 3)
    assert not pool.wait()
    for g, a, x in zip(gs, alone, got):
        for p, q, r in zip(g.state(), a, x):
            assert np.array_equal(p, q) and np.array_equal(r, q)
    pool.close()

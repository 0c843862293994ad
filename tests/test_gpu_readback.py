"""fm_problem_get_state: every field in the problem's own order, for a problem
alone, behind others in a pool, and larger than one piece of the read-back
(349,525 elements of subscales, 1,048,576 nodes)."""
import numpy as np
import pytest

from femorph_b200 import api, mesh

pytestmark = pytest.mark.gpu


def centroid(sd):
    """The quarter-weighted sums over the Gauss points, in point order."""
    s = np.zeros((sd.shape[0], 3))
    for g in range(4):
        s += sd[:, 3 * g:3 * g + 3] * 0.25
    return s


@pytest.mark.parametrize("precision", [api.FM_FP64, api.FM_MIXED])
@pytest.mark.parametrize("n", [1, 5, 39])
def test_vms_fields(n, precision, tmp_path):
    """Every value is the one that the checkpoint file holds, whose columns the
    host permutes; 39^3 cells have 355,914 tets: two pieces of subscales."""
    p = mesh.cavity(n, seed=n, noise=1e-2)
    g = api.GpuProblem(p, precision)
    b = api.Batch([g])
    b.step(2)
    b.sync()
    u, pr, el, sd = g.state()
    path = str(tmp_path / "state.fmck")
    g.checkpoint(path)
    raw = np.fromfile(path, np.uint8)[160:]
    N, E = p.n_nodes, p.n_elems
    nodes = raw[:64 * N].view(np.float64).reshape(8, N)  # after BCs u v w p, then before
    kind = np.float32 if precision == api.FM_MIXED else np.float64
    rows = raw[64 * N:64 * N + 12 * E * kind().itemsize].view(kind).reshape(12, E)
    assert np.array_equal(u, nodes[:3].T) and np.array_equal(pr, nodes[3])
    assert np.array_equal(sd, rows.T.astype(np.float64))
    assert np.array_equal(el, centroid(sd))
    u2, p2, none_el, none_sd = g.state(elements=False)
    assert np.array_equal(u, u2) and np.array_equal(pr, p2) and none_el is None and none_sd is None
    b.close()
    g.close()


def test_initial_state_larger_than_a_piece():
    """1,061,208 nodes: the state at placement is the given one in node order
    (no boundary rows)."""
    p = mesh.channel(101, 101, 101, seed=1, noise=1.0)
    p.vel_node, p.vel_vals, p.vel_dir = np.zeros(0, np.int32), np.zeros((0, 4)), np.zeros(0, np.int32)
    p.dir_node, p.dir_vals = np.zeros(0, np.int32), np.zeros((0, 3))
    g = api.GpuProblem(p)
    b = api.Batch([g])
    u = g.state(elements=False)[0]
    assert np.array_equal(u, p.init_state[:, :3])
    b.close()
    g.close()


@pytest.mark.parametrize("solver,npe", [(mesh.VMS, 4), (mesh.SUPG, 8)])
def test_behind_others_in_a_pool(solver, npe):
    """The same fields at an offset in a pool, twice (the element map is made
    once), and again after the problem moved."""
    def make(n, seed):
        if npe == 8:
            p = mesh.channel(n + 2, n, n, seed=seed, noise=1e-2)
            p.glob_fixed = "Y"
            return p
        return mesh.cavity(n, seed=seed, noise=1e-2)
    ps = [make(3, 1), make(5, 2)]
    alone = []
    for p in ps:
        g = api.GpuProblem(p)
        b = api.Batch([g])
        b.step(3)
        b.sync()
        alone.append(g.state())
        b.close()
        g.close()
    gs = [api.GpuProblem(p) for p in ps]
    pool = api.Pool(solver, npe, max_problems=2, max_elems=20000, max_nodes=6000)
    for order in ((0, 1), (1, 0)):
        for i in order:
            assert pool.add(gs[i])
        pool.step(gs, [3, 3])
        assert not pool.wait()
        for g, ref in zip(gs, alone):
            for _ in range(2):
                for x, y in zip(g.state(), ref):
                    assert (x is None and y is None) or np.array_equal(x, y)
        for g in gs:
            pool.remove(g)
    pool.close()

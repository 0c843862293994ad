"""The work that users of this framework have it do, as timed cases.

Every case is a plain dict.  `prepare` makes what a user's program holds
before the call (mesh and boundary conditions of a seed, the problem placed on
the GPU), `run` is one pass through the public Python API (femorph_b200.api),
`work` the bytes and operations of one pass and `exact` the same results in
64-bit torch.  The kinds:

  vms      one lid-driven box of Kuhn tets, femVMSExplicitFluidSolver's step:
           advance to the next output time, then read velocity and pressure
           (with "subscales": also the Gauss-point subscales)
  batch    many independent VMS boxes of different sizes in one Batch, replayed
           from CUDA graphs
  serve    requests that join a Pool, run and leave it (continuous batching)
  supg     femSUPGExplicitFluidSolver's step on a tet box ("npe" 4) or a hexa
           channel ("npe" 8), forward Euler or AB2, with or without B-bar
  poisson  femPoissonSolver on an assembled system: one solve from x = 0 and
           the nodal solution (and the wall distance)

Time steps are small enough that a flow stays bounded however often a state
is advanced again.
"""
import itertools
import math

import numpy as np
import torch

from femorph_b200 import api, mesh

VMS_PROPS = dict(rho=1.0, inv_eps=400.0, c1=4.0, c2=2.0)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest solves of a design sweep: a coarse box, a few steps
        # between two looks at the flow; latency and launches count
        dict(name="vms_small", kind="vms", nx=8, ny=8, nz=8, precision="fp64", dual=0, steps=10, subscales=False),
        # the 16^3 cavity validation run of 200 steps
        dict(name="vms_cavity16", kind="vms", nx=16, ny=16, nz=16, precision="fp64", dual=0, steps=200,
             subscales=False),
        # a ragged box with dual iterations, read out with its subscales as a
        # restartable state is
        dict(name="vms_dual", kind="vms", nx=41, ny=27, nz=33, precision="fp64", dual=2, steps=20, subscales=True),
        # the headline size: 5.3 M tets, 100 steps between two outputs
        dict(name="vms_cavity96", kind="vms", nx=96, ny=96, nz=96, precision="fp64", dual=0, steps=100,
             subscales=False),
        # the mixed form at an ordinary, odd size
        dict(name="vms_mixed", kind="vms", nx=61, ny=47, nz=53, precision="mixed", dual=0, steps=100,
             subscales=False),
        # a parameter study: independent cavities of 8..48 cells a side
        dict(name="vms_batch", kind="batch", count=32, n_lo=8, n_hi=48, precision="fp64", steps=50),
        # served requests: four flows admitted to the pool, run 100 steps,
        # read and retired
        dict(name="serve_mixed", kind="serve", count=4, n_lo=12, n_hi=32, precision="mixed", steps=100),
        # SUPG on tets, forward Euler
        dict(name="supg_tet", kind="supg", npe=4, nx=64, ny=64, nz=64, precision="fp64", ab2=False, bbar=False,
             steps=50),
        # SUPG on a hexa channel of 1 M elements, forward Euler
        dict(name="supg_channel", kind="supg", npe=8, nx=256, ny=64, nz=64, precision="fp64", ab2=False, bbar=False,
             steps=50),
        # the mixed form on an odd hexa channel with AB2 and B-bar
        dict(name="supg_channel_mixed", kind="supg", npe=8, nx=93, ny=37, nz=29, precision="mixed", ab2=True,
             bbar=True, steps=50),
        # a pressure / potential solve on tets: sources, fluxes, fixed values
        dict(name="poisson_tet", kind="poisson", npe=4, nx=64, ny=64, nz=64, problem="classic"),
        # the wall distance on a small odd hexa mesh
        dict(name="poisson_distance", kind="poisson", npe=8, nx=33, ny=27, nz=21, problem="distance"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: kinds in turn of their use, sizes log-uniform."""
    kind = rng.choice(["vms", "vms", "vms", "batch", "serve", "supg", "supg", "poisson"])
    prec = rng.choice(["fp64", "fp64", "mixed"])
    if kind == "batch":
        lo = rng.randint(8, 16)
        return dict(kind="batch", count=rng.randint(3, 32), n_lo=lo, n_hi=rng.randint(lo + 4, 48), precision=prec,
                    steps=rng.randint(10, 50))
    if kind == "serve":
        lo = rng.randint(8, 16)
        return dict(kind="serve", count=rng.randint(1, 6), n_lo=lo, n_hi=rng.randint(lo + 4, 40), precision=prec,
                    steps=rng.randint(20, 150))
    if kind == "poisson":
        npe = rng.choice([4, 8])
        n = _logint(rng, 8, 60)
        dims = [max(5, int(round(n * rng.uniform(0.7, 1.3)))) for _ in range(3)]
        return dict(kind="poisson", npe=npe, nx=dims[0], ny=dims[1], nz=dims[2],
                    problem=rng.choice(["classic", "ppe", "distance"]))
    npe = rng.choice([4, 8]) if kind == "supg" else 4
    n = _logint(rng, 8, 80)
    dims = [max(5, int(round(n * rng.uniform(0.75, 1.15)))) for _ in range(3)]
    if kind == "vms":
        return dict(kind="vms", nx=dims[0], ny=dims[1], nz=dims[2], precision=prec, dual=rng.choice([0, 0, 0, 1, 2]),
                    steps=rng.randint(10, 30) if n > 40 else rng.randint(10, 100), subscales=False)
    ab2 = rng.random() < 0.4
    return dict(kind="supg", npe=npe, nx=dims[0], ny=dims[1], nz=dims[2], precision=prec, ab2=ab2,
                bbar=npe == 8 and rng.random() < 0.4, steps=rng.randint(10, 50))


# ---------------------------------------------------------------- the meshes
def _grid(nx, ny, nz, size, seed, jitter):
    """Nodes of a box of nx x ny x nz cells, interior nodes moved by a seeded
    fraction of the cell size."""
    rng = np.random.default_rng(seed)
    dims, h = np.array([nx, ny, nz]), np.array(size, float) / np.array([nx, ny, nz])
    ijk = np.stack(np.meshgrid(*[np.arange(m + 1, dtype=np.int32) for m in dims], indexing="ij"), -1).reshape(-1, 3)
    X = ijk * h
    inner = np.all((ijk > 0) & (ijk < dims), axis=1)
    X[inner] += rng.uniform(-jitter, jitter, (int(inner.sum()), 3)) * h
    cell = np.stack(np.meshgrid(*[np.arange(m, dtype=np.int32) for m in dims], indexing="ij"), -1).reshape(-1, 3)
    base = (cell[:, 0] * np.int32(ny + 1) + cell[:, 1]) * np.int32(nz + 1) + cell[:, 2]
    step = np.array([(ny + 1) * (nz + 1), nz + 1, 1], np.int32)
    return X, ijk, dims, base.astype(np.int32), step, rng


def _kuhn(base, step, origin):
    """Six tets a cell; `origin` is the corner that the solver's Jacobian takes
    differences to (0 for VMS, 3 for the shape functions of femTetra4), so
    that every element's determinant is positive."""
    conn = np.empty((base.size, 6, 4), np.int32)
    for k, perm in enumerate(itertools.permutations(range(3))):
        at = [base]
        for ax in perm:
            at.append(at[-1] + step[ax])
        even = perm in ((0, 1, 2), (1, 2, 0), (2, 0, 1))
        if even == (origin == 3):
            at[0], at[1] = at[1], at[0]
        for a in range(4):
            conn[:, k, a] = at[a]
    return conn.reshape(-1, 4)


def _hexa(base, step):
    sx, sy, sz = step
    off = np.array([0, sx, sx + sy, sy, sz, sx + sz, sx + sy + sz, sy + sz], np.int32)
    return base[:, None] + off


def _cavity(nx, ny, nz, seed, solver, dual=0, mu=0.01, lid=1.0, ab2=False):
    X, ijk, dims, base, step, rng = _grid(nx, ny, nz, (nx / max(nx, ny, nz), ny / max(nx, ny, nz), nz / max(nx, ny, nz)),
                                          seed, 0.1)
    conn = _kuhn(base, step, 0 if solver == mesh.VMS else 3)
    h = 0.75 / max(nx, ny, nz)
    top = ijk[:, 2] == nz
    wall = np.any((ijk == 0) | (ijk == dims), axis=1) & ~top
    N = X.shape[0]
    init = np.zeros((N, 4))
    init[:, :3] = rng.uniform(-1e-3, 1e-3, (N, 3))
    c2 = VMS_PROPS["inv_eps"]
    if solver == mesh.VMS:
        dt = min(0.05 * h / (lid + math.sqrt(c2)), mu / c2)
        props = (VMS_PROPS["rho"], mu, c2, VMS_PROPS["c1"], VMS_PROPS["c2"])
    else:
        dt = min(0.05 * h / lid, 0.1 * h * h / mu)
        props = (1.0, mu, 1.0, 4.0, 0.0)
    lidn, walln = np.nonzero(top)[0].astype(np.int32), np.nonzero(wall)[0].astype(np.int32)
    vals = np.zeros((lidn.size, 4))
    vals[:, 0] = lid
    pin = 1 if solver == mesh.VMS else 0
    return mesh.Problem(
        coords=X, conn=conn, solver=solver, props=props, time_step=dt, total_steps=2, dual_step=dt / (dual + 1),
        tot_dual_steps=dual, ex_opts=(0 if ab2 else 1, 0, 1, 1, 1, 1), max_node_dofs=4 if pin else 3, vel_node=lidn,
        vel_vals=vals, vel_dir=np.full(lidn.size, 6, np.int32), dir_node=walln, dir_vals=np.zeros((walln.size, 3)),
        pres_node=np.zeros(pin, np.int32), pres_vals=np.zeros(pin), init_state=init)


def _channel(nx, ny, nz, seed, ab2, bbar):
    X, ijk, dims, base, step, rng = _grid(nx, ny, nz, (4.0, 1.0, 1.0), seed, 0.05)
    conn = _hexa(base, step)
    h, mu = min(4.0 / nx, 1.0 / ny, 1.0 / nz), 0.005
    N = X.shape[0]
    y, z = X[:, 1], X[:, 2]
    prof = 16.0 * y * (1 - y) * z * (1 - z)
    inlet = np.nonzero(ijk[:, 0] == 0)[0].astype(np.int32)
    side = (ijk[:, 1] == 0) | (ijk[:, 1] == ny) | (ijk[:, 2] == 0) | (ijk[:, 2] == nz)
    walls = np.nonzero(side & (ijk[:, 0] > 0))[0].astype(np.int32)
    init = np.zeros((N, 4))
    init[:, 0] = prof
    init[:, :3] += rng.uniform(-1e-3, 1e-3, (N, 3))
    vals = np.zeros((inlet.size, 4))
    vals[:, 0] = prof[inlet]
    return mesh.Problem(
        coords=X, conn=conn, solver=mesh.SUPG, props=(1.0, mu, 1.0, 4.0, 0.0), time_step=min(0.05 * h, 0.1 * h * h / mu),
        total_steps=2, ex_opts=(0 if ab2 else 1, 1 if bbar else 0, 1, 1, 1, 1), max_node_dofs=3, vel_node=inlet,
        vel_vals=vals, vel_dir=np.full(inlet.size, 6, np.int32), dir_node=walls, dir_vals=np.zeros((walls.size, 3)),
        init_state=init)


def _poisson(case, seed):
    nx, ny, nz, npe = case["nx"], case["ny"], case["nz"], case["npe"]
    X, ijk, dims, base, step, rng = _grid(nx, ny, nz, (1.0, 1.0, 1.0), seed, 0.1)
    conn = _kuhn(base, step, 3) if npe == 4 else _hexa(base, step)
    E, N = conn.shape[0], X.shape[0]
    empty = np.zeros(0, np.int32)
    if case["problem"] == "distance":  # unit source, zero on the walls, isotropic
        diff = np.ones((E, 3))
        src, val = np.arange(E, dtype=np.int32), np.full(E, float(rng.uniform(0.8, 1.2)))
        off, nodes, nval = np.zeros(1, np.int32), empty, np.zeros(0)
        dn = np.nonzero(np.any((ijk[:, 1:] == 0) | (ijk[:, 1:] == dims[1:]), axis=1))[0].astype(np.int32)
        dv = np.zeros(dn.size)
    else:
        diff = rng.uniform(0.5, 2.0, (E, 3))
        src = np.arange(0, E, 4, dtype=np.int32)
        val = rng.uniform(-1.0, 1.0, src.size)
        # a flux through the faces on x = 1
        out = ijk[:, 0] == nx
        quads = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)] if npe == 4 else [(1, 2, 6, 5)]
        last = np.arange(E).reshape(nx, -1)[-1]
        faces = [conn[last][:, q][np.all(out[conn[last][:, q]], axis=1)] for q in quads]
        faces = np.concatenate(faces)
        nodes, k = faces.reshape(-1).astype(np.int32), faces.shape[1]
        off = np.arange(0, nodes.size + 1, k, dtype=np.int32)
        nval = rng.uniform(0.0, 1.0, faces.shape[0]) * (1.0 / (ny * nz))
        if case["problem"] == "ppe":  # pure Neumann
            dn, dv = empty, np.zeros(0)
        else:
            dn = np.nonzero(ijk[:, 0] == 0)[0].astype(np.int32)
            dv = np.sin(np.pi * X[dn, 1]) * np.cos(np.pi * X[dn, 2])
    kind = {"classic": mesh.POISSON_CLASSIC, "ppe": mesh.POISSON_PPE, "distance": mesh.POISSON_DISTANCE}[case["problem"]]
    return mesh.PoissonProblem(X, conn, diff, src, val, off, nodes, nval, dn, dv, kind)


def _sizes(case):
    """Cells a side of a batch's or a pool's members: the case's, whatever the seed."""
    rng = np.random.default_rng(case["count"] * 1009 + case["n_lo"] * 31 + case["n_hi"])
    return [int(n) for n in rng.integers(case["n_lo"], case["n_hi"] + 1, case["count"])]


def _problems(case, seed):
    if case["kind"] == "vms":
        return [_cavity(case["nx"], case["ny"], case["nz"], seed, mesh.VMS, case["dual"])]
    if case["kind"] == "supg":
        if case["npe"] == 4:
            return [_cavity(case["nx"], case["ny"], case["nz"], seed, mesh.SUPG, ab2=case["ab2"])]
        return [_channel(case["nx"], case["ny"], case["nz"], seed, case["ab2"], case["bbar"])]
    rng = np.random.default_rng(seed)
    return [_cavity(n, n, n, seed * 1009 + i, mesh.VMS, mu=float(np.exp(rng.uniform(np.log(5e-3), np.log(1e-1)))),
                    lid=float(rng.uniform(0.5, 2.0))) for i, n in enumerate(_sizes(case))]


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    if case["kind"] == "poisson":
        return dict(kind="poisson", solver=api.GpuPoisson(_poisson(case, seed)))
    prec = api.FM_MIXED if case["precision"] == "mixed" else api.FM_FP64
    gps = [api.GpuProblem(p, prec) for p in _problems(case, seed)]
    st = dict(kind=case["kind"], steps=case["steps"], gps=gps, subscales=bool(case.get("subscales")))
    if case["kind"] == "serve":
        for g in gps:
            g.prepare()
        st["pool"] = api.Pool(mesh.VMS, mesh.TET4, max_problems=len(gps),
                              max_elems=2 * sum(g.n_elems for g in gps) + 65536,
                              max_nodes=2 * sum(g.n_nodes for g in gps) + 65536, precision=prec)
    else:
        st["batch"] = api.Batch(gps, graph_steps=50 if case["kind"] == "batch" else 0)
    return st


def run(st):
    if st["kind"] == "poisson":
        st["solver"].solve()
        x, dist = st["solver"].solution()
        return dict(x=x) if dist is None else dict(x=x, distance=dist)
    gps = st["gps"]
    if st["kind"] == "serve":
        pool = st["pool"]
        for g in gps:
            if not pool.add(g):
                raise RuntimeError("the pool has no room")
        pool.step(gps, [st["steps"]] * len(gps))
        if pool.wait():
            raise RuntimeError("a request failed")
        out = [dict(u=u, p=p) for u, p, _, _ in (g.state(elements=False) for g in gps)]
        for g in gps:
            pool.remove(g)
        return out
    st["batch"].step(st["steps"])
    st["batch"].sync()
    if st["subscales"]:
        u, p, _, sd = gps[0].state()
        return dict(u=u, p=p, subscales=sd)
    out = [dict(u=u, p=p) for u, p, _, _ in (g.state(elements=False) for g in gps)]
    return out[0] if len(out) == 1 else out


# ---------------------------------------------------------------- bytes and operations
def _counts(case):
    if case["kind"] in ("batch", "serve"):
        ns = _sizes(case)
        return sum(6 * n ** 3 for n in ns), sum((n + 1) ** 3 for n in ns)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    per = 6 if case["kind"] == "vms" or case["npe"] == 4 else 1
    return per * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)


def work(case):
    """Time steps: each streams the element and node state once (VMS: 16 B
    connectivity and the subscales read and written an element; SUPG: 2 B a
    corner, lambda and regime, with AB2 the history read and written;
    coordinates, state and mass a node) and evaluates every element once.
    Poisson: the assembled matrix and the vectors read once, the solution
    written, and the operations of one product."""
    E, N = _counts(case)
    if case["kind"] == "poisson":
        nnz = (15 if case["npe"] == 4 else 27) * N
        return dict(bytes=12 * nnz + 32 * N, flops=2 * nnz)
    k, fp32 = case["steps"], case["precision"] == "mixed"
    if case["kind"] == "supg":
        npe = case["npe"]
        elem = 2 * npe + 16 + (48 * npe if case["ab2"] else 0)
        return dict(bytes=k * (elem * E + 84 * N), flops=k * (800 if npe == 4 else 3600) * E)
    k *= case.get("dual", 0) + 1
    return dict(bytes=k * ((112 if fp32 else 208) * E + 96 * N), flops=k * 884 * E)


# ---------------------------------------------------------------- the same in 64-bit torch
def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "poisson":
        return _exact_poisson(_poisson(case, seed), dev)
    ps = _problems(case, seed)
    if case["kind"] == "supg":
        return _exact_supg(ps[0], case["steps"], dev)
    out = [_exact_vms(p, case["steps"], dev) for p in ps]
    if case["kind"] == "vms":
        return out[0] if case["subscales"] else dict(u=out[0]["u"], p=out[0]["p"])
    return [dict(u=o["u"], p=o["p"]) for o in out]


def _t(a, dev, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=dev).to(dtype)


def _scatter(conn, vals, N):
    """Sum of per-corner values (E, npe, C) at the nodes."""
    out = torch.zeros((N, vals.shape[-1]), dtype=torch.float64, device=vals.device)
    return out.index_add_(0, conn.reshape(-1), vals.reshape(-1, vals.shape[-1]))


def _apply_bc(p, s, dev):
    """The constant lid / inlet rows, then the pinned pressures, then the walls."""
    s[_t(p.vel_node, dev, torch.int64), :3] = _t(p.vel_vals[:, :3], dev)
    if p.solver == mesh.VMS and p.pres_node.size:
        s[_t(p.pres_node, dev, torch.int64), 3] = _t(p.pres_vals, dev)
    s[_t(p.dir_node, dev, torch.int64), :3] = _t(p.dir_vals, dev)
    return s


def _exact_vms(p, steps, dev):
    A, B = 0.58541020, 0.13819660
    S = A + 3.0 * B
    X, conn = _t(p.coords, dev), _t(p.conn, dev, torch.int64)
    E, N = conn.shape[0], X.shape[0]
    J = (X[conn[:, 1:]] - X[conn[:, :1]]).transpose(1, 2)  # J[i][k] = x_{k+1,i} - x_{0,i}
    det = torch.det(J)
    inv = torch.linalg.inv(J)                               # grad of barycentric k+1: row k
    DN = torch.cat([-inv.sum(1, keepdim=True), inv], 1)     # (E, 4, 3)
    V = det / 6.0
    ih = (6.0 * V) ** (-1.0 / 3.0)
    mass = _scatter(conn, (V / 4.0)[:, None, None].expand(E, 4, 1), N)
    rho, mu, inv_eps, c1, c2 = p.props
    nu, dt, ds, per = mu / rho, p.time_step, p.dual_step, p.tot_dual_steps + 1
    bc = torch.zeros(N, dtype=torch.bool, device=dev)
    for nodes in (p.vel_node, p.dir_node, p.pres_node):
        bc[_t(nodes, dev, torch.int64)] = True
    post = _apply_bc(p, _t(p.init_state, dev).clone(), dev)
    pre = post.clone()
    sdu = torch.zeros((E, 4, 3), dtype=torch.float64, device=dev)
    pq = torch.zeros(4, dtype=torch.float64, device=dev)
    for it in range(steps * per):
        first = it % per == 0
        Q = pre[:, :3][conn]
        if it > 0:  # the subscales of the iteration before
            G = torch.einsum("eai,eaj->eij", Q, DN)
            gp = torch.einsum("a,eai->ei", pq, DN)
            hah = B * Q.sum(1, keepdim=True) + (A - B) * Q + sdu
            r = torch.einsum("eij,egj->egi", G, hah) + gp[:, None]
            a = hah.square().sum(-1).amax(1).sqrt()
            tau = 1.0 / (1.0 / dt + c1 * nu * ih * ih + c2 * a * ih)
            proj = (B * r.sum(1, keepdim=True) + (A - B) * r) / S          # P_a
            back = B * proj.sum(1, keepdim=True) + (A - B) * proj          # at the points
            sdu = (sdu / dt + back - r) * tau[:, None, None]
        U, P = post[:, :3][conn], post[:, 3][conn]
        G = torch.einsum("eai,eaj->eij", U, DN)
        ug = B * U.sum(1, keepdim=True) + (A - B) * U
        hah = ug + sdu
        Xg = torch.einsum("eij,egj->egi", G, hah)
        if not first:
            Xg = Xg + (ug - (B * Q.sum(1, keepdim=True) + (A - B) * Q)) / dt
        K = 4.0 * nu * G - torch.einsum("egi,egk->eik", sdu, hah)
        K = K - S * P.sum(1)[:, None, None] * torch.eye(3, dtype=torch.float64, device=dev)
        res = torch.empty((E, 4, 4), dtype=torch.float64, device=dev)
        w = (V * 0.25)[:, None, None]
        res[..., :3] = w * (B * Xg.sum(1, keepdim=True) + (A - B) * Xg + torch.einsum("eik,eak->eai", K, DN))
        tr = G.diagonal(dim1=1, dim2=2).sum(-1)
        res[..., 3] = w[..., 0] * inv_eps * (tr[:, None] * S - torch.einsum("ei,eai->ea", sdu.sum(1), DN))
        s = post if first else torch.where(bc[:, None], pre, post)
        pre = s - ds * _scatter(conn, res, N) / mass
        pq = pre[:4, 3].clone()
        post = _apply_bc(p, pre.clone(), dev)
    return dict(u=post[:, :3], p=post[:, 3], subscales=sdu.reshape(E, 12))


def _rule(npe, dev):
    """Gauss points' shape values (g, a), local derivatives (g, a, 3), weight."""
    if npe == 4:
        a, b = 0.58541020, 0.13819660
        q = torch.tensor([[a, b, b], [b, a, b], [b, b, a], [b, b, b]], dtype=torch.float64, device=dev)
        N = torch.cat([q, 1.0 - q.sum(1, keepdim=True)], 1)
        d = torch.cat([torch.eye(3, dtype=torch.float64, device=dev), -torch.ones((1, 3), dtype=torch.float64, device=dev)])
        return N, d.expand(4, 4, 3), 1.0 / 24.0
    sgn = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                        [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64, device=dev)
    f = 1.0 + (sgn / math.sqrt(3.0))[:, None] * sgn[None]                  # (g, a, 3)
    d = torch.stack([sgn[:, 0] * f[..., 1] * f[..., 2], sgn[:, 1] * f[..., 0] * f[..., 2],
                     sgn[:, 2] * f[..., 0] * f[..., 1]], -1) / 8.0
    return f.prod(-1) / 8.0, d, 1.0


def _geometry(Xe, d):
    """Global derivatives (E, a, 3) and determinant at a point with local derivatives d."""
    J = torch.einsum("na,enb->eab", d, Xe)
    inv = torch.linalg.inv(J)
    return inv, torch.einsum("ebc,nc->enb", inv, d), torch.det(J)


def _exact_supg(p, steps, dev):
    npe = p.conn.shape[1]
    N_, d_, wq = _rule(npe, dev)
    X, conn = _t(p.coords, dev), _t(p.conn, dev, torch.int64)
    E, N = conn.shape[0], X.shape[0]
    rho, mu, alpha, cI, _ = p.props
    nu, dt = mu / rho, p.time_step
    euler, bbar = p.ex_opts[0] == 1, p.ex_opts[1] == 1
    Xe = X[conn]
    geo = []
    for g in range(1 if npe == 4 else 8):  # a tet's derivatives are the same at every point
        inv, gd, det = _geometry(Xe, d_[g])
        G = torch.einsum("eca,ecb->eab", inv, inv)
        geo.append((gd, det * wq, G, torch.linalg.inv(G)))
    if npe == 4:
        geo = geo * 4
    vol = sum(q[1] for q in geo)
    mass = _scatter(conn, sum(rho * N_[g][None, :, None] * geo[g][1][:, None, None] for g in range(len(geo))), N)
    Dbar = sum(q[0] * q[1][:, None, None] for q in geo) / vol[:, None, None] if bbar else None
    s = _apply_bc(p, _t(p.init_state, dev).clone(), dev)
    prev, lam_e = None, None
    for it in range(steps):
        U = s[:, :3][conn]
        k = torch.zeros((E, npe, 3), dtype=torch.float64, device=dev)
        lam_int = torch.zeros(E, dtype=torch.float64, device=dev)
        for g, (gd, w, G, iG) in enumerate(geo):
            u = torch.einsum("a,eac->ec", N_[g], U)
            gr = torch.einsum("ead,eac->ecd", gd, U)
            div = gr.diagonal(dim1=1, dim2=2).sum(-1)
            tau = 1.0 / torch.sqrt(torch.einsum("ea,eab,eb->e", u, G, u) + nu * nu * cI * G.square().sum((1, 2)))
            nuC = 1.0 / (G.diagonal(dim1=1, dim2=2).sum(-1) * tau)
            l2 = torch.sqrt(torch.einsum("ea,eab,eb->e", u, iG, u))
            lam = alpha * torch.clamp(l2, min=nu)
            lam_int += lam * w
            conv = torch.einsum("ec,edc->ed", u, gr)
            eps = gr + gr.transpose(1, 2)                   # off-diagonal: engineering shear
            diag = gr.diagonal(dim1=1, dim2=2)
            if bbar:
                db = (Dbar - gd) / 3.0                       # B1, B3, B5 per node and direction
                q = (db * U).sum(1)                          # (E, 3)
                diag = diag - q + (q.sum(-1, keepdim=True) - q)
            sig_n = lam[:, None] * diag.sum(-1, keepdim=True) + 2.0 * mu * diag
            sig = mu * eps
            sig = sig - torch.diag_embed(sig.diagonal(dim1=1, dim2=2))
            f = torch.einsum("ead,ecd->eac", gd, sig)
            if bbar:
                tot = sig_n.sum(-1, keepdim=True)
                f = f + (gd - db) * sig_n[:, None] + db * (tot - sig_n)[:, None]
            else:
                f = f + gd * sig_n[:, None]
            f = f + (rho * N_[g][None, :] + rho * tau[:, None] * torch.einsum("eac,ec->ea", gd, u))[..., None] * conv[:, None]
            f = f + (rho * nuC * div)[:, None, None] * gd
            k += f * w[:, None, None]
        k *= -dt
        acc = k if euler or it == 0 else 1.5 * k - 0.5 * prev
        prev, lam_e = k, lam_int / vol
        s[:, :3] += _scatter(conn, acc, N) / mass
        s = _apply_bc(p, s, dev)
    U = s[:, :3][conn]
    num = sum(torch.einsum("eac,eac->e", q[0], U) * q[1] for q in geo)
    return dict(u=s[:, :3], p=-lam_e * (num / vol))


def _exact_poisson(p, dev):
    npe = p.conn.shape[1]
    N_, d_, wq = _rule(npe, dev)
    X, conn = _t(p.coords, dev), _t(p.conn, dev, torch.int64)
    E, N = conn.shape[0], X.shape[0]
    Xe, diff = X[conn], _t(p.diffusivity, dev)
    K = torch.zeros((E, npe, npe), dtype=torch.float64, device=dev)
    fe = torch.zeros((E, npe), dtype=torch.float64, device=dev)
    src = torch.zeros(E, dtype=torch.float64, device=dev)
    src[_t(p.source_elem, dev, torch.int64)] = _t(p.source_value, dev)
    for g in range(N_.shape[0]):
        _, gd, det = _geometry(Xe, d_[g])
        K += torch.einsum("ead,ed,ebd->eab", gd, diff, gd) * (det * wq)[:, None, None]
        fe += N_[g][None] * (src * det * wq)[:, None]
    b = _scatter(conn, fe[..., None], N)[:, 0]
    if p.neumann_value.size:
        k = np.diff(p.neumann_off)
        b.index_add_(0, _t(p.neumann_nodes, dev, torch.int64), _t(np.repeat(p.neumann_value / k, k), dev))
    row = conn[:, :, None].expand(E, npe, npe).reshape(-1)
    col = conn[:, None, :].expand(E, npe, npe).reshape(-1)
    M = torch.sparse_coo_tensor(torch.stack([row, col]), K.reshape(-1), (N, N)).coalesce().to_sparse_csr()
    free = torch.ones(N, dtype=torch.float64, device=dev)
    x = torch.zeros(N, dtype=torch.float64, device=dev)
    if p.dir_node.size:
        dn = _t(p.dir_node, dev, torch.int64)
        free[dn] = 0.0
        x[dn] = _t(p.dir_value, dev)
        b = (b - M @ x) * free
    else:
        b = b - b.mean()
    D = 1.0 / _scatter(conn, K.diagonal(dim1=1, dim2=2)[..., None], N)[:, 0]
    r, y = b.clone(), torch.zeros_like(b)
    z = D * r * free
    q, rz, stop = z.clone(), torch.dot(r, z), 1e-15 * float(b.norm())
    for it in range(20000):
        Mq = (M @ q) * free
        al = rz / torch.dot(q, Mq)
        y += al * q
        r -= al * Mq
        if it % 16 == 0 and float(r.norm()) <= stop:
            break
        z = D * r * free
        rz, old = torch.dot(r, z), rz
        q = z + (rz / old) * q
    x = x + y * free
    if p.problem == mesh.POISSON_PPE:
        x = x - x.mean()
    if p.problem != mesh.POISSON_DISTANCE:
        return dict(x=x)
    if npe == 4:
        n0 = torch.tensor([0.0, 0, 0, 1], dtype=torch.float64, device=dev)
        d0 = d_[0]
    else:
        n0 = torch.full((8,), 0.125, dtype=torch.float64, device=dev)
        d0 = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                           [-1, 1, 1]], dtype=torch.float64, device=dev) / 8.0
    _, gd, _ = _geometry(Xe, d0)
    xe = x[conn]
    grad = torch.einsum("ead,ea->ed", gd, xe).square().sum(-1)
    return dict(x=x, distance=-torch.sqrt(grad) + torch.sqrt(grad + 2.0 * (xe * n0).sum(-1)))

"""The workloads that the cloth framework is timed on, through its public entry points.

A case is a dict of plain values whose ``"kind"`` picks one of the paths below:

* ``frame``   -- one ``Solver.forward`` from a given state (positions and velocities are put back before every pass,
  as a rollout from a snapshot does): a sheet a few frames into resting on a box or on a sphere.
* ``contact`` -- the contact part of a substep as its four calls: BVH builds, broad phase, pair list, contact sweep.
* ``sweep``   -- ``Solver.spring_sweep``, one Jacobi sweep over springs and bending pairs of a large sheet.
* ``batch``   -- one ``BatchedSolver.forward`` over many independent cloths, each over its own box.
* ``lbvh``    -- ``LBVH.build`` over a triangle soup and ``LBVH.query`` with one point per triangle.
* ``color``   -- ``GraphColoring`` of a sheet's edges, as built once per mesh.
* ``mlp``     -- ``WarmStartMLP.forward`` on feature rows (inference of the learned warm start).
* ``train``   -- ``WarmStartMLP.gradients`` on a minibatch (one training step's gradients).
"""
import math
import random

import numpy as np
import torch

import __graft_entry__

sx = __graft_entry__.load_package()


def listed():
    return [
        # the drop-in use: reference schedule (one sweep per substep, BVHs once a frame), launched eagerly, a small mesh
        dict(name="frame_eager_33x27", kind="frame", nx=33, ny=27, obstacle="box", substeps=20, iters=1, graph=False,
             fast=False),
        # the 64 x 64 cloth on a box at 10 x 20 iterations, as a replayed graph: an interactive scene
        dict(name="frame_box_64x64", kind="frame", nx=64, ny=64, obstacle="box", substeps=10, iters=20, graph=True,
             fast=False),
        # the headline scene: 256 x 256 with self contact on a 20 480-face sphere, 10 x 30 iterations
        dict(name="frame_sphere_256x256", kind="frame", nx=256, ny=256, obstacle="sphere", substeps=10, iters=30,
             graph=True, fast=False),
        # a production sheet's contact phase by itself, sides that divide nothing
        dict(name="contact_181x139", kind="contact", nx=181, ny=139),
        # one sweep of a sheet far larger than the SMs hold at once
        dict(name="sweep_601x599", kind="sweep", nx=601, ny=599),
        # a small batch of cloths (rollouts for one policy update), reference arithmetic
        dict(name="batch_24", kind="batch", instances=24, lo=16, hi=128, substeps=10, iters=20, fast=False),
        # a data-generation batch: near 600 000 vertices, fast arithmetic
        dict(name="batch_96_fast", kind="batch", instances=96, lo=16, hi=128, substeps=10, iters=20, fast=True),
        # standalone broad phase, an asset-sized soup
        dict(name="lbvh_20011", kind="lbvh", tris=20011, cap=64),
        # standalone broad phase, the benchmark's 2^20 triangles and queries
        dict(name="lbvh_1048576", kind="lbvh", tris=1 << 20, cap=64),
        # colouring of the 256 x 256 sheet's 195 585 edges
        dict(name="color_256x256", kind="color", nx=256, ny=256),
        # warm-start inference for a batch of a million vertices (odd count)
        dict(name="mlp_1000003", kind="mlp", rows=1000003),
        # the training minibatch of the warm start
        dict(name="train_65536", kind="train", rows=65536, samples=262144),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "contact", "sweep", "batch", "batch", "lbvh", "color", "mlp", "train"])
    if kind == "frame":
        obstacle = rng.choice(["box", "sphere"])
        graph = rng.random() < 0.7
        return dict(kind=kind, nx=_logint(rng, 20, 220), ny=_logint(rng, 20, 220), obstacle=obstacle,
                    substeps=rng.randint(3, 10), iters=rng.choice([1, 2, 5, 10, 20, 21]) if graph else 1, graph=graph,
                    fast=rng.random() < 0.3)
    if kind in ("contact", "color"):
        return dict(kind=kind, nx=_logint(rng, 20, 220), ny=_logint(rng, 20, 220))
    if kind == "sweep":
        return dict(kind=kind, nx=_logint(rng, 30, 600), ny=_logint(rng, 30, 600))
    if kind == "batch":
        lo = rng.randint(8, 40)
        return dict(kind=kind, instances=_logint(rng, 4, 60), lo=lo, hi=lo + rng.randint(0, 80),
                    substeps=rng.randint(3, 10), iters=rng.choice([5, 10, 20, 21]), fast=rng.random() < 0.5)
    if kind == "lbvh":
        return dict(kind=kind, tris=_logint(rng, 500, 1000000), cap=rng.choice([40, 64]))
    if kind == "mlp":
        return dict(kind=kind, rows=_logint(rng, 200, 1000000))
    samples = _logint(rng, 4000, 200000)
    return dict(kind=kind, rows=_logint(rng, 500, 65536), samples=samples)


# ---- geometry -------------------------------------------------------------------------------------------------------
def _sheet(nx, ny, rng, height=0.0, size=1.0, jitter=1e-4):
    """A jittered nx x ny sheet of two triangles per square, its longer side ``size``: (float32[V, 3], int32[F, 3])."""
    step = size / (max(nx, ny) - 1)
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    x = np.stack([0.5 + (i - 0.5 * (nx - 1)) * step, 0.5 + (j - 0.5 * (ny - 1)) * step, np.full(i.shape, height)], -1)
    x = x.reshape(-1, 3) + rng.uniform(-jitter, jitter, (nx * ny, 3))
    a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1)
    b, c, d = a + 1, a + ny, a + ny + 1
    f = np.stack([np.stack([a, c, b], -1), np.stack([b, c, d], -1)], 1).reshape(-1, 3)
    return x.astype(np.float32), f.astype(np.int32)


def _topology(x, f):
    """Springs (unique edges), bending pairs (the vertices opposite an inner edge), their rest lengths and the inverse
    masses 1 / sum(l0 / 2), in numpy."""
    e = np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]), axis=1).astype(np.int64)
    opp = np.concatenate([f[:, 2], f[:, 0], f[:, 1]])
    key = e[:, 0] * x.shape[0] + e[:, 1]
    order = np.argsort(key, kind="stable")
    key, e, opp = key[order], e[order], opp[order]
    first = np.concatenate([[True], key[1:] != key[:-1]])
    edges = e[first]
    twin = np.nonzero(~first)[0]
    bend = np.stack([opp[twin - 1], opp[twin]], -1).astype(np.int64)
    length = lambda p: np.sqrt(((x[p[:, 0]] - x[p[:, 1]]) ** 2).sum(1, dtype=np.float32)).astype(np.float32)  # noqa: E731
    l0 = length(edges)
    half = np.repeat(0.5 * l0.astype(np.float64), 2)
    m_inv = 1.0 / np.bincount(edges.reshape(-1), weights=half, minlength=x.shape[0])
    return edges, bend, l0, length(bend), m_inv.astype(np.float32)


STRETCH, BENDING, GRAVITY, DT = 1e5, 1e8, (0.0, 0.0, -9.81), 1.0 / 60.0


def _solver(case, seed, settle):
    """A solver whose sheet starts a few millimetres above its obstacle and has come down on it for ``settle`` frames."""
    rng = np.random.default_rng(seed)
    nx, ny, sphere = case["nx"], case["ny"], case.get("obstacle", "sphere") == "sphere"
    thickness = 2e-3 if sphere else 4e-3
    if sphere:
        ox, of = sx.icosphere(5, 0.3, (0.5, 0.5, 0.5))
        top = 0.8
    else:
        ox, of = sx.box_mesh(0.5, center=(0.5, 0.5, 0.3))
        top = 0.55
    x, f = _sheet(nx, ny, rng, height=top + 2.5 * thickness)
    reference = not case.get("graph", True)
    cloth = sx.TriMesh(x, f, device="cuda")
    sim = sx.Solver(cloth, sx.TriMesh(ox, of, device="cuda", is_static=True), dHat=thickness * thickness,
                    stiffness_stretch=STRETCH, stiffness_bending=BENDING, g=GRAVITY, dt=DT, n_iter=case.get("iters", 10),
                    rebuild="frame" if reference else "substep", bending_on="x" if reference else "y")
    sim.padding = thickness if sphere else 2 * thickness
    sim.enable_collision_handling = True
    sim.fast_math = case.get("fast", False)
    mask = np.zeros(x.shape[0], np.int32)
    if not sphere:
        mask[[0, ny - 1]] = 1  # two corners hold the sheet on the box
    sim.set_fixed_vertices(torch.from_numpy(mask))
    cloth.v4[:, 2] = -0.3
    sim.use_graph = case.get("graph", True)
    for _ in range(settle):
        sim.forward(case.get("substeps", 10))
    return sim


def _sweep_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x, f = _sheet(case["nx"], case["ny"], rng, jitter=1e-4)
    p = rng.uniform(0, 2 * np.pi, 6)
    u, v = x[:, 0], x[:, 1]
    bend = np.stack([0.003 * np.sin(5 * u + p[0]) * np.cos(4 * v + p[1]), 0.003 * np.cos(6 * u + p[2]),
                     0.02 * np.sin(7 * u + p[3]) * np.sin(6 * v + p[4])], -1)
    y = (x + bend + rng.normal(0.0, 2e-5, x.shape)).astype(np.float32)
    fixed = np.ones(x.shape[0], np.float32)
    fixed[: case["ny"]: 3] = 0.0
    return x, f, y, fixed


def _mlp_params(rng):
    parts = []
    for shape, fan, used in (((64, 32), 24, 24), ((64,), 0, 64), ((64, 64), 64, 64), ((64,), 0, 64), ((8, 64), 64, 3),
                             ((8,), 0, 3)):
        a = rng.uniform(-1, 1, shape) * (math.sqrt(3.0 / fan) if fan else 0.05)
        if shape == (64, 32):
            a[:, used:] = 0.0
        if shape[0] == 8:
            a[used:] = 0.0
        parts.append(a.astype(np.float32).ravel())
    return np.concatenate(parts)


def _mlp_inputs(case, seed):
    """Parameters and feature rows: 24 columns of the scales the warm start's features have, 8 zero columns."""
    rows = case.get("samples", case["rows"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    feat = torch.randn((rows, 32), generator=gen, device="cuda")
    scale = torch.tensor([0.02] * 6 + [0.05] * 4 + [0.3] * 6 + [0.0] * 3 + [0.3, 0.3] + [0.0] * 3 + [0.0] * 8,
                         device="cuda")
    shift = torch.tensor([0.0] * 16 + [1.0, 1.0, 0.9] + [0.0] * 4 + [-0.6] + [0.0] * 8, device="cuda")
    feat = (feat * scale + shift).to(torch.bfloat16)
    return _mlp_params(np.random.default_rng(seed)), feat, gen


def _train_inputs(case, seed):
    params, feat, gen = _mlp_inputs(case, seed)
    target = torch.randn((feat.shape[0], 4), generator=gen, device="cuda") * 0.2
    target[:, 3] = 1.0
    idx = torch.randint(feat.shape[0], (case["rows"],), generator=gen, device="cuda", dtype=torch.int32)
    return params, feat, target, idx


# ---- the state a program holds, one pass, its outputs ------------------------------------------------------------------
class _State:
    def __init__(self, kind, **kw):
        self.kind = kind
        self.__dict__.update(kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        sim = _solver(case, seed, settle=4)
        m = sim.mesh_dy
        return _State(kind, sim=sim, x=m.x4.clone(), v=m.v4.clone(), substeps=case["substeps"])
    if kind == "contact":
        sim = _solver(dict(case, obstacle="sphere", substeps=10, iters=10), seed, settle=4)
        sim.build_bvhs()
        sim.compute_y(DT / 10)
        return _State(kind, sim=sim, y=sim.mesh_dy.y4.clone())
    if kind == "sweep":
        x, f, y, fixed = _sweep_inputs(case, seed)
        mesh = sx.TriMesh(x, f, device="cuda")
        sim = sx.Solver(mesh, None, 4e-6, STRETCH, BENDING, GRAVITY, DT, bending_on="y")
        sim.set_fixed_vertices(torch.from_numpy(1 - fixed.astype(np.int32)))
        mesh.y4[:, :3] = torch.from_numpy(y).cuda()
        return _State(kind, sim=sim, y=mesh.y4.clone())
    if kind == "batch":
        sizes, rng = random.Random(case["instances"]), np.random.default_rng(seed)
        out, cols = [], int(math.ceil(math.sqrt(case["instances"])))
        for k in range(case["instances"]):
            nx = sizes.randint(case["lo"], case["hi"])
            ny = max(case["lo"], nx - sizes.randint(0, 3))
            where = np.array([1.5 * (k % cols), 1.5 * (k // cols), 0.0])
            centre = where + np.array([0.5 + rng.uniform(-0.2, 0.2), 0.5 + rng.uniform(-0.2, 0.2), 0.3])
            x, f = _sheet(nx, ny, rng, height=0.55 + 0.01)
            bx, bf = sx.box_mesh(0.5, center=tuple(centre))
            out.append(sx.Instance((x + where).astype(np.float32), f, np.array([0, ny - 1]), bx, bf))
        batch = sx.BatchedSolver(out, 1.6e-5, STRETCH, BENDING, GRAVITY, DT, n_iter=case["iters"])
        batch.fast_math = case["fast"]
        batch.use_graph = True
        batch.v4[:, 2] = -0.3
        for _ in range(2):
            batch.forward(case["substeps"])
        return _State(kind, sim=batch, x=batch.x4.clone(), v=batch.v4.clone(), substeps=case["substeps"])
    if kind == "lbvh":
        verts, _, queries = sx.scenes.triangle_soup(case["tris"], seed)
        tri = torch.from_numpy(verts).cuda().view(-1, 3, 3)
        q4 = torch.zeros((case["tris"], 4), device="cuda")
        q4[:, :3] = torch.from_numpy(queries).cuda()
        lo, hi = torch.zeros_like(q4), torch.zeros_like(q4)
        lo[:, :3], hi[:, :3] = tri.amin(1), tri.amax(1)
        box6 = torch.cat([lo[:, :3].amin(0), hi[:, :3].amax(0)]).contiguous()
        # a query box wide enough for a few hits in a soup of this density
        pad = 2e-3 * (2.0 ** 20 / case["tris"]) ** (1.0 / 3.0)
        i32 = dict(dtype=torch.int32, device="cuda")
        return _State(kind, tree=sx.LBVH(case["tris"]), lo=lo, hi=hi, box=box6, q=q4, pad=pad, cap=case["cap"],
                      cand=torch.zeros((case["tris"], case["cap"]), **i32), num=torch.zeros(case["tris"], **i32))
    if kind == "color":
        rng = np.random.default_rng(seed)
        x, f = _sheet(case["nx"], case["ny"], rng)
        edges = _topology(x, f)[0]
        # a few edges less, as along the cuts of a pattern
        edges = np.delete(edges, rng.choice(len(edges), 2 + len(edges) // 1000, replace=False), axis=0)
        return _State(kind, verts=x.shape[0], edges=torch.from_numpy(edges.astype(np.int32)).cuda())
    if kind == "mlp":
        params, feat, _ = _mlp_inputs(case, seed)
        return _State(kind, net=sx.WarmStartMLP(params=params), feat=feat,
                      out=torch.zeros((feat.shape[0], 4), device="cuda"))
    params, feat, target, idx = _train_inputs(case, seed)
    return _State(kind, net=sx.WarmStartMLP(params=params), feat=feat, target=target, idx=idx)


def run(s):
    if s.kind in ("frame", "batch"):
        m = s.sim.mesh_dy if s.kind == "frame" else s.sim
        m.x4.copy_(s.x)
        m.v4.copy_(s.v)
        s.sim.forward(s.substeps)
        return [m.x4, m.v4]
    if s.kind == "contact":
        sim = s.sim
        sim.mesh_dy.y4.copy_(s.y)
        sim.build_bvhs()
        sim.broadphase_lbvh()
        sim.build_contact_pairs()
        sim.solve_collision_constraints_x()
        return [sim.vt_st_candidates, sim.vt_st_candidates_num, sim.vt_dy_candidates, sim.vt_dy_candidates_num,
                sim.tv_st_candidates, sim.tv_st_candidates_num, sim.mesh_dy.y4]
    if s.kind == "sweep":
        s.sim.mesh_dy.y4.copy_(s.y)
        s.sim.spring_sweep(DT / 10)
        return s.sim.mesh_dy.y4
    if s.kind == "lbvh":
        s.tree.build(s.lo, s.hi, s.box)
        cand, num = s.tree.query(s.q, s.pad, s.cap, s.cand, s.num)
        return [cand, num, s.tree.node_min4, s.tree.node_max4]
    if s.kind == "color":
        g = sx.GraphColoring(s.verts, s.edges)
        return [g.edges_color, g.sorted_edges_sequence_for_color, g.color_prefix_sum]
    if s.kind == "mlp":
        return s.net.forward(s.feat, s.out)
    grad, stats = s.net.gradients(s.feat, s.target, s.idx, s.idx.shape[0])
    return [grad, stats]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _sheet_counts(nx, ny):
    faces = 2 * (nx - 1) * (ny - 1)
    edges = (nx - 1) * ny + nx * (ny - 1) + (nx - 1) * (ny - 1)
    return nx * ny, faces, edges, 3 * faces - edges


def work(case):
    kind = case["kind"]
    if kind in ("frame", "contact", "sweep", "color"):
        V, F, E, B = _sheet_counts(case["nx"], case["ny"])
        per_sweep = 2 * (E + B) * 30 + 10 * V  # about 30 operations per constraint end
        if kind == "frame":
            n = case["substeps"] * case["iters"]
            return {"bytes": V * (2 * 32 + 8) + 12 * F + 12 * (E + B), "flops": n * per_sweep}
        if kind == "sweep":
            return {"bytes": V * (16 + 16 + 4) + 12 * (E + B), "flops": per_sweep}
        if kind == "contact":
            # positions and faces of both meshes in, the candidates (about 25 a vertex) and positions out
            return {"bytes": V * (16 + 16 + 16 + 4 * 26) + 12 * F + 20480 * 12 + 10242 * 16, "flops": 25 * V * 60}
        E -= 2 + E // 1000
        return {"bytes": 8 * E + 8 * E + 400, "flops": 0}
    if kind == "batch":
        sizes, b, fl = random.Random(case["instances"]), 0, 0
        for _ in range(case["instances"]):
            nx = sizes.randint(case["lo"], case["hi"])
            V, F, E, B = _sheet_counts(nx, max(case["lo"], nx - sizes.randint(0, 3)))
            b += V * (2 * 32 + 8) + 12 * F + 12 * (E + B)
            fl += case["substeps"] * case["iters"] * (2 * (E + B) * 30 + 10 * V)
        return {"bytes": b, "flops": fl}
    if kind == "lbvh":
        n = case["tris"]
        # face boxes and queries in; nodes, and per query its count and a few candidates out
        return {"bytes": n * (32 + 16) + 2 * n * 32 + n * (4 + 12), "flops": 0}
    rows = case["rows"]
    flops = 2 * (24 * 64 + 64 * 64 + 64 * 3)
    if kind == "mlp":
        return {"bytes": rows * (64 + 16) + 13000, "flops": rows * flops}
    return {"bytes": rows * (64 + 16 + 4) + 2 * 27000, "flops": rows * 3 * flops}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------
def _exact_sweep(case, seed):
    x, f, y, fixed = _sweep_inputs(case, seed)
    edges, bend, l0, bl0, m_inv = _topology(x, f)
    w = (fixed * m_inv).astype(np.float64)
    y = y.astype(np.float64)
    dt = DT / 10
    dx, cnt = np.zeros_like(y), np.zeros(y.shape[0])
    for pairs, rest, k in ((edges, l0, BENDING * dt * dt), (bend, bl0, STRETCH * dt * dt)):
        a, b = pairs[:, 0], pairs[:, 1]
        d = y[a] - y[b]
        length = np.sqrt((d * d).sum(1))
        ld = k * (length - rest) / (k * (w[a] + w[b]) + 1.0)
        t = (ld / length)[:, None] * d
        for c in range(3):
            dx[:, c] -= np.bincount(a, weights=w[a] * t[:, c], minlength=y.shape[0])
            dx[:, c] += np.bincount(b, weights=w[b] * t[:, c], minlength=y.shape[0])
        cnt += np.bincount(a, minlength=y.shape[0]) + np.bincount(b, minlength=y.shape[0])
    out = y + fixed[:, None] * dx / np.maximum(cnt, 1)[:, None]
    return torch.from_numpy(np.concatenate([out, w[:, None]], 1))


def _net64(params, feat):
    """Weights as the bfloat16 the network holds, biases as they are, everything else in 64 bits."""
    sizes = [(64, 32), (64,), (64, 64), (64,), (8, 64), (8,)]
    p, o = [], 0
    for s in sizes:
        n = int(np.prod(s))
        t = torch.from_numpy(params[o:o + n]).cuda().view(s)
        p.append((t.to(torch.bfloat16) if len(s) == 2 else t).double())
        o += n
    z1 = feat.double() @ p[0].T + p[1]
    h1 = z1 * torch.sigmoid(z1)
    z2 = h1 @ p[2].T + p[3]
    h2 = z2 * torch.sigmoid(z2)
    return p, z1, h1, z2, h2, h2 @ p[4].T + p[5]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "mlp":
        params, feat, _ = _mlp_inputs(case, seed)
        return torch.cat([_net64(params, part)[-1][:, :4] for part in feat.split(1 << 18)])
    if kind == "train":
        params, feat, target, idx = _train_inputs(case, seed)
        rows = feat[idx.long()]
        p, z1, h1, z2, h2, o = _net64(params, rows)
        t = target[idx.long()].double()
        e = t[:, 3:] * (o[:, :3] - t[:, :3])
        d_out = torch.zeros_like(o)
        d_out[:, :3] = 2.0 * e / rows.shape[0]
        slope = lambda z: torch.sigmoid(z) * (1.0 + z * (1.0 - torch.sigmoid(z)))  # noqa: E731
        d2 = (d_out @ p[4]) * slope(z2)
        d1 = (d2 @ p[2]) * slope(z1)
        grad = torch.cat([(d1.T @ rows.double()).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0),
                          (d_out.T @ h2).reshape(-1), d_out.sum(0)])
        stats = torch.zeros(4, dtype=torch.float64, device="cuda")
        stats[0] = (e * (o[:, :3] - t[:, :3])).sum()
        return [grad, stats]
    # frames: hundreds of sweeps and contact passes over changing candidate lists, far over 20 seconds in 64 bits;
    # contact: whole numbers and, in the last place, positions after thousands of region decisions;
    # broad phase and colouring: whole numbers and copies of the inputs' bounds
    return None

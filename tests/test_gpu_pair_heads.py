"""Chunk heads of the vertex-vs-cloth pair list: frames with and without them
end in the same state bit for bit -- a chunk is passed over only when none of
its pairs could have added anything."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene(pkg, nx, ny, seed, *, renumber, layers, speed):
    """A wavy sheet (or two, 3 mm apart and moving into each other) falling on
    a box, with edges about eight contact distances long."""
    rng = np.random.default_rng(seed)
    X, F = [], []
    h = 0.03
    for k in range(layers):
        i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
        x = np.stack([h * i, h * j, 0.004 * np.sin(1.3 * i) * np.cos(0.9 * j) + 0.003 * k], -1).reshape(-1, 3)
        X.append(x + rng.normal(0, 2e-4, x.shape))
        a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1)
        f = np.stack([np.stack([a, a + ny, a + 1], -1), np.stack([a + 1, a + ny, a + ny + 1], -1)], 1).reshape(-1, 3)
        F.append(f + k * nx * ny)
    x, f = np.concatenate(X).astype(np.float32), np.concatenate(F).astype(np.int32)
    v = np.zeros((x.shape[0], 3), np.float32)
    v[:, 2] = -0.5
    v[:nx * ny, 2] = speed if layers > 1 else -speed
    v += rng.normal(0, 0.2 * speed, v.shape).astype(np.float32)
    if renumber:
        p = rng.permutation(x.shape[0])
        inv = np.empty_like(p)
        inv[p] = np.arange(p.shape[0])
        x, v, f = x[p], v[p], inv[f].astype(np.int32)
    sx, sf = pkg.box_mesh(0.4, center=(h * nx / 2, h * ny / 2, -0.206))
    return x, f, v, sx, sf


def _run(pkg, args, heads, opt, graph):
    x, f, v, sx, sf = _scene(pkg, **args)
    m, s = pkg.TriMesh(x, f, device="cuda"), pkg.TriMesh(sx, sf, device="cuda", is_static=True)
    sim = pkg.Solver(m, s, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8, g=(0, 0, -9.81),
                     dt=1 / 60, n_iter=opt.pop("n_iter", 9), rebuild="substep", bending_on=opt.pop("bending_on", "y"))
    sim.enable_collision_handling = True
    sim.use_graph = graph
    sim.HEADS_MIN_PAIRS, sim.HEADS_MIN_ITERATIONS = opt.pop("min_pairs", 1), 2
    sim.pair_heads = heads
    sewing = opt.pop("sewing", None)
    sim._packed_sweep = opt.pop("packed", False)
    for k, val in opt.items():
        assert hasattr(sim, k), k
        setattr(sim, k, val)
    if sewing is not None:
        sim.set_sewing_pairs(sewing, 1e5)
    m.v4[:, :3] = torch.from_numpy(v).cuda()
    for _ in range(3):
        sim.forward(4)
    torch.cuda.synchronize()
    return sim, m.x4.cpu().numpy().copy(), m.v4.cpu().numpy().copy()


BASE = dict(nx=37, ny=29, seed=1, renumber=False, layers=1, speed=0.3)


@pytest.mark.parametrize("args,opt,graph", [
    (BASE, {}, False),
    (BASE, dict(n_iter=6), True),
    (BASE, dict(bending_on="x"), True),
    (dict(BASE, layers=2, speed=2.0), {}, True),                # layers that come into contact within a substep
    (dict(BASE, layers=2, speed=2.0), dict(bending_on="x", n_iter=8), False),
    (dict(BASE, renumber=True), {}, True),                      # chunks with too many blocks
    (dict(BASE, layers=2, speed=1.0, renumber=True), dict(n_iter=7), False),
    (BASE, dict(min_pairs=37 * 29 * 20, padding=0.005), True),  # fewer pairs, which the device alone knows
    (dict(BASE, nx=3, ny=3), {}, False),
    (dict(BASE, nx=90, ny=64, layers=2, speed=1.0), dict(fast_math=True), True),
    (dict(BASE, layers=2, speed=1.5), dict(enable_edge_edge=True), False),
    (dict(BASE, layers=2, speed=1.5), dict(sewing=np.array([[0, 900], [40, 80], [500, 1500]], np.int32)), True),
    (dict(BASE, layers=2, speed=1.5), dict(packed=True, packed_form=0), True),
    (dict(BASE, layers=2, speed=1.5), dict(packed=True, packed_form=1, fast_math=True), True),
])
def test_frames_with_and_without(pkg, args, opt, graph):
    on, x1, v1 = _run(pkg, args, True, dict(opt), graph)
    off, x0, v0 = _run(pkg, args, False, dict(opt), graph)
    assert np.array_equal(x1, x0) and np.array_equal(v1, v0)
    assert np.isfinite(x1).all()
    assert off._heads is None and on._heads is not None
    if not args["renumber"]:
        used = (on._heads[0][:-16].view(torch.float32).view(-1, 16)[:, 0] > 0).any().item()
        assert used == (opt.get("min_pairs", 1) == 1)


@pytest.mark.parametrize("variant", range(13))
def test_every_sweep_and_projection_configuration(pkg, variant):
    from starlab_physics_gb300 import _lib
    from starlab_physics_gb300.autotune import variants

    args = dict(BASE, layers=2, speed=1.5)
    n_pairs = int(_lib.sx.sx_contact_pairs_project_variants())
    for by in ("x", "y"):
        opt = dict(sweep_variant=variant % len(variants()), pairs_variant=variant % n_pairs, bending_on=by)
        _, x1, _ = _run(pkg, args, True, dict(opt), True)
        _, x0, _ = _run(pkg, args, False, dict(opt), True)
        assert np.array_equal(x1, x0)


def test_positions_that_are_not_numbers(pkg):
    """A vertex that loses its position within the iterations hides no contact
    of the others, and its own pairs are tested."""
    out = []
    for heads in (True, False):
        x, f, v, sx, sf = _scene(pkg, **dict(BASE, layers=2, speed=2.0))
        m, s = pkg.TriMesh(x, f, device="cuda"), pkg.TriMesh(sx, sf, device="cuda", is_static=True)
        sim = pkg.Solver(m, s, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8, g=(0, 0, -9.81),
                         dt=1 / 60, n_iter=8, rebuild="substep", bending_on="y")
        sim.enable_collision_handling = True
        sim.HEADS_MIN_PAIRS, sim.HEADS_MIN_ITERATIONS = 1, 2
        sim.pair_heads, sim._in_substep = heads, True
        m.v4[:, :3] = torch.from_numpy(v).cuda()
        sim.build_bvhs()
        sim.compute_y(1 / 600)
        for it in range(8):
            sim.solve_constraints_jacobi_x(1 / 600, it == 0, it)
            assert sim._heads_on == heads
            if it == 2:
                m.y4[500, 0] = float("nan")
                m.y4[700, 1] = float("inf")
        torch.cuda.synchronize()
        out.append(m.y4.cpu().numpy().copy())
    assert np.isnan(out[0]).any() and np.isfinite(out[0]).any() and np.array_equal(out[0], out[1], equal_nan=True)


def test_own_steps_are_not_skipped_over(pkg):
    """A solver whose collision step moves vertices itself tests every pair."""
    class Pushed(pkg.Solver):
        def solve_collision_constraints_x(self, *a, **k):
            self.mesh_dy.y4[: self.mesh_dy.num_verts // 2, 2] += 2e-3
            super().solve_collision_constraints_x(*a, **k)

    out = []
    for heads in (True, False):
        x, f, v, sx, sf = _scene(pkg, **dict(BASE, layers=2, speed=1.0))
        m, s = pkg.TriMesh(x, f, device="cuda"), pkg.TriMesh(sx, sf, device="cuda", is_static=True)
        sim = Pushed(m, s, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8, g=(0, 0, -9.81),
                     dt=1 / 60, n_iter=8, rebuild="substep", bending_on="y")
        sim.enable_collision_handling = True
        sim.HEADS_MIN_PAIRS, sim.HEADS_MIN_ITERATIONS, sim.pair_heads = 1, 2, heads
        m.v4[:, :3] = torch.from_numpy(v).cuda()
        sim.forward(3)
        out.append(m.x4.cpu().numpy().copy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])


def test_refuses(pkg):
    from starlab_physics_gb300 import _lib

    sx = _lib.sx
    t = torch.zeros(4096, device="cuda")
    p = t.data_ptr()
    need = int(sx.sx_contact_pairs_heads_bytes(4, 8))
    s = torch.cuda.current_stream().cuda_stream
    with pytest.raises(Exception):
        sx.sx_contact_pairs_heads(4, 0, 8, p, p, p, 1e-4, 1, p, p, p, need - 1, s)
    with pytest.raises(Exception):
        sx.sx_contact_pairs_heads(4, 0, 8, p, p, p, 1e-4, 1, p, p, p + 4, need, s)
    with pytest.raises(Exception):
        sx.sx_jacobi_sweep_tracked(p, p, p, p, p, p, 4, 1.0, 1.0, 1, 0, 0, p, p, None, s)

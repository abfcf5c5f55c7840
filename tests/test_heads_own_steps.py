"""Chunk heads stay off where a solver brings a step of its own that could move
vertices between a tracked sweep and the projection, and only there."""
import numpy as np
import pytest
import torch

STEPS = ["solve_constraints_jacobi_x", "spring_sweep", "solve_collision_constraints_x",
         "solve_edge_edge_constraints_x", "contact_cull_d2"]


def _sheet(nx, ny, h=0.03, layers=1, gap=3e-3):
    X, F = [], []
    for k in range(layers):
        i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
        X.append(np.stack([h * i, h * j, 0.004 * np.sin(1.3 * i) * np.cos(0.9 * j) + gap * k], -1).reshape(-1, 3))
        a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1) + k * nx * ny
        F += [np.stack([a, a + ny, a + 1], -1), np.stack([a + 1, a + ny, a + ny + 1], -1)]
    return np.concatenate(X).astype(np.float32), np.concatenate(F).astype(np.int32)


def _solver(pkg, cls, device, **kw):
    x, f = _sheet(37, 29, **kw)
    sim = cls(pkg.TriMesh(x, f, device=device), None, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8,
              g=(0, 0, -9.81), dt=1 / 60, n_iter=8, rebuild="substep", bending_on="y")
    sim.enable_collision_handling = True
    sim.HEADS_MIN_PAIRS, sim.HEADS_MIN_ITERATIONS = 1, 2
    return sim


@pytest.fixture
def stubbed(monkeypatch, pkg):
    from starlab_physics_gb300 import solver

    monkeypatch.setattr(solver, "LBVH_CELL", lambda *a, **k: None)  # its constructor launches kernels


@pytest.mark.parametrize("name", STEPS)
def test_a_step_of_ones_own(pkg, stubbed, name):
    base = getattr(pkg.Solver, name)
    own = type("Own", (pkg.Solver,), {name: lambda self, *a, **k: base(self, *a, **k)})
    assert not _solver(pkg, own, "cpu")._heads_wanted()
    sim = _solver(pkg, pkg.Solver, "cpu")
    assert sim._heads_wanted()
    before = getattr(sim, name)
    setattr(sim, name, lambda *a, **k: before(*a, **k))  # as a profiler wraps a step
    assert not sim._heads_wanted()
    setattr(sim, name, before)
    assert sim._heads_wanted()
    setattr(sim, name, getattr(_solver(pkg, pkg.Solver, "cpu"), name))  # another solver's
    assert not sim._heads_wanted()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["solve_constraints_jacobi_x", "solve_edge_edge_constraints_x"])
def test_own_motion_is_seen(pkg, name):
    """Vertices moved between a sweep and the projection: the same state with and
    without heads."""
    def push(self):
        self.mesh_dy.y4[: self.mesh_dy.num_verts // 2, 2] += 2e-3

    class Own(pkg.Solver):
        def solve_constraints_jacobi_x(self, dt, first_iteration=True, iteration=0, loop=0, in_loop=False):
            if first_iteration or name != "solve_constraints_jacobi_x":
                return super().solve_constraints_jacobi_x(dt, first_iteration, iteration, loop, in_loop)
            self.spring_sweep(dt, iteration, loop)
            push(self)
            self.solve_collision_constraints_x(iteration=iteration)

    class OwnEdges(pkg.Solver):
        def solve_edge_edge_constraints_x(self, *a, **k):
            push(self)

    out = []
    for heads in (True, False):
        sim = _solver(pkg, Own if name == "solve_constraints_jacobi_x" else OwnEdges, "cuda", layers=2, gap=3e-2)
        sim.enable_edge_edge = name == "solve_edge_edge_constraints_x"
        sim.padding, sim.pair_heads = 0.05, heads
        sim.forward(3)
        out.append(sim.mesh_dy.x4.cpu().numpy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])

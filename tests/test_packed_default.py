"""Which adjacency a default sweep reads.  The packed copy stands in for
``mesh.adj`` only while it is a copy of it: rest lengths edited after the mesh was
made count, whenever the solver was made."""
import copy

import numpy as np
import pytest
import torch


def _mesh(pkg, nx=410, ny=395):
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    x = np.stack([0.01 * i, 0.01 * j, 0.001 * np.sin(0.7 * i)], -1).reshape(-1, 3).astype(np.float32)
    a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1)
    f = np.stack([np.stack([a, a + ny, a + 1], -1), np.stack([a + 1, a + ny, a + ny + 1], -1)], 1).reshape(-1, 3)
    return pkg.TriMesh(x, f.astype(np.int32), device="cpu")


def _solver(pkg, mesh, monkeypatch):
    from starlab_physics_gb300 import solver

    monkeypatch.setattr(solver, "LBVH_CELL", lambda *a, **k: None)  # its constructor launches kernels
    sim = pkg.Solver(mesh, None, 4e-6, 1e5, 1e8, (0.0, 0.0, -9.81), 1 / 60, bending_on="y")
    assert sim._default_packed == [-1, 3]
    return sim


def _shrink(mesh):
    mesh.adj[:, 1] = (0.9 * mesh.adj[:, 1].contiguous().view(torch.float32)).view(torch.int32)


def test_edits_of_the_adjacency_count_whenever_the_solver_is_made(pkg, monkeypatch):
    mesh = _mesh(pkg)
    before = _solver(pkg, mesh, monkeypatch)
    assert before._packed_choice(1) == 3 and before._packed_choice(0) == -1
    _shrink(mesh)
    after = _solver(pkg, mesh, monkeypatch)
    assert not np.array_equal(mesh.adj_rest32.numpy().view(np.uint32) & 0x7fffffff, mesh.adj[:, 1].numpy().view(np.uint32))
    assert before._packed_choice(1) == -1 and after._packed_choice(1) == -1


@pytest.mark.parametrize("change", ["replace", "packed", "copy", "deepcopy", "inference"])
def test_other_ways_to_part_from_the_copy(pkg, monkeypatch, change):
    if change == "inference":
        with torch.inference_mode():
            mesh = _mesh(pkg)
    else:
        mesh = _mesh(pkg)
    same = False
    if change == "replace":
        mesh.adj = mesh.adj.clone()
    elif change == "packed":
        mesh.adj_rest32 ^= 1
    elif change == "copy":
        mesh, same = copy.copy(mesh), True
    elif change == "deepcopy":  # counts as changed: its tensors' versions start anew
        _shrink(mesh)
        mesh = copy.deepcopy(mesh)
    assert _solver(pkg, mesh, monkeypatch)._packed_choice(1) == (3 if same else -1)
    mesh._packed_state.__reduce__()


def test_explicit_choices_stand(pkg, monkeypatch):
    mesh = _mesh(pkg)
    sim = _solver(pkg, mesh, monkeypatch)
    sim.sweep_variant = 5
    assert sim._packed_choice(1) == -1
    sim.sweep_variant, sim._packed_sweep, sim.packed_form = 0, True, 1
    assert sim._packed_choice(1) == 1


@pytest.mark.gpu
def test_a_users_own_graph_reads_the_adjacency(pkg):
    """Captured by a user, a sweep sees the rest lengths that stand in ``mesh.adj`` at
    each replay."""
    host = _mesh(pkg)
    mesh = pkg.TriMesh(host.x0_np, host.fid_np, device="cuda")
    sim = pkg.Solver(mesh, None, 4e-6, 1e5, 1e8, (0.0, 0.0, -9.81), 1 / 60, bending_on="y")
    sim.fast_math = True
    assert sim._packed_choice(1) == 3
    noise = np.random.default_rng(2).normal(0, 1e-4, mesh.x0_np.shape).astype(np.float32)
    mesh.y4[:, :3] = mesh.x0 + torch.from_numpy(noise).cuda()
    start, src = mesh.y4.clone(), mesh.y4
    sim.spring_sweep(1e-3)
    sim._swap_y()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sim.spring_sweep(1e-3)
    out = mesh.y4
    _shrink(mesh)
    src.copy_(start)
    graph.replay()
    got = out.clone()
    sim.sweep_variant = sim._default_variant[1]
    src.copy_(start)
    sim._swap_y()
    sim.spring_sweep(1e-3)
    torch.cuda.synchronize()
    assert torch.equal(got, mesh.y4) and not torch.equal(got, start)


def test_meshes_without_the_copys_state(pkg, monkeypatch):
    """A mesh from a file that has no state, and one of a user's own class without
    packed arrays: swept over ``mesh.adj``."""
    mesh = _mesh(pkg)
    sim = _solver(pkg, mesh, monkeypatch)
    del mesh._packed_state
    assert sim._packed_choice(1) == -1

    class Own:
        def __init__(self, m):
            self.__dict__.update({k: v for k, v in vars(m).items() if k not in ("adj_nbr16", "adj_rest32")})

    sim = pkg.Solver(Own(mesh), None, 4e-6, 1e5, 1e8, (0.0, 0.0, -9.81), 1 / 60, bending_on="y")
    assert sim._default_packed == [-1, -1] and sim._packed_choice(1) == -1

"""A solver with a tree of a user's own, whose ``traverse`` takes the arguments it
always took: called so, and on the stream its work belongs to."""
import numpy as np
import pytest
import torch


def _solver(pkg, device):
    x, f = pkg.grid_cloth(9)[:2]
    box = pkg.box_mesh(0.5, center=(0.5, 0.5, 0.6))
    sim = pkg.Solver(pkg.TriMesh(x, f, device=device), pkg.TriMesh(*box, device=device, is_static=True), 1e-4, 1e5, 1e8,
                     (0, 0, -9.81), 1 / 60)
    sim.enable_collision_handling = True
    return sim


def test_arguments(pkg, monkeypatch):
    from starlab_physics_gb300 import solver

    class Tree:
        def __init__(self, *a, **k):
            self.calls = 0

        def traverse(self, points4, padding, cap, cand, num, status):
            self.calls += 1

    monkeypatch.setattr(solver, "LBVH_CELL", Tree)
    sim = _solver(pkg, "cpu")
    sim.broadphase_lbvh()
    assert sim.lbvh_st.calls == 1 and sim.lbvh_dy.calls == 2


@pytest.mark.gpu
def test_stream(pkg):
    from starlab_physics_gb300 import lbvh

    streams = []

    class Tree(lbvh.LBVH_CELL):
        def traverse(self, points4, padding, cap, cand, num, status):
            streams.append(torch.cuda.current_stream().cuda_stream)
            num.zero_()  # work of its own on the current stream
            super().traverse(points4, padding, cap, cand, num, status)

    want = _solver(pkg, "cuda")
    got = _solver(pkg, "cuda")
    got.lbvh_st.__class__ = got.lbvh_dy.__class__ = Tree
    for sim in (want, got):
        for _ in range(3):
            sim.forward(4)
    assert torch.equal(want.mesh_dy.x4, got.mesh_dy.x4) and len(set(streams)) == 3
    assert np.isfinite(got.mesh_dy.x4.cpu().numpy()).all()

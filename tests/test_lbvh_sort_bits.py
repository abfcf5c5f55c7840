"""The sort under a hierarchy takes all code bits whatever ``sort_bits`` says: a
Karras build over codes in no full order has nodes without a parent, whose
uninitialised links a refit would follow."""
import numpy as np
import pytest
import torch


@pytest.mark.parametrize("sort_bits,want", [(1, 30), (16, 30), (30, 30), (32, 32)])
def test_bits_of_the_sort(pkg, monkeypatch, sort_bits, want):
    from starlab_physics_gb300 import lbvh

    tree, bits = pkg.LBVH(50, "cpu", sort_bits=sort_bits), []

    class Recorder:
        def sx_radix_sort_pairs(self, keys, vals, n, b, *rest):
            bits.append(b)

    monkeypatch.setattr(lbvh, "sx", Recorder())
    monkeypatch.setattr(lbvh, "stream_handle", lambda stream=None: 0)
    tree.sort()
    assert bits == [want]


@pytest.mark.gpu
def test_tree_is_the_fully_sorted_one(pkg):
    rng = np.random.default_rng(1)
    n = 5000
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    lo, hi = torch.zeros((n, 4), device="cuda"), torch.zeros((n, 4), device="cuda")
    lo[:, :3], hi[:, :3] = torch.from_numpy(c - 0.01).cuda(), torch.from_numpy(c + 0.01).cuda()
    box = torch.tensor([0, 0, 0, 1, 1, 1.0], device="cuda")
    out = []
    for bits in (12, 32):
        T = pkg.LBVH(n, sort_bits=bits)
        T.build(lo, hi, box)
        out.append([*T.query(lo, 0.01, 64, cand=torch.zeros((n, 64), dtype=torch.int32, device="cuda")), T.parent])
    assert all(torch.equal(a, b) for a, b in zip(*out))

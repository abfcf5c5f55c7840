"""``LBVH.query`` walks the tree's arrays as they are: its child records stand in
for them only until one is edited.  And the records against the arrays, on trees
that nothing has touched."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tree(pkg, n, kind="soup", **kw):
    rng = np.random.default_rng(n + len(kind))
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    if kind == "repeated":
        c = c[rng.integers(0, max(n // 5, 1), n)]
    r = rng.uniform(0.001, 0.02, (n, 3)).astype(np.float32)
    lo, hi = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    lo[:, :3], hi[:, :3] = c - r, c + r
    if kind == "odd":
        lo[::11, 0] = np.nan
        hi[3::17, 1] = np.nan
        lo[5::23, 2], hi[5::23, 2] = -np.inf, np.inf
    T = pkg.LBVH(n, **kw)
    lo, hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()
    T.build(lo, hi, torch.tensor([0, 0, 0, 1, 1, 1.0], device="cuda"))
    p = np.zeros((3001, 4), np.float32)
    p[:, :3] = rng.uniform(-0.1, 1.1, (3001, 3))
    return T, torch.from_numpy(p).cuda(), lo, hi


def _walk(T, p4, pad, cap):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    cand = torch.full((p4.shape[0], cap), -7, dtype=torch.int32, device="cuda")
    num = torch.zeros(p4.shape[0], dtype=torch.int32, device="cuda")
    sx.sx_face_bvh_traverse(T.n, ptr(p4), p4.shape[0], pad, ptr(T.child_a), ptr(T.child_b), ptr(T.sorted_ids),
                            ptr(T.node_min4), ptr(T.node_max4), cap, ptr(cand), ptr(num), ptr(T.status),
                            stream_handle())
    return cand, num


def _query(T, p4, pad, cap):
    return T.query(p4, pad, cap, cand=torch.full((p4.shape[0], cap), -7, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("n", [1, 2, 8, 9, 65, 512, 4097, 32769])
@pytest.mark.parametrize("kind", ["soup", "repeated", "odd"])
@pytest.mark.parametrize("coherent", [0, 1 << 30])
def test_records_equal_the_arrays(pkg, n, kind, coherent):
    T, p4, _, _ = _tree(pkg, n, kind)
    T.COHERENT_MIN_QUERIES = coherent
    assert T._aux_of.unchanged(*T._tree())
    for cap, pad in ((3, 0.1), (16, 0.01)):
        for a, b in zip(_query(T, p4, pad, cap), _walk(T, p4, pad, cap)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("edit", ["boxes", "ids", "replaced", "hierarchy", "tie"])
def test_edited_arrays_count(pkg, edit):
    T, p4, lo, hi = _tree(pkg, 4000)
    before = _query(T, p4, 0.01, 64)
    if edit == "boxes":
        T.node_min4[:, :3] -= 0.05
        T.node_max4[:, :3] += 0.05
    elif edit == "ids":
        T.sorted_ids += 1
    elif edit == "replaced":
        T.node_min4 = T.node_min4 - 0.05
    elif edit == "hierarchy":  # other faces under the old boxes
        T.morton(lo.flip(0).contiguous(), hi.flip(0).contiguous(), T.box6)
        T.sort()
    else:
        T.tie = 0
        T.refit(lo + 0.05, hi + 0.05)
        T.tie = 1
    got = _query(T, p4, 0.01, 64)
    for a, b in zip(got, _walk(T, p4, 0.01, 64)):
        assert torch.equal(a, b)
    assert not torch.equal(got[0], before[0])
    T.build(lo, hi, T.box6)
    assert all(torch.equal(a, b) for a, b in zip(_query(T, p4, 0.01, 64), before))


def test_tie_rule_changed_after_construction(pkg):
    T, p4, lo, hi = _tree(pkg, 4000, tie=0)
    T.tie = 1
    T.build(lo, hi, T.box6)
    for a, b in zip(_query(T, p4, 0.01, 64), _walk(T, p4, 0.01, 64)):
        assert torch.equal(a, b)

"""Refit by ranges and child records: node boxes equal to the climb's and query results (lists in
order, counts, overflow flag) equal to the stack traversal's, at sizes around
the level boundaries, with repeated codes, truncated lists, NaN and infinite
boxes, and in both query orders."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 255, 256, 257, 511, 512, 513, 4095, 4097, 32768, 32769,
                               262145])
@pytest.mark.parametrize("kind", ["soup", "repeated", "odd"])
def test_levels_equal_climb_and_stack(pkg, n, kind):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

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
        lo[7::29, :3] = -0.0
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    mn, mx = t(lo), t(hi)
    box = t(np.array([0, 0, 0, 1, 1, 1], np.float32))
    T = pkg.LBVH(n)
    T.build(mn, mx, box)
    got = (T.node_min4.clone(), T.node_max4.clone())
    T.node_min4.fill_(3.0)
    T.node_max4.fill_(3.0)
    sx.sx_face_bvh_refit_tiled(n, ptr(T.sorted_ids), ptr(mn), ptr(mx), ptr(T.child_a), ptr(T.child_b), ptr(T.parent),
                               ptr(T.range_l), ptr(T.range_r), ptr(T.node_min4), ptr(T.node_max4), ptr(T.flags),
                               ptr(T.status), stream_handle())
    for a, b in zip(got, (T.node_min4, T.node_max4)):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=True)
    for q, cap, pad in ((1, 8, 0.05), (37, 3, 0.1), (20000, 16, 0.003)):
        p = np.zeros((q, 4), np.float32)
        p[:, :3] = rng.uniform(-0.1, 1.1, (q, 3))
        p[::13, 0] = np.nan
        p4 = t(p)
        want_c = torch.full((q, cap), -7, dtype=torch.int32, device="cuda")
        want_n = torch.zeros(q, dtype=torch.int32, device="cuda")
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        sx.sx_face_bvh_traverse(n, ptr(p4), q, pad, ptr(T.child_a), ptr(T.child_b), ptr(T.sorted_ids),
                                ptr(T.node_min4), ptr(T.node_max4), cap, ptr(want_c), ptr(want_n), ptr(st),
                                stream_handle())
        for coherent in (0, 1 << 30):
            T.COHERENT_MIN_QUERIES = coherent
            cand = torch.full((q, cap), -7, dtype=torch.int32, device="cuda")
            num = torch.zeros(q, dtype=torch.int32, device="cuda")
            st2 = torch.zeros(1, dtype=torch.int32, device="cuda")
            T.query(p4, pad, cap, cand, num, st2)
            assert torch.equal(num, want_n) and torch.equal(cand, want_c) and torch.equal(st, st2)


@pytest.mark.parametrize("n,first,bits", [(1, 3, 8), (3000, 14, 16), (70001, 0, 30), (70001, 20, 12), (2049, 31, 1)])
def test_sort_by_bit_range(pkg, n, first, bits):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    rng = np.random.default_rng(n + first)
    k = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    K = torch.from_numpy(k.view(np.int32).copy()).cuda()
    V = torch.arange(n, dtype=torch.int32, device="cuda")
    ws = torch.empty(int(sx.sx_radix_sort_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    sx.sx_radix_sort_pairs_bits(ptr(K), ptr(V), n, first, bits, ptr(ws), ws.numel(), stream_handle())
    order = np.argsort((k >> np.uint32(first)) & np.uint32((1 << bits) - 1), kind="stable")
    assert np.array_equal(V.cpu().numpy(), order) and np.array_equal(K.cpu().numpy().view(np.uint32), k[order])

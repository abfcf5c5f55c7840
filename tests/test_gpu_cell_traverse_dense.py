"""Cell-grid queries over cells of a few to a few hundred faces, with more
queries than warps resident at once: candidate lists equal the oracle's walk,
order included."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces,edges,pad,cap", [
    (40, 9001, 0.3, 40),          # few faces in a large grid: whole columns empty
    (3000, 20011, 0.02, 24),      # cells of a handful, the lists overflow at times
    (60000, 9001, 0.004, 64),     # hundreds a cell: one cell after the other
    (60000, 1, 0.004, 64),
    (1, 300, 0.1, 1),
])
def test_dense_cells(pkg, po, faces, edges, pad, cap):
    rng = np.random.default_rng(faces + edges)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    # a curved sheet through the grid, a cluster of faces in one corner
    c = rng.uniform(0, 1, (faces, 3))
    c[:, 2] = 0.5 + 0.3 * np.sin(3 * c[:, 0])
    c[: faces // 5] = 0.02 + 0.03 * rng.uniform(0, 1, (faces // 5, 3))
    e = rng.uniform(0, 0.006, (faces, 3))
    mn, mx = np.zeros((faces, 4), np.float32), np.zeros((faces, 4), np.float32)
    mn[:, :3], mx[:, :3] = c - e, c + e
    box = np.array([0, 0, 0, 1, 1, 1], np.float32)
    bvh = pkg.LBVH_CELL(faces, "cuda")
    bvh.build(None, t(box), face_min4=t(mn), face_max4=t(mx))
    ref = po.CellBVH()
    ref.build(mn, mx, box)
    assert np.array_equal(bvh.sorted_face_ids.cpu().numpy(), ref.sorted_face_ids)
    pts = np.zeros((2 * edges, 4), np.float32)
    pts[:, :3] = c[rng.integers(0, faces, 2 * edges)] + rng.normal(0, 0.01, (2 * edges, 3))
    pts[::97, 1] += 2.0  # outside the grid
    ends = np.arange(2 * edges, dtype=np.int32).reshape(-1, 2)
    pts[1::2, :3] = pts[::2, :3] + rng.normal(0, 0.005, (edges, 3)).astype(np.float32)
    i32 = dict(dtype=torch.int32, device="cuda")
    for by_edge in (False, True):
        n = edges if by_edge else 2 * edges
        cand, num, status = torch.full((n, cap), -1, **i32), torch.zeros(n, **i32), torch.zeros(1, **i32)
        if by_edge:
            bvh.traverse_edges(t(ends), n, t(pts), pad, cap, cand, num, status)
            qmn, qmx = po.edge_query_boxes(pts, ends, pad)
        else:
            bvh.traverse(t(pts), pad, cap, cand, num, status)
            qmn, qmx = po.query_boxes(pts, pad)
        rc, rn, rs = ref.traverse(qmn, qmx, cap)
        assert np.array_equal(num.cpu().numpy(), rn) and int(status.item()) == rs
        live = np.arange(cap)[None, :] < np.minimum(rn, cap)[:, None]
        assert np.array_equal(np.where(live, cand.cpu().numpy(), 0), np.where(live, rc, 0))

"""Cell-grid builds at the edges of their launches: one face, all faces in one cell,
cells at both ends of the grid, both sorts; everything equal to the oracle's bit for
bit, twice on one object."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("faces", [1, 2, 255, 256, 257, 5000, 65536, 65537, 140001])
@pytest.mark.parametrize("where", ["spread", "one cell", "ends"])
def test_build(pkg, po, faces, where):
    rng = np.random.default_rng(faces)
    c = rng.uniform(0, 1, (faces, 3))
    if where == "one cell":
        c = 0.5 + 0.01 * c
    elif where == "ends":
        c = np.where(rng.random((faces, 1)) < 0.5, 0.001, 0.999) * np.ones((1, 3))
    e = rng.uniform(0, 0.01, (faces, 3))
    mn, mx = np.zeros((faces, 4), np.float32), np.zeros((faces, 4), np.float32)
    mn[:, :3], mx[:, :3] = c - e, c + e
    bvh = pkg.LBVH_CELL(faces, "cuda")
    ref = po.CellBVH()
    for k, box in enumerate(([0, 0, 0, 1, 1, 1], [-0.1, -0.2, 0, 1.5, 1.2, 1.1])):
        box = np.array(box, np.float32)
        if k == 0:
            bvh.build(None, _t(box), face_min4=_t(mn), face_max4=_t(mx))
        else:
            bvh.build(None, tuple(box[:3]), tuple(box[3:]), face_min4=_t(mn), face_max4=_t(mx))
        ref.build(mn, mx, box)
        for got, want in ((bvh.prefix_sum_cell, ref.prefix), (bvh.sorted_face_ids, ref.sorted_face_ids),
                          (bvh.num_faces, ref.num_faces), (bvh.node_min4, ref.nmin4), (bvh.node_max4, ref.nmax4),
                          (bvh.cell_size, ref.cell_size), (bvh.box6, box)):
            assert np.array_equal(got.cpu().numpy(), want)
        assert (bvh.grid8[6:8].cpu().numpy() == 0).all()
        occ = bvh.grid8[8:].view(torch.int32).cpu().numpy().view(np.uint32)
        full = np.diff(ref.prefix, prepend=0).reshape(1024, 32) > 0
        assert np.array_equal(occ, (full << np.arange(32)).sum(1).astype(np.uint32))

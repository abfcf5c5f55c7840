"""Colourings that keep many messages waiting: larger sheets with and without their
bending pairs, and graphs whose edges wait for a vertex at the other end of a long
path.  The single block finishes them all (the spill word of the workspace stays
0), and the colours are the sequential ones."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sheet(pkg, n, bending):
    from starlab_physics_gb300.mesh import bending_pairs, edges_from_faces

    f = pkg.grid_cloth(n)[1]
    e = edges_from_faces(f)
    return n * n, np.concatenate([e, bending_pairs(f)]) if bending else e


def _path(n, kind):
    """A path of n edges, then edges between vertices as far apart as the path is
    long: half of them wait for their second vertex at one time."""
    path = np.stack([np.arange(n), np.arange(1, n + 1)], 1)
    i = np.arange(n // 2)
    far = np.stack([i, n - i], 1)
    if kind == "shuffled":
        far = far[np.random.default_rng(n).permutation(len(far))]
    if kind == "twice":  # a repeated edge gets both its messages from the one before it, in one step
        far = np.repeat(far, 2, axis=0)
    if kind == "hubs":  # colours past 30: messages whose sets lie in memory
        far = np.concatenate([far] + [np.stack([np.full(40, h), n + 1 + np.arange(40) + 40 * k], 1)
                                      for k, h in enumerate((5, n // 2 - 7, n - 5))] + [far[::3]])
    return int(max(path.max(), far.max())) + 1, np.concatenate([path, far])


CASES = {"sheet256": lambda p: _sheet(p, 256, True), "sheet512": lambda p: _sheet(p, 512, False),
         "sheet512+": lambda p: _sheet(p, 512, True), "sheet1024": lambda p: _sheet(p, 1024, False)}
for _n, _k in ((200, "plain"), (20000, "plain"), (20000, "shuffled"), (24000, "twice"), (20000, "hubs"),
               (300000, "shuffled"), (1800000, "plain")):
    CASES[f"path{_n}-{_k}"] = lambda p, n=_n, k=_k: _path(n, k)


@pytest.mark.parametrize("name", list(CASES))
def test_the_block_finishes(pkg, po, name):
    from starlab_physics_gb300._lib import sx

    nv, e = CASES[name](pkg)
    e = np.ascontiguousarray(e, np.int32)
    E = e.shape[0]
    t = torch.from_numpy(e).cuda()
    ws = torch.zeros(int(sx.sx_color_workspace_bytes(nv, E)), dtype=torch.uint8, device="cuda")
    out = torch.empty((2, E), dtype=torch.int32, device="cuda")
    prefix = torch.zeros(100, dtype=torch.int32, device="cuda")
    sx.sx_color_edges_greedy(t.data_ptr(), E, nv, 100, out[0].data_ptr(), out[1].data_ptr(), prefix.data_ptr(),
                             ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    status, spill = ws[:8].view(torch.int32).tolist()
    color, order, start = po.color_edges(nv, e)
    assert status == 0 and spill == 0
    assert np.array_equal(out[0].cpu().numpy(), color) and np.array_equal(out[1].cpu().numpy(), order)
    assert np.array_equal(prefix.cpu().numpy(), start)


def _paths(n, length):
    """n paths of as many edges, one seed each, numbered one after the other."""
    first = np.arange(n)[:, None] * (length + 1)
    a = (first + np.arange(length)[None]).reshape(-1)
    return n * (length + 1), np.stack([a, a + 1], 1)


@pytest.mark.parametrize("name", ["64 paths", "65 paths", "153 paths", "20000 paths", "matching", "icosphere",
                                  "shuffled", "few blocks"])
def test_many_seeds(pkg, po, name):
    from starlab_physics_gb300.mesh import edges_from_faces

    rng = np.random.default_rng(7)
    if name.endswith("paths"):
        n = int(name.split()[0])
        nv, e = _paths(n, 37 if n < 1000 else 4)
    elif name == "matching":
        nv, e = 40000, np.arange(40000).reshape(-1, 2)
    elif name == "few blocks":  # fewer edges than a block of each SM takes, most of them seeds
        nv, e = _paths(90, 2)
    else:
        f = pkg.icosphere(5, 0.3, (0.0, 0.0, 0.0))[1] if name == "icosphere" else pkg.grid_cloth(150)[1]
        e, nv = edges_from_faces(f), int(f.max()) + 1
        if name == "shuffled":
            e = e[rng.permutation(len(e))]
    gc = pkg.GraphColoring(nv, e.astype(np.int32))
    color, order, start = po.color_edges(nv, np.ascontiguousarray(e, np.int32))
    assert np.array_equal(gc.edges_color.cpu().numpy(), color)
    assert np.array_equal(gc.sorted_edges_sequence_for_color.cpu().numpy(), order)
    assert np.array_equal(gc.color_prefix_sum.cpu().numpy(), start)

"""The colouring against the oracle's sequential first-fit on graphs that reach
every branch of the propagation: hubs with more than 30 and more than 100
colours, too few colours, self loops and repeated edges, one seed or many, wide
fronts that overflow a block's ring, and sizes around the block and share edges."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tree(levels):
    """Every coloured edge makes two more ready: the front doubles per level."""
    edges, front, nv = [(0, 1)], [(0, 1)], 2
    for _ in range(levels):
        nxt = []
        for u, v in front:
            for w in (u, v):
                nxt.append((w, nv))
                nv += 1
        edges += nxt
        front = nxt
    return nv, np.asarray(edges, np.int32)


def _graph(kind, rng):
    if kind.startswith("random"):
        n = int(kind[6:])
        e = rng.integers(0, max(n // 3, 2), (n, 2)).astype(np.int32)
        return max(n // 3, 2), e
    if kind == "hub35":
        return 400, np.concatenate([np.stack([np.zeros(35, int), np.arange(1, 36)], 1),
                                    rng.integers(1, 400, (900, 2))]).astype(np.int32)
    if kind == "hubs":  # two hubs of 110 joined by edges in the middle of their lists
        a = np.stack([np.zeros(110, int), np.arange(2, 112)], 1)
        b = np.stack([np.ones(110, int), np.arange(112, 222)], 1)
        e = np.concatenate([a[:60], b[:50], [[0, 1]], a[60:], [[1, 0]], b[50:]])
        return 222, e.astype(np.int32)
    if kind == "clique":
        i, j = np.triu_indices(60, 1)
        e = np.stack([i, j], 1)
        return 60, e[rng.permutation(len(e))].astype(np.int32)
    if kind == "loops":
        e = rng.integers(0, 40, (600, 2))
        e[::9, 1] = e[::9, 0]
        e[100:120] = e[80:100]
        return 40, e.astype(np.int32)
    if kind == "sheet":
        n = 97
        i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        v = i * n + j
        e = np.concatenate([np.stack([v[:-1].ravel(), v[1:].ravel()], 1), np.stack([v[:, :-1].ravel(), v[:, 1:].ravel()], 1),
                            np.stack([v[:-1, :-1].ravel(), v[1:, 1:].ravel()], 1)])
        e = e[np.lexsort((e[:, 1], e[:, 0]))]
        return n * n, e.astype(np.int32)
    if kind == "matching":
        return 60000, rng.permutation(60000).reshape(-1, 2).astype(np.int32)
    return _tree(int(kind[4:]))


@pytest.mark.parametrize("kind,max_colors", [
    ("random1", 100), ("random2", 100), ("random511", 100), ("random2048", 100), ("random2049", 100),
    ("random50000", 100), ("hub35", 128), ("hub35", 33), ("hub35", 20), ("hubs", 128), ("hubs", 100), ("clique", 128),
    ("clique", 31), ("loops", 128), ("loops", 3), ("sheet", 100), ("sheet", 1), ("matching", 100), ("tree4", 100),
    ("tree13", 100), ("tree15", 100)])
def test_equals_sequential(pkg, po, kind, max_colors):
    rng = np.random.default_rng(sum(map(ord, kind)))
    nv, e = _graph(kind, rng)
    gc = pkg.GraphColoring(nv, e, max_num_colors=max_colors)
    color, order, prefix = po.color_edges(nv, e, max_colors) if max_colors != 100 else po.color_edges(nv, e)
    assert np.array_equal(gc.edges_color.cpu().numpy(), color)
    assert np.array_equal(gc.sorted_edges_sequence_for_color.cpu().numpy(), order)
    assert np.array_equal(gc.color_prefix_sum.cpu().numpy(), prefix)


def test_unaligned_workspace(pkg, po):
    """The workspace only has to be aligned for its status word."""
    from starlab_physics_gb300._lib import sx

    nv, e = _graph("hub35", np.random.default_rng(5))
    E = e.shape[0]
    nb = int(sx.sx_color_workspace_bytes(nv, E))
    buf = torch.zeros(nb + 64, dtype=torch.uint8, device="cuda")
    t = torch.from_numpy(e).cuda()
    out = torch.empty((2, E), dtype=torch.int32, device="cuda")
    prefix = torch.zeros(128, dtype=torch.int32, device="cuda")
    sx.sx_color_edges_greedy(t.data_ptr(), E, nv, 128, out[0].data_ptr(), out[1].data_ptr(), prefix.data_ptr(),
                             buf.data_ptr() + 4, nb, torch.cuda.current_stream().cuda_stream)
    color, order, _ = po.color_edges(nv, e, 128)
    assert np.array_equal(out[0].cpu().numpy(), color) and np.array_equal(out[1].cpu().numpy(), order)

"""The dense pair list equals a walk of the candidate lists in query order without
incident faces: lists shorter and longer than a round of lanes, truncated ones,
one query more or less than a block, more blocks than are added up directly."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_dy,n_st,cap", [(1, 0, 1), (5, 3, 40), (63, 1, 7), (64, 0, 33), (500, 28, 100), (2000, 77, 40),
                                           (262144, 5, 2), (270001, 3, 3)])
def test_list_in_query_order(pkg, n_dy, n_st, cap):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    rng = np.random.default_rng(n_dy + cap)
    F, Fs = max(2 * n_dy, 4), 50
    fd = rng.integers(0, n_dy, (F, 3)).astype(np.int32)
    fs = rng.integers(0, max(n_st, 1), (Fs, 3)).astype(np.int32)
    def lists(n, faces):
        c = rng.integers(0, faces, (max(n, 1), cap)).astype(np.int32)
        num = rng.integers(0, cap + 3, max(n, 1)).astype(np.int32)
        num[rng.random(max(n, 1)) < 0.3] = 0
        return c, num
    (sc, sn), (dc, dn), (tc, tn) = lists(n_dy, Fs), lists(n_dy, F), lists(n_st, F)
    # a third of the cloth's candidates are incident
    near = rng.random(dc.shape) < 0.3
    fd[dc[:, 0], rng.integers(0, 3)] = np.arange(n_dy)
    dc[near] = np.broadcast_to(dc[:, :1], dc.shape)[near]

    def walk(n, c, num, faces, own):
        q, j = np.nonzero(np.arange(cap)[None, :] < np.minimum(num[:n], cap)[:, None])
        t = faces[c[q, j]]
        out = np.concatenate([q[:, None].astype(np.int32), t], 1)
        return out[~(t == q[:, None]).any(1)] if own else out
    want = [walk(n_dy, sc, sn, fs, False), walk(n_dy, dc, dn, fd, True), walk(n_st, tc, tn, fd, False)]
    t = {k: torch.from_numpy(v).cuda() for k, v in dict(fd=fd, fs=fs, sc=sc, sn=sn, dc=dc, dn=dn, tc=tc, tn=tn).items()}
    P = lambda k: ptr(t[k])  # noqa: E731
    pairs = torch.full(((2 * n_dy + n_st) * cap, 4), -7, dtype=torch.int32, device="cuda")
    ws = torch.empty(int(sx.sx_contact_pairs_workspace_bytes(n_dy, n_st)), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        sx.sx_contact_pairs_build(n_dy, n_st, P("fd"), P("fs"), cap, P("sc"), P("sn"), P("dc"), P("dn"), P("tc"),
                                  P("tn"), ptr(pairs), pairs.shape[0], ptr(ws), ws.numel(), stream_handle())
    meta = ws[-256:].view(torch.int32)[:4].cpu().tolist()
    assert meta == [len(want[0]), len(want[0]) + len(want[1]), sum(map(len, want)), 0]
    got = pairs.cpu().numpy()
    assert np.array_equal(got[:meta[2]], np.concatenate(want))
    assert (got[meta[2]:] == -7).all()

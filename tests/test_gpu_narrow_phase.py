"""The pair list's straight-line narrow phase, its fallback and the fixed-point
conversions: random, degenerate, tiny, huge and coincident point-triangle pairs
of all three kinds, in every launch configuration, against the oracle's walk of
the same candidate lists, bit for bit (corrections, counts and status)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CAP = 8


def _soup(kind, rng, n):
    """n cloth triangles and n static ones with a query point near each."""
    tri = rng.normal(0, 1, (2 * n, 3, 3))
    scale = {"unit": 1e-2, "tiny": 1e-7, "denormal": 1e-11, "huge": 1e5, "far": 3e7}.get(kind, 1e-2)
    if kind == "sliver":
        tri[:, 2] = tri[:, 0] + (tri[:, 1] - tri[:, 0]) * rng.uniform(0, 1, (2 * n, 1)) + rng.normal(0, 1e-6, (2 * n, 3))
    elif kind == "coincident":
        tri[:, 1] = tri[:, 0]
        tri[1::3, 2] = tri[1::3, 0]
    elif kind == "flat":
        tri[:, :, 2] = 0.0
    tri *= scale
    bary = rng.dirichlet(np.ones(3) * 0.6, 2 * n) * rng.choice([1.0, 1.3], (2 * n, 1))
    p = np.einsum("nk,nkd->nd", bary, tri) + rng.normal(0, 0.2 * scale, (2 * n, 3))
    if kind == "flat":
        p[::2, 2] = 0.0
    if kind == "coincident":
        p[::5] = tri[::5, 0]
    return tri.astype(np.float32), p.astype(np.float32), scale


@pytest.mark.parametrize("kind", ["unit", "flat", "tiny", "denormal", "huge", "far", "sliver", "coincident"])
def test_pair_list_equals_walk(pkg, po, kind):
    from starlab_physics_gb300 import _lib

    rng = np.random.default_rng(sum(map(ord, kind)))
    n = 700
    tri, p, scale = _soup(kind, rng, n)
    # cloth: its n triangles, then its n points; obstacle the same
    def mesh(k):
        x = np.concatenate([tri[k * n:(k + 1) * n].reshape(-1, 3), p[k * n:(k + 1) * n]])
        f = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
        x4 = np.zeros((4 * n, 4), np.float32)
        x4[:, :3] = x
        return x4, f
    y4, fd = mesh(0)
    xs4, fs = mesh(1)
    V = 4 * n
    fixed = (rng.random(V) < 0.9).astype(np.float32)
    m_inv = rng.uniform(0.5, 80.0, V).astype(np.float32)
    y4[:, 3] = fixed * m_inv
    none = lambda q: (np.zeros((q, CAP), np.int32), np.zeros(q, np.int32))  # noqa: E731
    st_c, st_n = none(V)
    dy_c, dy_n = none(V)
    tv_c, tv_n = none(V)
    near = rng.integers(0, n, (n, 2))
    for c, num in ((st_c, st_n), (dy_c, dy_n), (tv_c, tv_n)):
        c[3 * n:, 0] = np.arange(n)
        c[3 * n:, 1:3] = near
        num[3 * n:] = rng.integers(0, 4, n)
    dy_c[:3 * n:7, 0] = np.arange(0, 3 * n, 7) // 3  # a face's own vertex: skipped
    dy_n[:3 * n:7] = 1
    # obstacle vertices near cloth triangles and the reverse
    xs4[3 * n:, :3] = y4[3 * n:, :3] + rng.normal(0, 0.1 * scale, (n, 3)).astype(np.float32)
    xs4[:3 * n, :3] = y4[:3 * n, :3] + rng.normal(0, 0.05 * scale, (3 * n, 3)).astype(np.float32)
    dHat = np.float32((0.5 * scale) ** 2)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    D = dict(fd=t(fd), fs=t(fs), xs=t(xs4), fx=t(fixed), mi=t(m_inv), sc=t(st_c), sn=t(st_n), dc=t(dy_c), dn=t(dy_n),
             tc=t(tv_c), tn=t(tv_n))
    s = torch.cuda.current_stream().cuda_stream
    P = lambda k: D[k].data_ptr()  # noqa: E731
    acc = torch.zeros(3 * V, dtype=torch.int64, device="cuda")
    nc = torch.zeros(V, dtype=torch.int32, device="cuda")

    Y = t(y4)
    st0 = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.sx.sx_collision_sweep(V, V, P("fd"), P("fs"), Y.data_ptr(), P("xs"), P("fx"), P("mi"), dHat, 1e8, CAP,
                               P("sc"), P("sn"), P("dc"), P("dn"), P("tc"), P("tn"), acc.data_ptr(), nc.data_ptr(),
                               None, None, None, None, st0.data_ptr(), s)
    want, want_status = Y.cpu().numpy(), int(st0.item())
    ref = y4.copy()
    with np.errstate(all="ignore"):
        po.collision_sweep(fd, fs, ref, xs4, fixed, m_inv, float(dHat), 1e8, CAP, (st_c, st_n), (dy_c, dy_n),
                           (tv_c, tv_n))
    assert np.array_equal(want[:, :3], ref[:, :3], equal_nan=True)
    if kind not in ("denormal", "coincident"):
        assert not np.array_equal(want[:, :3], y4[:, :3])  # something is in contact

    pairs = torch.zeros((3 * V * CAP, 4), dtype=torch.int32, device="cuda")
    ws = torch.zeros(int(_lib.load().sx_contact_pairs_workspace_bytes(V, V)), dtype=torch.uint8, device="cuda")
    _lib.sx.sx_contact_pairs_build(V, V, P("fd"), P("fs"), CAP, P("sc"), P("sn"), P("dc"), P("dn"), P("tc"), P("tn"),
                                   pairs.data_ptr(), pairs.shape[0], ws.data_ptr(), ws.numel(), s)
    for cull in (0.0, float(dHat) * 1.0625):
        for v in range(int(_lib.load().sx_contact_pairs_project_variants())):
            Y = t(y4)
            st = torch.zeros(1, dtype=torch.int32, device="cuda")
            _lib.sx.sx_contact_pairs_project_v(V, V, pairs.data_ptr(), ws.data_ptr(), Y.data_ptr(), P("xs"), P("fx"),
                                               P("mi"), dHat, 1e8, cull, acc.data_ptr(), nc.data_ptr(), st.data_ptr(),
                                               None, 0, v, s)
            _lib.sx.sx_contact_apply(V, Y.data_ptr(), P("fx"), acc.data_ptr(), nc.data_ptr(), None, 0, s)
            assert np.array_equal(Y.cpu().numpy(), want, equal_nan=True), (cull, v)
            if cull == 0.0:
                assert int(st.item()) == want_status
    assert int(acc.abs().max()) == 0 and int(nc.max()) == 0

"""The exact sweep's straight-line arithmetic and its fallback: inputs inside,
at the edge of and far outside the operand range the straight-line form covers
give the oracle's result bit for bit (NaN where the oracle has NaN), in every
kind of launch configuration."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases():
    out = []
    for scale in (1.0, 1e-6, 2e-7, 1e-13, 1e-30, 1e5, 1e6, 1e13, 1e25):
        out.append((scale, 277.0, 0.277, "plain"))
    for k in (0.0, 1e-7, 1e-5, 2e12, 1e30, -3.0):
        out.append((1.0, k, 0.5 * k, "plain"))
    out += [(1.0, 277.0, 0.277, "coincident"), (1.0, 277.0, 0.277, "rest"), (1.0, 277.0, 0.277, "nan"),
            (1.0, 277.0, 0.277, "heavy")]
    return out


@pytest.mark.parametrize("scale,ks,kb,kind", _cases())
def test_sweep_operand_range(pkg, po, scale, ks, kb, kind):
    from starlab_physics_gb300 import _lib

    rng = np.random.default_rng(11)
    sc = pkg.scenes.plain64(n=13, seed=4)
    m = pkg.TriMesh(sc.cloth_x, sc.cloth_faces, device="cuda")
    m.fixed[sc.pinned] = 0.0
    m.refresh_weights()
    V = m.num_verts
    x4 = m.x4.cpu().numpy().copy()
    y4 = x4.copy()
    y4[:, :3] += rng.normal(0, 2e-3, (V, 3)).astype(np.float32)
    y4[:, :3] *= np.float32(scale)
    x4[:, :3] *= np.float32(scale)
    adj = m.adj_np.copy()
    rest = adj[:, 1].view(np.float32).copy() * np.float32(scale)
    m_inv = m.m_inv_np.copy()
    if kind == "coincident":
        y4[40, :3] = y4[41, :3]
        y4[90, :3] = y4[91, :3] + np.float32(1e-7)
    elif kind == "rest":
        rest[::7] = 0.0
        rest[3::11] = np.float32(1e-42)
        rest[5::13] *= np.float32(-1.0)
    elif kind == "nan":
        y4[55, 1] = np.nan
        y4[100, 0] = np.inf
    elif kind == "heavy":
        m_inv[::9] *= np.float32(1e12)
        m_inv[4::9] *= np.float32(1e-30)
    adj[:, 1] = rest.view(np.int32)
    fixed = m.fixed.cpu().numpy()
    for a in (x4, y4):
        a[:, 3] = fixed * m_inv
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    from starlab_physics_gb300.mesh import packed_adjacency

    X, Y, A = t(x4), t(y4), t(adj)
    nbr, r32 = (t(p) for p in packed_adjacency(m.adj_ptr_np, adj))
    s = torch.cuda.current_stream().cuda_stream
    lib = _lib.load()
    negative_rest = bool((rest < 0).any())  # the packed form keeps the bending flag in the sign bit
    for bend_y in (0, 1):
        want = y4.copy()
        with np.errstate(all="ignore"):
            po.spring_sweep_gather(x4, want, fixed, m_inv, m.adj_ptr_np, adj, ks, kb, bend_on_y=bend_y)
        out = torch.empty_like(Y)
        for v in range(int(lib.sx_jacobi_sweep_variants())):
            out.fill_(7.0)
            _lib.sx.sx_jacobi_sweep_v(X.data_ptr(), Y.data_ptr(), out.data_ptr(), m.fixed.data_ptr(),
                                      m.adj_ptr.data_ptr(), A.data_ptr(), V, ks, kb, bend_y, v, s)
            assert np.array_equal(out.cpu().numpy()[:, :3], want[:, :3], equal_nan=True), (v, bend_y)
        for form in range(0 if negative_rest else int(lib.sx_jacobi_sweep_packed_forms())):
            out.fill_(7.0)
            _lib.sx.sx_jacobi_sweep_packed_v(X.data_ptr(), Y.data_ptr(), out.data_ptr(), m.fixed.data_ptr(),
                                             m.adj_ptr.data_ptr(), nbr.data_ptr(), r32.data_ptr(), V, ks, kb, bend_y,
                                             form, 0, s)
            assert np.array_equal(out.cpu().numpy()[:, :3], want[:, :3], equal_nan=True), (form, bend_y)


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [1, 30000, 30001, 49152, 49153, 200000, 200001, 1 << 30])
def test_default_variant_is_compiled(pkg, n, fast):
    from starlab_physics_gb300 import _lib

    lib = _lib.load()
    assert 0 <= int(lib.sx_jacobi_sweep_default_variant(n, fast)) < int(lib.sx_jacobi_sweep_variants())


@pytest.mark.parametrize("n", [1, 30000, 160000, 160001, 200001, 1 << 30])
def test_default_packed_form_is_compiled(pkg, n):
    from starlab_physics_gb300 import _lib

    lib = _lib.load()
    assert int(lib.sx_jacobi_sweep_default_packed_form(n, 0)) == -1
    assert -1 <= int(lib.sx_jacobi_sweep_default_packed_form(n, 1)) < int(lib.sx_jacobi_sweep_packed_forms())


def test_default_packed_form_equals_the_int2_sweep(pkg):
    """A sheet past the packed form's line, fast arithmetic: the default and the
    int2 variant of its size end in the same positions bit for bit."""
    out = []
    x, f = _grid(410, 395)
    for variant in (None, 5):
        m = pkg.TriMesh(x, f, device="cuda")
        sim = pkg.Solver(m, None, 4e-6, 1e5, 1e8, (0.0, 0.0, -9.81), 1 / 60, n_iter=3, bending_on="y")
        sim.fast_math, sim.sweep_variant = True, variant
        assert sim._default_packed == [-1, 3]
        m.v4[:, :3] = torch.from_numpy(np.random.default_rng(3).normal(0, 0.2, x.shape).astype(np.float32)).cuda()
        sim.forward(2)
        out.append(m.x4.cpu().numpy())
    assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1])
    # rest lengths edited in place: the packed copy is out of date and stays unused
    sim.sweep_variant = None
    assert sim._packed_choice(1) == 3
    m.adj[:, 1] += 0
    assert sim._packed_choice(1) == -1


def _grid(nx, ny):
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    x = np.stack([0.01 * i, 0.01 * j, 0.001 * np.sin(0.7 * i)], -1).reshape(-1, 3).astype(np.float32)
    a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1)
    f = np.stack([np.stack([a, a + ny, a + 1], -1), np.stack([a + 1, a + ny, a + ny + 1], -1)], 1).reshape(-1, 3)
    return x, f.astype(np.int32)

"""The headed projection against the plain one where its cull is not the heads':
none (every pair is evaluated), and a wider one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sheets(nx, ny, h, gap):
    X, F = [], []
    for k in range(2):
        i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
        X.append(np.stack([h * i, h * j, 0.004 * np.sin(1.3 * i) * np.cos(0.9 * j) + gap * k], -1).reshape(-1, 3))
        a = (i[:-1, :-1] * ny + j[:-1, :-1]).reshape(-1) + k * nx * ny
        F += [np.stack([a, a + ny, a + 1], -1), np.stack([a + 1, a + ny, a + ny + 1], -1)]
    return np.concatenate(X).astype(np.float32), np.concatenate(F).astype(np.int32)


@pytest.fixture(scope="module")
def scene(pkg):
    """A pair list with heads in use, after a few tracked iterations."""
    h = 0.03
    x, f = _sheets(37, 29, h, 6e-3)
    m = pkg.TriMesh(x, f, device="cuda")
    s = pkg.TriMesh(*pkg.box_mesh(0.4, center=(h * 18, h * 14, -0.206)), device="cuda", is_static=True)
    sim = pkg.Solver(m, s, dHat=(4e-3) ** 2, stiffness_stretch=1e5, stiffness_bending=1e8, g=(0, 0, -9.81), dt=1 / 60,
                     n_iter=8, rebuild="substep", bending_on="y")
    sim.enable_collision_handling = True
    sim.HEADS_MIN_PAIRS, sim.HEADS_MIN_ITERATIONS, sim._in_substep = 1, 2, True
    sim.build_bvhs()
    sim.compute_y(1 / 600)
    for it in range(4):
        sim.solve_constraints_jacobi_x(1 / 600, it == 0, it)
    torch.cuda.synchronize()
    assert sim._heads_on and int(sim._pairs_ws[-256:].view(torch.int32)[3].item()) == 1
    return sim


def _sums(sim, dHat, cull_d2, variant, headed):
    from starlab_physics_gb300._lib import stream_handle, sx

    m, s = sim.mesh_dy, sim.mesh_st
    dx, nc = torch.zeros_like(sim._dx_fix), torch.zeros_like(sim._nc)
    common = (m.num_verts, s.num_verts, sim._pairs.data_ptr(), sim._pairs_ws.data_ptr(), m.y4.data_ptr(),
              s.x4.data_ptr(), m.fixed.data_ptr(), m.m_inv.data_ptr(), dHat, sim.compliance_collision, cull_d2,
              dx.data_ptr(), nc.data_ptr(), sim.status.data_ptr(), None, 0, variant)
    if headed:
        sx.sx_contact_pairs_project_headed(*common, sim._heads[0].data_ptr(), sim._heads[2].data_ptr(),
                                           stream_handle())
    else:
        sx.sx_contact_pairs_project_v(*common, stream_handle())
    torch.cuda.synchronize()
    return dx.cpu().numpy(), nc.cpu().numpy()


@pytest.mark.parametrize("variant", range(7))
@pytest.mark.parametrize("wider,cull", [(1.0, True), (36.0, False), (36.0, True), (1.0, False)])
def test_equals_the_plain_projection(scene, variant, wider, cull):
    dHat = scene.dHat * wider
    cull_d2 = dHat * scene.CULL_MARGIN if cull else 0.0
    dx1, nc1 = _sums(scene, dHat, cull_d2, variant, True)
    dx0, nc0 = _sums(scene, dHat, cull_d2, variant, False)
    assert np.array_equal(nc1, nc0) and np.array_equal(dx1, dx0)
    assert wider == 1.0 or nc0.any()

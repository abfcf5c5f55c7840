"""The persistent substep's projection on obstacle triangles that leave the straight-
line arithmetic's range (no area, tiny, a needle) and on ordinary ones, against the
grid-wide launches bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _instances(pkg):
    out = []
    for k, n in enumerate((9, 23, 40)):
        x, f = pkg.grid_cloth(n)[:2]
        x = np.asarray(x, np.float32).copy()
        x[:, 2] = 0.003 + 0.001 * np.sin(9 * x[:, 0])
        ox, of = pkg.box_mesh(0.5, center=(0.5, 0.5, -0.25))
        ox, of = np.asarray(ox, np.float32), np.asarray(of, np.int32)
        m = len(ox)
        extra = np.array([[0.5, 0.5, 0.002], [0.5, 0.5, 0.002], [0.6, 0.5, 0.002],          # no area
                          [0.3, 0.3, 0.003], [0.3 + 1e-7, 0.3, 0.003], [0.3, 0.3 + 1e-7, 0.003],  # tiny
                          [0.2, 0.7, 0.002], [0.8, 0.7, 0.002], [0.5, 0.7 + 1e-6, 0.002]], np.float32)  # needle
        tri = np.arange(9, dtype=np.int32).reshape(3, 3) + m
        out.append(pkg.Instance(x, f, np.array([0, n - 1]), np.concatenate([ox, extra[:3 * k]]),
                                np.concatenate([of, tri[:k]]).astype(np.int32)))
    return out


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("variant", [0, 2, 6, 10])
def test_equals_grid_launches(pkg, fast, variant):
    out = []
    for persistent in (True, False):
        b = pkg.BatchedSolver(_instances(pkg), 1.6e-5, 1e5, 1e8, (0.0, 0.0, -9.81), 1 / 60, n_iter=6)
        b.fast_math, b.persistent, b.persistent_variant = fast, persistent, variant
        b.v4[:, 2] = -0.4
        for _ in range(2):
            b.forward(4)
        torch.cuda.synchronize()
        out.append((b.x4.cpu().numpy(), b.v4.cpu().numpy()))
    assert np.isfinite(out[0][0]).all()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

"""SiLU and its derivative, as the mma inference and the training step evaluate
them, over the whole range of float32 pre-activations."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, 1e-38, -1e-38, 1e-30, 3e-8, -3e-8, 0.7, -0.7, 4.0, -4.0, 16.0, -16.6, 17.4, 60.0, -60.0, -69.0,
          -69.5, -75.0, -86.9, -87.1, -88.5, -89.0, -104.0, 1e4, -1e4, 1e25, -1e25, 1e30, -1e30, 1e35, -1e35, 3e38,
          -3e38, np.inf]


def _net(pkg, v):
    """Second-layer pre-activations of v in every unit, summed by output 0."""
    p = {"W1": np.zeros((64, 32)), "b1": np.zeros(64), "W2": np.zeros((64, 64)), "b2": np.full(64, v),
         "W3": np.zeros((8, 64)), "b3": np.zeros(8)}
    p["W3"][0] = 1.0
    return pkg.WarmStartMLP(params=np.concatenate([p[k].astype(np.float32).ravel() for k, _ in pkg.learned.SHAPES]),
                            tcgen05=False)


def _silu(v):
    with np.errstate(over="ignore"):
        return float(v) if np.isposinf(v) else float(v) / (1.0 + np.exp(-np.float64(v)))


@pytest.mark.parametrize("v", VALUES)
def test_silu(pkg, v):
    feat = torch.zeros((3, 32), dtype=torch.bfloat16, device="cuda")
    out = _net(pkg, v).forward(feat, torch.zeros((3, 4), device="cuda")).cpu().numpy().astype(np.float64)
    exact = 64.0 * _silu(np.float32(v))
    assert (out[:, 0] == out[0, 0]).all()
    if np.isinf(exact):
        assert out[0, 0] == exact
    elif abs(exact) < 3.38e38:
        # BF16 of the exact value, give or take the few last places of float32 before the rounding
        near = torch.tensor([exact / 64 * (1 + k * 2.0 ** -21) + k * 2e-36 for k in (-1, 1)], dtype=torch.float64)
        lo, hi = np.sort(64 * near.to(torch.bfloat16).to(torch.float64).numpy())
        assert lo <= out[0, 0] <= hi


@pytest.mark.parametrize("v", [v for v in VALUES if v < 1e4])
def test_derivative(pkg, v):
    """Bias gradient of the second layer for an output gradient of 2."""
    net = _net(pkg, v)
    feat = torch.zeros((1, 32), dtype=torch.bfloat16, device="cuda")
    o = net.forward(feat, torch.zeros((1, 4), device="cuda"))[0, 0].item()
    target = torch.tensor([[o - 1.0, 0.0, 0.0, 1.0]], device="cuda")
    diff = np.float32(o) - np.float32(target[0, 0].item())
    grad, _ = net.gradients(feat, target, torch.zeros(1, dtype=torch.int32, device="cuda"), 1)
    db2 = grad.cpu().numpy()[64 * 32 + 64 + 64 * 64:][:64].astype(np.float64)
    z = np.float64(np.float32(v))
    with np.errstate(over="ignore"):
        s = 1.0 / (1.0 + np.exp(-z))
    exact = s + z * s * (1.0 - s)
    d_out = float(torch.tensor(2.0 * diff).to(torch.bfloat16))
    # 1 - s loses up to 2^-24 absolutely, times z s; the other roundings are relative
    assert np.abs(db2 - d_out * exact).max() <= abs(d_out) * (2.0 ** -20 * (s + abs(z) * s) + 2e-36)

"""The MLP kernels at the edges of their tiles (16, 64 and 128 rows), of the
training grid, and with weights that are only aligned to a value: gradients
against the oracle's, inference and gradients bit for bit against the aligned
call and, row by row, against a batch of another size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(rng, n):
    feat = torch.zeros((n, 32), dtype=torch.bfloat16, device="cuda")
    x = rng.normal(0, 0.4, (n, 24)).astype(np.float32)
    x[:, 16] = rng.random(n) < 0.9
    feat[:, :24] = torch.from_numpy(x).cuda().to(torch.bfloat16)
    t = rng.normal(0, 0.2, (n, 4)).astype(np.float32)
    t[:, 3] = 1.0
    u16 = feat.view(torch.int16).cpu().numpy().view(np.uint16)
    return u16, t, feat, torch.from_numpy(t).cuda()


@pytest.mark.parametrize("n", [1, 15, 17, 63, 64, 65, 127, 129, 64 * 304, 64 * 304 + 1, 64 * 305 - 1])
def test_gradients_at_tile_edges(pkg, po, n):
    rng = np.random.default_rng(n)
    u16, t, feat, tt = _batch(rng, n)
    p = pkg.learned.init_params(3)
    p[-8:-5] = 0.1
    net = pkg.WarmStartMLP(params=p)
    perm = rng.permutation(n).astype(np.int32)
    grad, st = net.gradients(feat, tt, torch.from_numpy(perm).cuda(), n)
    ref, loss, _ = po.mlp_gradients(u16[perm], t[perm], p)
    # one BF16 rounding (2^-9) per operand of the products and of the activations
    assert np.linalg.norm(grad.cpu().numpy() - ref) <= 2e-2 * np.linalg.norm(ref)
    assert abs(float(st[0].item()) - loss) <= 2e-3 * loss


@pytest.mark.parametrize("n", [1, 127, 128, 129, 128 * 760 + 1])
def test_unaligned_weights_and_row_independence(pkg, n):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    rng = np.random.default_rng(n)
    _, t, feat, tt = _batch(rng, n)
    net = pkg.WarmStartMLP(params=pkg.learned.init_params(5))
    shifted = torch.zeros(net.w16.numel() + 1, dtype=torch.bfloat16, device="cuda")
    shifted[1:] = net.w16
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = []
    for w in (ptr(net.w16), ptr(shifted) + 2):
        a = torch.full((n, 4), float("nan"), device="cuda")
        b = torch.full((n, 4), float("nan"), device="cuda")
        sx.sx_mlp_forward_tc(ptr(feat), n, w, ptr(net.p32), ptr(a), ptr(st), stream_handle())
        sx.sx_mlp_forward(ptr(feat), n, w, ptr(net.p32), ptr(b), stream_handle())
        ws = torch.zeros(int(sx.sx_mlp_train_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
        g = torch.full_like(net.p32, float("nan"))
        s4 = torch.zeros(4, device="cuda")
        idx = torch.arange(n, dtype=torch.int32, device="cuda")
        sx.sx_mlp_gradients(ptr(feat), ptr(tt), ptr(idx), n, n, w, ptr(net.p32), ptr(g), ptr(s4), ptr(ws), ws.numel(),
                            stream_handle())
        outs.append([x.cpu().numpy() for x in (a, b, g, s4)])
    assert int(st.item()) == 0
    for x, y in zip(*outs):
        assert np.isfinite(x).all() and np.array_equal(x, y)
    k = max(n // 2, 1)
    part = torch.full((k, 4), float("nan"), device="cuda")
    net.forward(feat[n - k:].contiguous(), part)
    assert np.array_equal(part.cpu().numpy(), outs[0][0][n - k:])

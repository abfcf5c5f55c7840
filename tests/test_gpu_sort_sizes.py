"""Pair sorts on both sides of the one-launch limit and of its tiles, in every
digit count: stable, equal to numpy's, in a graph and out of one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 1023, 1024, 1025, 2049, 8193, 16384, 16385, 20011, 32769, 65535, 65536, 65537, 100003, 131073, 200000]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("first,bits", [(0, 32), (0, 15), (0, 8), (3, 17), (24, 8), (0, 1), (16, 16)])
def test_sorted_stable(pkg, n, first, bits):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    rng = np.random.default_rng(n + bits)
    cases = [rng.integers(0, 1 << 32, n, dtype=np.uint64), np.full(n, 0x9e3779b9, np.uint64),
             rng.integers(0, 5, n, dtype=np.uint64) << first, np.arange(n, 0, -1).astype(np.uint64)]
    ws = torch.empty(int(sx.sx_radix_sort_workspace_bytes(n)), dtype=torch.uint8, device="cuda")
    for keys in cases:
        keys = (keys & 0xffffffff).astype(np.uint32)
        K = torch.from_numpy(keys.view(np.int32).copy()).cuda()
        V = torch.arange(n, dtype=torch.int32, device="cuda")
        sx.sx_radix_sort_pairs_bits(ptr(K), ptr(V), n, first, bits, ptr(ws), ws.numel(), stream_handle())
        order = np.argsort((keys >> np.uint32(first)) & np.uint32((1 << bits) - 1), kind="stable")
        assert np.array_equal(V.cpu().numpy(), order)
        assert np.array_equal(K.cpu().numpy().view(np.uint32), keys[order])


def test_in_a_graph_and_on_two_streams(pkg):
    from starlab_physics_gb300._lib import ptr, stream_handle, sx

    n = 30011
    rng = np.random.default_rng(7)
    src = [torch.from_numpy(rng.integers(-2**31, 2**31, n, dtype=np.int64).astype(np.int32)).cuda() for _ in range(2)]
    K, V = [torch.empty_like(s) for s in src], [torch.empty_like(s) for s in src]
    iota = torch.arange(n, dtype=torch.int32, device="cuda")
    ws = [torch.empty(int(sx.sx_radix_sort_workspace_bytes(n)), dtype=torch.uint8, device="cuda") for _ in range(2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def sort(k):
        K[k].copy_(src[k])
        V[k].copy_(iota)
        sx.sx_radix_sort_pairs(ptr(K[k]), ptr(V[k]), n, 32, ptr(ws[k]), ws[k].numel(), stream_handle())

    def check(k):
        keys = src[k].cpu().numpy().view(np.uint32)
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(V[k].cpu().numpy(), order) and np.array_equal(K[k].cpu().numpy().view(np.uint32),
                                                                            keys[order])
    torch.cuda.synchronize()
    for _ in range(20):
        for k in range(2):
            with torch.cuda.stream(streams[k]):
                sort(k)
    torch.cuda.synchronize()
    check(0), check(1)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sort(0)
    V[0].zero_()
    g.replay()
    torch.cuda.synchronize()
    check(0)

"""Two expert blocks, and two split-K products, with different inputs over one workspace, queued without a synchronisation between them:
each gives what it gives alone.  All their launches may start before the one before has ended, and each has to wait for it."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


def _dev(cuda, *arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in arrays]


# few experts, one item each; items that fill the SMs, launched dependent; the decode path
@pytest.mark.parametrize("S,topk,E,H,MI", [(45, 4, 8, 512, 256), (80, 4, 64, 1024, 512), (6, 4, 16, 512, 768)])
def test_two_expert_blocks(w4a8, oracle, cuda, S, topk, E, H, MI):
    import torch
    gu, gs, dn, ds = _dev(cuda, *oracle.make_weights(E * 2 * MI, H, seed=1), *oracle.make_weights(E * H, MI, seed=2))
    gs *= 8.0
    g = torch.Generator(device=cuda).manual_seed(S)
    rows = [S, S - 3]                                                                # the second one's sort is another one
    x = [torch.randn((n, H), generator=g, device=cuda) * (i + 1) for i, n in enumerate(rows)]
    idx = [torch.stack([torch.randperm(E, generator=g, device=cuda)[:topk] for _ in range(n)]).to(torch.int32).reshape(-1).contiguous() for n in rows]
    dw = [torch.rand(n * topk, generator=g, device=cuda) for n in rows]
    nbytes = w4a8.moe_layout_for(S, topk, H, MI, E).bytes

    def block(i, out, ws):
        w4a8.moe_block(x[i], gu, gs, dn, ds, idx[i], dw[i], out, rows[i], topk, H, MI, E, ws)

    alone = []
    for i in range(2):
        alone.append(torch.empty((rows[i], H), device=cuda))
        block(i, alone[i], torch.full((nbytes,), 0x7F, dtype=torch.uint8, device=cuda))
        torch.cuda.synchronize()
    ws = torch.full((nbytes,), 0x7F, dtype=torch.uint8, device=cuda)
    busy = torch.zeros(32 << 20, device=cuda)
    for rep in range(4):
        outs = [torch.full((n, H), float("nan"), device=cuda) for n in rows]
        busy.add_(1.0)                                                               # all launches are queued before the first one runs
        for i in ((0, 1), (1, 0))[rep % 2]:
            block(i, outs[i], ws)
        torch.cuda.synchronize()
        for o, a in zip(outs, alone):
            assert torch.equal(o.view(torch.int32), a.view(torch.int32)) and bool(torch.isfinite(o).all())
    w4a8.device_status()


@pytest.mark.parametrize("M,N,K,splitk", [(40, 300, 2048, 4), (17, 1023, 1536, 3), (130, 2000, 1024, 2), (148, 1024, 512, 2), (148, 1025, 512, 2), (149, 1024, 512, 2)])
def test_two_split_k_products(w4a8, oracle, cuda, M, N, K, splitk):
    import torch
    ops = []
    for i in range(2):
        xq, xs, _ = oracle.quantize_x_q8(oracle.make_activations(M, K, seed=10 + i, outliers=True))
        ops.append(_dev(cuda, xq, xs, *oracle.make_weights(N, K, seed=20 + i)))
    nbytes = w4a8.gemm_splitk_workspace_bytes(M, N, K, splitk)
    assert nbytes > 0

    def product(i, Y, ws, stream=None):
        w4a8.launch_gemm_bm16_splitk(*ops[i], Y, M, N, K, splitk=splitk, workspace=ws, stream=stream)

    alone = []
    for i in range(2):
        alone.append(torch.empty((M, N), device=cuda))
        product(i, alone[i], torch.full((nbytes // 4,), float("nan"), device=cuda))
        torch.cuda.synchronize()
    ws = torch.full((nbytes // 4,), float("nan"), device=cuda)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:                # four columns a thread from 1024 outputs an SM on
        four = M * N > 1024 * 148
        names = launched_kernels(lambda stream: product(0, alone[0], ws, stream))
        assert ("splitk_reduce_kernelI6float4E" if four else "splitk_reduce_kernelIfE") in names[-1], names
    busy = torch.zeros(32 << 20, device=cuda)
    for rep in range(4):
        Ys = [torch.full((M, N), float("nan"), device=cuda) for _ in range(2)]
        busy.add_(1.0)
        for i in ((0, 1), (1, 0))[rep % 2]:
            product(i, Ys[i], ws)
        torch.cuda.synchronize()
        for y, a in zip(Ys, alone):
            assert torch.equal(y.view(torch.int32), a.view(torch.int32)) and bool(torch.isfinite(y).all())
    w4a8.device_status()

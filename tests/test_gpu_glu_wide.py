"""Activation + quantizer with eight elements a thread (32-byte aligned inputs, at least a CTA per SM) against the kernel for inputs
that are aligned to 16 bytes only, and the expert block with tokens of either alignment: the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("S,IN", [(64, 5120), (301, 1056), (1000, 768)])
def test_activation_equals_the_narrow_kernel(w4a8, cuda, S, IN, act):
    import torch
    g = torch.Generator(device=cuda).manual_seed(S + IN + act)
    data = [torch.randn(S * IN, generator=g, device=cuda) * 4 for _ in range(2)]
    data[0][:64] = 0.0
    data[0][100::997], data[1][500::1999] = float("nan"), float("inf")
    res = []
    for shift in (0, 4):
        G, U = (torch.zeros(S * IN + 8, device=cuda) for _ in range(2))
        G[shift:shift + S * IN], U[shift:shift + S * IN] = data
        Y = torch.full((S + 1, IN), 7.0, device=cuda)
        xq = torch.full((S + 1, IN), 77, dtype=torch.int8, device=cuda)
        xs = torch.full((S + 1, IN // 32), 7.0, device=cuda)
        xsum = torch.full((S + 1, IN // 32), 7, dtype=torch.int32, device=cuda)
        w4a8.launch_glu_quantize_x_q8(G[shift:], U[shift:], act, Y, xq, xs, xsum, IN, S)
        assert bool((Y[S] == 7.0).all() and (xq[S] == 77).all() and (xs[S] == 7.0).all() and (xsum[S] == 7).all())
        res.append([t[:S].cpu().numpy() for t in (Y, xq, xs, xsum)])
    for a, b in zip(*res):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("S,topk,E", [(40, 4, 16), (33, 9, 20)])
def test_expert_block_with_tokens_of_either_alignment(w4a8, oracle, cuda, S, topk, E):
    import torch
    H, MI = 512, 256
    g = torch.Generator(device=cuda).manual_seed(S)
    x = torch.randn(S * H, generator=g, device=cuda)
    gu, dn = (torch.from_numpy(a).to(cuda) for a in (oracle.make_weights(E * 2 * MI, H, seed=1)[0], oracle.make_weights(E * H, MI, seed=2)[0]))
    gs, ds = (torch.from_numpy(a).to(cuda) for a in (oracle.make_weights(E * 2 * MI, H, seed=1)[1], oracle.make_weights(E * H, MI, seed=2)[1]))
    idx = torch.stack([torch.randperm(E, generator=g, device=cuda)[:topk] for _ in range(S)]).to(torch.int32).reshape(-1).contiguous()
    dw = torch.rand(S * topk, generator=g, device=cuda)
    ws = torch.empty(w4a8.moe_layout_for(S, topk, H, MI, E).bytes, dtype=torch.uint8, device=cuda)
    outs = []
    for shift in (0, 4):
        n2 = torch.zeros(S * H + 8, device=cuda)
        n2[shift:shift + S * H] = x
        out = torch.full((S, H), float("nan"), device=cuda)
        w4a8.moe_block(n2[shift:], gu, gs, dn, ds, idx, dw, out, S, topk, H, MI, E, ws)
        w4a8.device_status()
        outs.append(out.cpu().numpy().view(np.uint32))
    assert np.array_equal(*outs) and not np.isnan(outs[0].view(np.float32)).any()

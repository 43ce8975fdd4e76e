"""Activation + quantizer with eight elements a thread (32-byte aligned inputs, CTAs that divide well over 148 SMs) against the kernel with
four, which serves inputs aligned to 16 bytes only: the same bits; and the expert block with tokens of either alignment."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


# CTAs of the wide kernel / takes it with SwiGLU / with GeGLU: the lines of the rule, whole and part-filled last CTAs
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("S,IN,wide", [(64, 5120, (0, 0)), (301, 1056, (0, 0)), (1000, 768, (0, 1)), (222, 2048, (0, 0)), (223, 2048, (1, 1)),
                                       (296, 2048, (1, 1)), (297, 2048, (0, 1)), (518, 2048, (0, 1)), (519, 2048, (1, 1)), (593, 2048, (0, 0)), (740, 2048, (0, 0)), (741, 2048, (0, 1)), (888, 2048, (1, 1)),
                                       (1723, 1056, (1, 1)), (3001, 1056, (1, 1))])
def test_activation_equals_the_narrow_kernel(w4a8, cuda, S, IN, wide, act):
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

        def call(stream):
            w4a8.launch_glu_quantize_x_q8(G[shift:], U[shift:], act, Y, xq, xs, xsum, IN, S, stream)

        call(None)
        torch.cuda.synchronize()
        if torch.cuda.get_device_properties(0).multi_processor_count == 148:
            assert ["glu_quantize_wide_kernel" in n for n in launched_kernels(call)] == [shift == 0 and bool(wide[act])]
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

        def call(stream):
            w4a8.moe_block(n2[shift:], gu, gs, dn, ds, idx, dw, out, S, topk, H, MI, E, ws, stream=stream)

        call(None)
        w4a8.device_status()
        names = launched_kernels(call)
        assert "moe_sort" in "".join(names) and any("quantize_x_q8" in n for n in names) == (shift != 0), names   # the sort quantizes, or a launch of its own
        outs.append(out.cpu().numpy().view(np.uint32))
    assert np.array_equal(*outs) and not np.isnan(outs[0].view(np.float32)).any()

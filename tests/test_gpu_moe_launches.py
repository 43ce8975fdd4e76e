"""How an expert block's grouped products are launched: dependent on the kernel before them where their items fill the SMs (more than two
units an SM on 148 SMs), after it where they do not."""
import pytest

pytestmark = pytest.mark.gpu


def dependent_launches(call):
    """(mangled name, whether it was launched dependent on the one before) of the kernels that call(stream) launches; captured, not run."""
    import torch
    from cuda.bindings import driver as D

    def ok(r):
        assert r[0] == D.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    stream = torch.cuda.Stream()
    ok(D.cuStreamBeginCapture(stream.cuda_stream, D.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL))
    try:
        call(stream.cuda_stream)
    finally:
        graph = ok(D.cuStreamEndCapture(stream.cuda_stream))
    edges = ok(D.cuGraphGetEdges_v2(graph, ok(D.cuGraphGetEdges_v2(graph))[-1]))
    programmatic = {int(to) for to, data in zip(edges[1], edges[2]) if data.type == D.CUgraphDependencyType.CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC.value}
    found = []
    for node in ok(D.cuGraphGetNodes(graph, ok(D.cuGraphGetNodes(graph))[1]))[0]:
        p = ok(D.cuGraphKernelNodeGetParams(node))
        found.append((ok(D.cuFuncGetName(p.func) if int(p.func) else D.cuKernelGetName(p.kern)).decode(), int(node) in programmatic))
    ok(D.cuGraphDestroy(graph))
    return found


@pytest.mark.parametrize("S,topk,E,H,MI,dependent", [
    (94, 8, 16, 1024, 512, [False, False]),          # 16 items x 8 columns of tiles, twice
    (362, 4, 32, 512, 1024, [True, False]),          # 32 x 16, 32 x 4
    (300, 8, 16, 1024, 512, [True, True]),           # three items an expert
    (400, 2, 64, 1024, 512, [True, True])])
def test_grouped_products(w4a8, cuda, S, topk, E, H, MI, dependent):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are those of 148 SMs")
    z = lambda *shape, dtype=torch.float32: torch.zeros(shape, dtype=dtype, device=cuda)
    gu, dn = z(E * 2 * MI, H // 2, dtype=torch.uint8), z(E * H, MI // 2, dtype=torch.uint8)
    args = (z(S, H), gu, z(E * 2 * MI, H // 32), dn, z(E * H, MI // 32), z(S * topk, dtype=torch.int32), z(S * topk), z(S, H), S, topk, H, MI, E,
            z(w4a8.moe_layout_for(S, topk, H, MI, E).bytes, dtype=torch.uint8))
    w4a8.moe_block(*args)                            # configures the kernels, which a capture does not allow
    w4a8.device_status()
    found = dependent_launches(lambda stream: w4a8.moe_block(*args, stream=stream))
    assert [d for n, d in found if "gemm_w4a8_mma_kernel" in n] == dependent, found

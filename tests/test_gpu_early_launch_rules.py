"""Which launches are put on the GPU early, and how many there are: read off captured graphs, whose edges say so."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


class _Edge(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def _captured(body):
    """Kernel nodes of the captured body, and how many of them may start before the one in front of them is complete."""
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        body()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        body()
    g, n, m, kind = C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(), C.c_size_t(), C.c_int()
    ok(cu.cuGraphGetNodes(g, None, C.byref(n)))
    nodes = (C.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(g, nodes, C.byref(n)))
    kernels = 0
    for x in nodes:
        ok(cu.cuGraphNodeGetType(C.c_void_p(x), C.byref(kind)))
        kernels += kind.value == 0                             # CU_GRAPH_NODE_TYPE_KERNEL
    ok(cu.cuGraphGetEdges_v2(g, None, None, None, C.byref(m)))
    a, b, data = (C.c_void_p * m.value)(), (C.c_void_p * m.value)(), (_Edge * m.value)()
    ok(cu.cuGraphGetEdges_v2(g, a, b, data, C.byref(m)))
    early = sum(d.type == 1 for d in data)                     # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    return kernels, early


@pytest.mark.parametrize("B,nh,T,early", [(1, 32, 4096, 2), (1, 32, 1024, 2), (1, 16, 1024, 4), (16, 32, 512, 4)])
def test_mat_vec(cuda, B, nh, T, early):
    """q . K^T and p . V twice, behind a kernel: clusters of 64 CTAs and more are launched in the ordinary way."""
    from kvmix_b200 import ops
    k = torch.randn((B, nh, T, 128), device=cuda, dtype=torch.float16)
    keys, values = ops.quantize_pack_last_dim_cuda(k.transpose(2, 3), 32, 2), ops.quantize_pack_last_dim_cuda(k, 32, 2)
    q, p, x = k[:, :, :1].contiguous(), torch.rand((B, nh, 1, T), device=cuda).half(), torch.zeros(4, device=cuda)

    def body():
        x.add_(1)
        for _ in range(2):
            ops.quantized_gemm(32, q, *keys, 2)
            ops.quantized_gemm(32, p, *values, 2)
    assert _captured(body) == (5, early)


@pytest.mark.parametrize("nh,hkv,T,early", [(128, 128, 700, 3), (144, 144, 700, 1), (148, 148, 700, 1), (149, 149, 700, 3), (592, 148, 700, 1), (32, 32, 700, 3)])
def test_whole_heads_for_all_sms(cuda, nh, hkv, T, early):
    """Whole heads for nearly all SMs are launched in the ordinary way; fewer, more, and cut ones early.  Attention
    twice, with a mat-vec between them, which is early here."""
    import kvmix_b200 as kv
    from kvmix_b200 import ops
    c = kv.KVmixLayerCache(1, hkv, 128, T + 64, 2, 2, 64, residual_length=128, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(1)
    c.prefill(*(torch.randn((1, hkv, T, 128), generator=g, device=cuda, dtype=torch.float16) for _ in range(2)))
    keys = ops.quantize_pack_last_dim_cuda(torch.randn((1, 8, 640, 128), device=cuda, dtype=torch.float16).transpose(2, 3), 32, 2)
    q, x = torch.randn((1, nh, 1, 128), generator=g, device=cuda, dtype=torch.float16), torch.zeros(4, device=cuda)
    out = torch.empty_like(q)

    def body():
        x.add_(1)
        c.attend(q, out=out)
        ops.quantized_gemm(32, q[:, :8], *keys, 2)
        c.attend(q, out=out)
    assert _captured(body) == (4, early)


@pytest.mark.parametrize("kb,vb,G,L,rotate,want", [(2, 2, 32, 600, True, 1), (4, 1, 64, 600, True, 1), (3, 3, 64, 600, True, 1), (1, 4, 128, 600, True, 1),
                                                   (2, 2, 32, 600, False, 3), (4, 4, 32, 128, True, 1), (3, 2, 32, 140, True, 2)])
def test_prefill_launches(cuda, kb, vb, G, L, rotate, want):
    """A prompt is one launch where it is rotated on the way and both packed parts have tokens, three where its keys arrive rotated,
    one less for each part without tokens.  What LAUNCHES counts is what was launched."""
    import kvmix_b200 as kv
    from kvmix_b200 import ops
    caches = [kv.KVmixLayerCache(2, 3, 128, L + 8, kb, vb, G, residual_length=128, device=cuda) for _ in range(2)]
    kp, vp = (torch.randn((2, L, 3 * 128), device=cuda, dtype=torch.float16) for _ in range(2))
    tables = [torch.rand((L, 128), device=cuda).half() for _ in range(2)] if rotate else []
    counted, x = [], torch.zeros(4, device=cuda)

    def body():
        x.add_(1)                                              # a graph of one kernel has no edges to look at
        n = ops.LAUNCHES[0]
        caches[len(counted)].prefill_projected(kp, vp, *tables)
        counted.append(ops.LAUNCHES[0] - n)
    kernels, _ = _captured(body)
    assert (kernels, counted) == (want + 1, [want, want])

"""Kernels that are launched while the one before them still runs its last CTAs: a chain in which every launch reads what the one before
wrote, and the forms of capture in which the launch before is a copy, a fill or another stream's work."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 8, 700, 2), (2, 8, 2, 3000, 4), (9, 32, 32, 600, 2)]


def _cache(cuda, B, hkv, T, bits, seed):
    import kvmix_b200 as kv
    g = torch.Generator(device=cuda).manual_seed(seed)
    c = kv.KVmixLayerCache(B, hkv, 128, T + 64, bits, bits, 64, residual_length=128, device=cuda)
    c.prefill(*(torch.randn((B, hkv, T, 128), generator=g, device=cuda, dtype=torch.float16) for _ in range(2)))
    return c


@pytest.mark.parametrize("B,nh,hkv,T,bits", SHAPES)
@pytest.mark.parametrize("fused", [False, True])
def test_chain(cuda, B, nh, hkv, T, bits, fused):
    """out of one launch is q (and the new key and value) of the next: as with a synchronisation behind every launch."""
    def run(sync):
        caches = [_cache(cuda, B, hkv, T, bits, 3 + i) for i in range(2)]
        x = torch.randn((B, nh, 1, 128), generator=torch.Generator(device=cuda).manual_seed(1), device=cuda, dtype=torch.float16)
        outs = []
        torch.cuda.synchronize()
        for i in range(40):
            c = caches[i % 2]
            if fused:
                n = x[:, :hkv].contiguous() if hkv != nh else x
                x = c.decode_step(x, n, n)
            else:
                x = c.attend(x)
            if sync:
                torch.cuda.synchronize()
            outs.append(x)
        torch.cuda.synchronize()
        return torch.stack(outs)
    assert torch.equal(run(True).view(torch.int16), run(False).view(torch.int16))


@pytest.mark.parametrize("bits", [2, 4])
def test_gemv_and_prefill_chain(cuda, bits):
    from kvmix_b200 import ops
    import kvmix_b200 as kv
    k = torch.randn((2, 8, 1024, 128), generator=torch.Generator(device=cuda).manual_seed(2), device=cuda, dtype=torch.float16)
    angle = torch.arange(1024, device=cuda).float()[:, None] / 10000.0 ** (torch.arange(0, 128, 2, device=cuda).float() / 128)
    cos, sin = (f(torch.cat((angle, angle), 1)).half() for f in (torch.cos, torch.sin))
    keys, values = ops.quantize_pack_last_dim_cuda(k.transpose(2, 3), 32, bits), ops.quantize_pack_last_dim_cuda(k, 32, bits)

    def run(sync):
        c = kv.KVmixLayerCache(2, 8, 128, 1100, bits, bits, 32, residual_length=128, device=cuda)
        for t in (c.kcode, c.kscale, c.kmn, c.vcode, c.vscale, c.vmn, c.kfull, c.vfull):
            t.zero_()
        x, outs = k[:, :, :1].contiguous(), []
        wait = torch.cuda.synchronize if sync else (lambda: None)
        wait()
        for _ in range(20):
            s = ops.quantized_gemm(32, x, *keys, bits); wait()
            x = ops.quantized_gemm(32, s * 0.01, *values, bits); wait()
            proj = (k + x).transpose(1, 2).reshape(2, 1024, 8 * 128)
            c.reset()
            c.prefill_projected(proj, proj, cos, sin); wait()
            x = c.attend(x); wait()
            outs += [s, x, c.kcode.clone(), c.vcode.clone(), c.kfull.clone()]
        torch.cuda.synchronize()
        return outs
    for a, b in zip(run(True), run(False)):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("before", ["copy", "fill", "host", "fork", "nothing"])
def test_capture(cuda, before):
    """In a captured stream the launch before may be a copy, a fill or a join of another stream."""
    from kvmix_b200 import ops
    c = _cache(cuda, 2, 2, 1500, 2, 5)
    keys = ops.quantize_pack_last_dim_cuda(torch.randn((2, 8, 640, 128), device=cuda, dtype=torch.float16).transpose(2, 3), 32, 2)
    host = torch.randn((2, 8, 1, 128), dtype=torch.float16).pin_memory()
    src = host.to(cuda)
    q, out, side = torch.zeros_like(src), torch.empty_like(src), torch.cuda.Stream()
    want, want_s = c.attend(src).clone(), ops.quantized_gemm(32, src, *keys, 2).clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()

    def body():
        if before == "copy":
            q.copy_(src)
        elif before == "host":
            q.copy_(host, non_blocking=True)
        elif before == "fill":
            q.copy_(src)
            out.zero_()
        elif before == "fork":
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                q.copy_(src * 1.0)
            torch.cuda.current_stream().wait_stream(side)
        else:
            q.copy_(src * 1.0)
        c.attend(q, out=out)
        s = ops.quantized_gemm(32, q, *keys, 2)
        q.zero_()                                              # only after both have read it
        return s
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        body()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        s = body()
    for _ in range(5):
        out.fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int16), want.view(torch.int16)) and torch.equal(s.view(torch.int16), want_s.view(torch.int16))

"""Quantizer edges: prefill tiles of 128 / 132 rotated tokens, and data whose quotients tie everywhere -- bit for bit."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,G", [(4, 32), (2, 32), (1, 32), (4, 64), (2, 128), (1, 128), (3, 32)])
@pytest.mark.parametrize("L", [33, 44, 160, 165, 176, 289, 417])
def test_rotated_prefill_tiles(cuda, kb, G, L):
    """Keys rotated on the way in equal keys rotated by torch's fp16 arithmetic and then quantized."""
    import kvmix_b200 as kv
    gen = torch.Generator(device=cuda).manual_seed(L + kb)
    B, H, D = 2, 2, 128
    kp, vp = (torch.randn((B, L, H * D), generator=gen, device=cuda, dtype=torch.float16) for _ in range(2))
    ang = torch.arange(L, device=cuda).float()[:, None] / 10000.0 ** (torch.arange(0, D, 2, device=cuda).float() / D)
    cos, sin = (f(torch.cat((ang, ang), 1)).half() for f in (torch.cos, torch.sin))
    k = kp.view(B, L, H, D).transpose(1, 2)
    rot = torch.cat((-k[..., D // 2:], k[..., :D // 2]), -1)
    k = (k * cos) + (rot * sin)
    a, b = (kv.KVmixLayerCache(B, H, D, L + 64, kb, 2 if G < 128 else 4, G, residual_length=0, device=cuda) for _ in range(2))
    for c in (a, b):
        for t in (c.kcode, c.kscale, c.kmn, c.kfull):
            t.zero_()
    a.prefill_projected(kp, vp, cos, sin)
    b.prefill(k, vp.view(B, L, H, D).transpose(1, 2))
    assert a.tkq == b.tkq and a.k_len == b.k_len
    for x, y in ((a.kcode, b.kcode), (a.kscale, b.kscale), (a.kmn, b.kmn), (a.kfull, b.kfull)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("bits,G", [(1, 32), (2, 32), (2, 64), (3, 11), (4, 32), (4, 128)])
@pytest.mark.parametrize("strided", [False, True])
def test_ties_and_constant_groups(cuda, bits, G, strided):
    """Small integers: every quotient of a group is a multiple of a small fraction, ties among them; constant groups too."""
    import kvmix_b200 as kv
    rng = np.random.default_rng(bits * G)
    S = G * 12
    x = rng.integers(0, 2 * (1 << bits) - 1, (2, 2, 128, S)).astype(np.float16)
    x[:, :, ::7, :G] = 3.0
    t = torch.from_numpy(x).to(cuda)
    if strided:                                                # groups along a strided axis, channels contiguous
        t = t.transpose(2, 3).contiguous().transpose(2, 3)
    got = kv.quantize_pack_last_dim_cuda(t, G, bits)
    for g, w in zip(got, oracle.quantize_pack_last_dim(x, G, bits)):
        assert (g.cpu().numpy() == w).all()

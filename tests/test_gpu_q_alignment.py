"""Queries that start at an odd fp16 (views of a larger buffer, odd strides): every attention kernel reads them as it reads aligned ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,vb,G,nh,hkv", [(2, 3, 64, 8, 2), (3, 3, 64, 4, 2), (4, 4, 64, 8, 2), (3, 2, 64, 4, 2), (2, 2, 32, 4, 4), (2, 2, 32, 8, 2)])
@pytest.mark.parametrize("offset,row", [(1, 129), (3, 128), (2, 130)])
def test_misaligned_q(cuda, kb, vb, G, nh, hkv, offset, row):
    import kvmix_b200 as kv
    gen = torch.Generator(device=cuda).manual_seed(kb + vb)
    B, T = 2, 700
    k, v = (torch.randn((B, hkv, T, 128), generator=gen, device=cuda, dtype=torch.float16) for _ in range(2))
    q = torch.randn((B, nh, 1, 128), generator=gen, device=cuda, dtype=torch.float16)
    cache = kv.KVmixLayerCache(B, hkv, 128, T, kb, vb, G, residual_length=128, device=cuda)
    cache.prefill(k, v)
    buf = torch.zeros(offset + B * nh * row, device=cuda, dtype=torch.float16)
    view = buf[offset:].view(B, nh, 1, row)[..., :128]
    view.copy_(q)
    assert view.data_ptr() % 16 and torch.equal(cache.attend(view), cache.attend(q))

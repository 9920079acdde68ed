"""The attention kernels' channel splits (2 or 4 warps share a key tile of a short segment) and the edges of their tiles,
against the numpy oracle with upstream's rounding of the raw scores."""
import numpy as np
import pytest
import torch

from oracle.glue import RefLayerCache
from util import row_rel

pytestmark = pytest.mark.gpu

# One tile (split 4), two and three tiles (split 2), a ragged fourth, more tiles than warps; 88-token tiles for 3-bit keys.
TOKENS = (257, 385, 600, 861, 1023, 2100)


@pytest.mark.parametrize("kb,vb,G,nh,hkv", [(4, 2, 32, 2, 2), (2, 4, 64, 2, 2), (3, 1, 32, 2, 2), (1, 2, 128, 2, 2),
                                            (4, 4, 64, 8, 2), (3, 2, 64, 8, 2), (2, 1, 64, 4, 2), (1, 1, 128, 4, 1), (3, 3, 64, 8, 2), (4, 3, 32, 4, 2), (1, 3, 128, 4, 1)])
def test_short_and_ragged_contexts(cuda, kb, vb, G, nh, hkv):
    import kvmix_b200 as kv
    for T in TOKENS:
        rng = np.random.default_rng(100 * T + kb)
        k, v = (rng.standard_normal((1, hkv, T + 1, 128)).astype(np.float16) for _ in range(2))
        k[..., 3] *= 8
        q = rng.standard_normal((1, nh, 1, 128)).astype(np.float16)
        ref = RefLayerCache(kb, vb, G, residual_length=128)
        ref.prefill(k[:, :, :T], v[:, :, :T])
        ref.append(k[:, :, T:], v[:, :, T:])
        cache = kv.KVmixLayerCache(1, hkv, 128, T + 40, kb, vb, G, residual_length=128, device=cuda)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
        cache.prefill(t(k[:, :, :T]), t(v[:, :, :T]))
        got = cache.decode_step(t(q), t(k[:, :, T:]), t(v[:, :, T:])).cpu().numpy()
        # raw scores rounded to fp16 as the library does; what is left is p * scale in fp16 (2^-12 a token) and a score that
        # falls on the other side of a rounding boundary (one unit of 2^-6 at |score| 16 .. 32, times 1 / sqrt(128))
        err = row_rel(got, ref.attend(q, ref_rounding=1)).max()
        assert err <= 2e-3, (T, err)

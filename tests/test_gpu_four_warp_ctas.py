"""Launches of more heads than eight-warp CTA slots (296): four-warp CTAs, or whole heads followed by heads cut into pieces.  Every bit
pair through the fused step, host- and device-driven, with and without a mask, over a step on which groups fall due: the same
cache as append + attend, and the oracle on a few heads."""
import numpy as np
import pytest
import torch

from oracle.glue import RefLayerCache
from util import row_rel

pytestmark = pytest.mark.gpu

# (sequences, context): 320 heads as 296 whole ones and 24 cut (or all whole where a head is one or two tiles), 608 heads; 3400 tokens:
# eight-warp CTAs, whole and cut
SHAPES = [(10, 290), (10, 505), (10, 900), (19, 380), (10, 3400)]
PAIRS = [(kb, vb) for kb in (1, 2, 3, 4) for vb in (1, 2, 4)]


def _caches(cuda, n, B, T, kb, vb, G, k, v, **kw):
    import kvmix_b200 as kv
    out = [kv.KVmixLayerCache(B, 32, 128, T + 64, kb, vb, G, residual_length=128, device=cuda, **kw) for _ in range(n)]
    for c in out:
        c.prefill(k, v)
    return out


@pytest.mark.parametrize("kb,vb", PAIRS)
@pytest.mark.parametrize("shape", range(len(SHAPES)))
def test_fused_steps(cuda, kb, vb, shape):
    B, T = SHAPES[shape]
    G, steps = (32, 64, 128)[(kb + vb + shape) % 3], 3
    T = T // 11 * 11 + 5 if kb == 3 else T // G * G + G - 2     # a group of keys falls due on the second step, beyond the window of 128
    gen = torch.Generator(device=cuda).manual_seed(100 * T + 10 * kb + vb)
    rnd = lambda *s: torch.randn(s, generator=gen, device=cuda, dtype=torch.float16)
    k, v = rnd(B, 32, T + steps, 128), rnd(B, 32, T + steps, 128)
    k[..., 5] *= 8
    fused, plain = _caches(cuda, 2, B, T, kb, vb, G, k[:, :, :T], v[:, :, :T])
    driven, = _caches(cuda, 1, B, T, kb, vb, G, k[:, :, :T], v[:, :, :T], device_state=True)
    tkq, qs, masks, outs = fused.tkq, [], [], []
    for s in range(steps):
        q, mask = rnd(B, 32, 1, 128), None
        if s == 1:
            mask = torch.zeros((B, 1, 1, T + s + 1), device=cuda)
            mask[1, ..., :T // 3] = torch.finfo(torch.float32).min
            mask[2, ..., 7] = -3.0
        kn, vn = k[:, :, T + s:T + s + 1], v[:, :, T + s:T + s + 1]
        got = fused.decode_step(q, kn, vn, attention_mask=mask)
        dev = driven.decode_step(q, kn, vn, attention_mask=mask)
        plain.append(kn, vn)
        want = plain.attend(q, attention_mask=mask)
        qs.append(q), masks.append(mask), outs.append(got)
        assert fused._fused and driven._fused
        assert torch.equal(got, want) and torch.equal(dev, want)
        for a, b, c in zip(fused.as_tuple()[:8], plain.as_tuple()[:8], driven.as_tuple()[:8]):
            assert torch.equal(a, b) and torch.equal(a, c)
    assert fused.tkq > tkq
    for b, h in [(0, 0), (1, 3), (2, 20), (9, 8), (B - 1, 31)]:  # the first heads, masked ones, cut ones
        ref = RefLayerCache(kb, vb, G, residual_length=128)
        kk, vv = (t[b:b + 1, h:h + 1].cpu().numpy() for t in (k, v))
        ref.prefill(kk[:, :, :T], vv[:, :, :T])
        for s in range(steps):
            ref.append(kk[:, :, T + s:T + s + 1], vv[:, :, T + s:T + s + 1])
            m = None if masks[s] is None else masks[s][b:b + 1].cpu().numpy()
            w = ref.attend(qs[s][b:b + 1, h:h + 1].cpu().numpy(), ref_rounding=1, attention_mask=m)
            err = row_rel(outs[s][b:b + 1, h:h + 1].cpu().numpy(), w).max()
            assert err <= 2e-3, (b, h, s, err)                 # see test_gpu_channel_splits.py


@pytest.mark.parametrize("kb,vb,B,T", [(2, 2, 10, 420), (4, 4, 10, 1400), (3, 2, 19, 600), (1, 4, 10, 300)])
def test_captured_steps(cuda, kb, vb, B, T):
    """The device-driven form replayed from a graph that was laid out for more tokens than it finds."""
    import kvmix_b200 as kv
    gen = torch.Generator(device=cuda).manual_seed(T)
    rnd = lambda *s: torch.randn(s, generator=gen, device=cuda, dtype=torch.float16)
    steps = 40
    k, v = rnd(B, 32, T + steps, 128), rnd(B, 32, T + steps, 128)
    host, = _caches(cuda, 1, B, T, kb, vb, 32, k[:, :, :T], v[:, :, :T])
    dev, = _caches(cuda, 1, B, T, kb, vb, 32, k[:, :, :T], v[:, :, :T], device_state=True)
    q, kn, vn = (torch.zeros((B, 32, 1, 128), device=cuda, dtype=torch.float16) for _ in range(3))
    out = torch.zeros_like(q)
    step = kv.CapturedDecodeStep([dev], [q], [kn], [vn], [out], max_replays=steps)
    worst = 0.0
    for s in range(steps):
        q.copy_(rnd(B, 32, 1, 128)); kn.copy_(k[:, :, T + s:T + s + 1]); vn.copy_(v[:, :, T + s:T + s + 1])
        step.replay()
        want = host.decode_step(q, kn, vn)
        worst = max(worst, float(row_rel(out.cpu().numpy(), want.cpu().numpy()).max()))
    assert worst <= 1e-3, worst                                # two plans: see test_gpu_device_state.py
    for a, b in zip(host.as_tuple()[:8], dev.as_tuple()[:8]):
        assert torch.equal(a, b)

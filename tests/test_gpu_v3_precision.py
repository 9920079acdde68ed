"""Attention over 3-bit values against 64 bits where a few tokens hold most of the weight and where the groups of a token are of
very different size.  The queries are zero, so the additive mask alone sets the weights."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _attend(cuda, nh, hkv, v, mask, window=128, edit=None):
    import kvmix_b200 as kv
    T = v.shape[2]
    cache = kv.KVmixLayerCache(1, hkv, 128, T, 2, 3, 64, residual_length=window, device=cuda)
    k = np.random.default_rng(T).standard_normal(v.shape).astype(np.float16)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    cache.prefill(t(k), t(v))
    if edit is not None:
        edit(cache)
    q = torch.zeros((1, nh, 1, 128), dtype=torch.float16, device=cuda)
    got = cache.attend(q, attention_mask=t(mask)).float().cpu().numpy()[0, :, 0].astype(np.float64)
    tup = [None if x is None or isinstance(x, int) else x.cpu().numpy() for x in cache.as_tuple()]
    codes = np.stack([(tup[4].view(np.uint32) >> np.uint32(3 * i)) & np.uint32(3 if i == 10 else 7) for i in range(11)], -1)
    with np.errstate(all="ignore"):
        vq = (codes * tup[6].astype(np.float64)[..., None] + tup[7].astype(np.float64)[..., None]).reshape(1, hkv, -1, 132)[..., :128]
        full = np.repeat(np.concatenate([vq, tup[5].astype(np.float64)], 2)[0], nh // hkv, 0)
        p = np.exp(mask.astype(np.float64) - mask.max(-1, keepdims=True))[0, :, 0]
        p = np.broadcast_to(p / p.sum(-1, keepdims=True), (nh, T))
        want, mag = np.einsum("ht,htc->hc", p, full), np.einsum("ht,htc->hc", p, np.abs(full))
        # 3-bit codes and their complements, and 16 products a block cut off at 2^-15 code units of the block's largest p * scale
        Tq = tup[6].shape[2]
        sc = np.repeat(np.repeat(np.abs(tup[6].astype(np.float64)), 11, -1)[..., :128][0], nh // hkv, 0)
        ps = p[:, :Tq, None] * sc
        mag += 7 * ps.sum(1)
        cut = 16 * 2.0 ** -15 * np.pad(ps, ((0, 0), (0, -Tq % 16), (0, 0))).reshape(nh, -1, 16, 128).max(2).sum(1)
        return got, want, 2.0 ** -19 * mag + cut


# One fp16 rounding of the result (half of 2^-24 where it is subnormal), fp32 sums and an exponential accurate to 2^-19 of the magnitude
# summed, and what the tensor core cuts off next to a larger operand (see test_gpu_gemv_tiles.py)
def _check(got, want, rest):
    assert (np.abs(got - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -25 + rest).all()


@pytest.mark.parametrize("nh,hkv", [(8, 2), (4, 2), (2, 2)])
@pytest.mark.parametrize("sink", [0.0, 0.5, 0.9, 0.99, 0.9999])
def test_sink(cuda, nh, hkv, sink):
    for T in (2176, 8320):
        for sigma in (1.0, 0.1, 0.03, 1e-3):
            rng = np.random.default_rng(T + int(100 * sink))
            v = rng.standard_normal((1, hkv, T, 128)) * sigma
            w = rng.random((1, 1, 1, T)) + 0.1
            w *= (1 - sink) / w.sum()
            if sink:
                v[:, :, 40] *= 0.01
                w[..., 40] = sink
            _check(*_attend(cuda, nh, hkv, v.astype(np.float16), np.log(w).astype(np.float32)))


@pytest.mark.parametrize("sink", [0.0, 0.99])
def test_equal_small_weights(cuda, sink):
    """Weights that round the same way: an error per token does not average out."""
    v = np.abs(np.random.default_rng(1).standard_normal((1, 2, 2176, 128))) + 0.5
    w = np.full((1, 1, 1, 2176), (1 - sink) / 2176)
    if sink:
        w[..., 9], v[:, :, 9] = sink, v[:, :, 9] * 1e-3
    _check(*_attend(cuda, 8, 2, v.astype(np.float16), np.log(w).astype(np.float32)))


def test_groups_of_many_sizes(cuda):
    """Channel groups between 1e-4 and 1e3 times the others, rows between 0.01 and 10: every channel to its own accuracy."""
    rng = np.random.default_rng(5)
    v = rng.standard_normal((1, 2, 2400, 128)) * np.repeat(10.0 ** rng.integers(-4, 4, (1, 2, 1, 12)), 11, -1)[..., :128]
    v *= 10.0 ** rng.integers(-2, 2, (1, 2, 2400, 1))
    w = rng.random((1, 8, 1, 2400)) ** 4 + 1e-3
    _check(*_attend(cuda, 8, 2, np.clip(v, -60000, 60000).astype(np.float16), np.log(w).astype(np.float32)))


@pytest.mark.parametrize("token", [0, 20, 1000, 2170])
def test_infinite_scale(cuda, token):
    """An infinite scale: every channel of its group infinite (or NaN where a code of 0 meets it), the other channels as ever."""
    v = np.abs(np.random.default_rng(token).standard_normal((1, 2, 2400, 128)))
    w = np.random.default_rng(9).random((1, 8, 1, 2400)) + 0.1
    word = {}

    def edit(cache):
        cache.vscale[0, 1, token, 4] = float("inf")
        word[0] = int(cache.vcode[0, 1, token, 4]) & 0xffffffff
    got, want, mag = _attend(cuda, 8, 2, v.astype(np.float16), np.log(w).astype(np.float32), edit=edit)
    hit = np.zeros((8, 128), bool)
    hit[4:, 44:55] = True
    _check(got[~hit], want[~hit], mag[~hit])
    codes = np.array([(word[0] >> (3 * i)) & (3 if i == 10 else 7) for i in range(11)])
    assert (np.isnan(got[4:, 44:55]) == (codes == 0)).all() and (got[4:, 44:55][:, codes > 0] == np.inf).all()

"""quantized_gemm at the edges of its tensor-core form: column tiles of 128, stages of 32 rows, chunks of 2048 rows, clusters
that cut the rows, rows aligned to 16, 8 and 4 bytes -- against the same sum in 64 bits."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _case(bits, G, B, nh, hkv, K, N, seed, softmax=False):
    rng = np.random.default_rng(seed)
    w = rng.standard_normal((B, hkv, K, N)).astype(np.float16)
    c, s, m = oracle.quantize_pack_last_dim(w, G, bits)
    x = rng.standard_normal((B, nh, 1, K)).astype(np.float32)
    if softmax:
        x = np.exp(3 * x)
        x /= x.sum(-1, keepdims=True)
    return x.astype(np.float16), c, s, m


def _exact(x, c, s, m, bits, G, hkv):
    f = 32 // bits
    cu = c.view(np.uint32)
    codes = np.stack([(cu >> np.uint32(bits * i)) & np.uint32((1 << bits) - 1) for i in range(f)], -1).reshape(*c.shape[:3], -1)
    w = codes.astype(np.float64) * np.repeat(s.astype(np.float64), G, -1) + np.repeat(m.astype(np.float64), G, -1)
    w = np.repeat(w, x.shape[1] // hkv, 1)
    return np.einsum("bhk,bhkn->bhn", x[:, :, 0].astype(np.float64), w), np.einsum(
        "bhk,bhkn->bhn", np.abs(x[:, :, 0].astype(np.float64)), np.abs(w))


@pytest.mark.parametrize("bits,G", [(4, 32), (4, 128), (2, 32), (2, 64), (1, 32), (1, 64), (1, 128)])
@pytest.mark.parametrize("K,groups", [(128, 1), (128, 3), (128, 40), (32, 4), (100, 5), (1, 8), (700, 0), (4129, 0), (8192, 0)])
def test_tiles(cuda, bits, G, K, groups):
    import kvmix_b200 as kv
    N = groups * G if groups else 128                          # 0: the value side, 128 columns
    x, c, s, m = _case(bits, G, 1, 4, 2, K, N, K + bits + G, softmax=groups == 0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    got = kv.quantized_gemm(G, t(x), t(c), t(s), t(m), bits).float().cpu().numpy()[:, :, 0].astype(np.float64)
    want, mag = _exact(x, c, s, m, bits, G, 2)
    # One fp16 rounding of the result, and the tensor core's cut-off: it drops what lies 2^-25 below the largest operand exponents
    # of its 16 rows, and a code is a subnormal (exponent 2^-14, unit 2^-22 at 4 bits, 2^-20 at 1 and 2 bits), so a product loses
    # up to 2^-17 / 2^-19 code units of the largest in * scale next to it: of softmax weights exp(3 x), the largest of 16 is
    # some 8 times the mean, which makes 1e-5 .. 8e-5 of the magnitude summed if nothing cancelled; the alternating signs
    # leave a small part of it.
    assert (np.abs(got - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -24 + 2e-5 * mag).all()


@pytest.mark.parametrize("bits", [1, 2, 4])
def test_magnitudes(cuda, bits):
    """Inputs up to 60000 with scales of 1, results in range; and an infinite scale stays in its own group."""
    import kvmix_b200 as kv
    x, c, s, m = _case(bits, 32, 1, 1, 1, 64, 128, 7)
    x[0, 0, 0, 3] = 60000.0
    s[0, 0, 3], m[0, 0, 3] = 2.0 ** -6, 2.0 ** -6
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    got = kv.quantized_gemm(32, t(x), t(c), t(s), t(m), bits).float().cpu().numpy()[:, :, 0].astype(np.float64)
    want, mag = _exact(x, c, s, m, bits, 32, 1)
    assert (np.abs(got - want) <= 2.0 ** -11 * np.abs(want) + 2e-5 * mag).all()
    s[0, 0, 5, 2] = np.inf
    got2 = kv.quantized_gemm(32, t(x), t(c), t(s), t(m), bits).float().cpu().numpy()[:, :, 0]
    assert not np.isfinite(got2[..., 64:96]).any()
    assert (np.delete(got2, np.s_[64:96], -1) == np.delete(got.astype(np.float32), np.s_[64:96], -1)).all()

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


def _check(got, x, c, s, m, bits, G, hkv):
    """Within one fp16 rounding of the result (half of 2^-24 where it is subnormal) and what fp32 products and sums leave, whatever the
    sizes of scales and inputs: 16 accumulations in a row that the tensor core cuts off, 2^-23 of the terms' magnitude each
    (a code and its complement counted), and the cut-off described in test_tiles, 16 products a block at 2^-19 code units
    (2^-17 at 4 bits) of the block's largest in * scale."""
    want, _ = _exact(x, c, s, m, bits, G, hkv)
    xa = np.abs(x[:, :, 0].astype(np.float64))
    sa, za = (np.repeat(np.repeat(np.abs(t.astype(np.float64)), G, -1), x.shape[1] // hkv, 1) for t in (s, m))
    mag = np.einsum("bhk,bhkn->bhn", xa, sa * ((1 << bits) - 1) + za)
    pad = -x.shape[3] % 16
    xs = np.pad(xa[..., None] * sa, ((0, 0), (0, 0), (0, pad), (0, 0)))
    cut = 16 * xs.reshape(*xs.shape[:2], -1, 16, xs.shape[3]).max(3).sum(2) * 2.0 ** (-17 if bits == 4 else -19)
    ok = np.abs(want) < 65000
    assert (np.abs(got - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -25 + 2.0 ** -19 * mag + cut)[ok].all()


@pytest.mark.parametrize("bits,G", [(4, 32), (2, 32), (1, 32), (4, 128), (2, 64)])
@pytest.mark.parametrize("sink", [0.0, 0.5, 0.9, 0.99, 1.0])
def test_softmax_with_a_sink(cuda, bits, G, sink):
    """One token holds most of the weight and its value row is next to nothing: the others decide the result."""
    import kvmix_b200 as kv
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    for K in (2048, 8192):
        for sigma in (1.0, 0.1, 0.03, 1e-3):
            rng = np.random.default_rng(K + int(100 * sink))
            w = rng.standard_normal((1, 2, K, 128)) * sigma
            p = rng.random((1, 4, 1, K)) + 0.1
            p *= max(1 - sink, K * 2.0 ** -23) / p.sum(-1, keepdims=True)
            if sink:
                w[:, :, 5] *= 0.01
                p[..., 5] = sink
            c, s, m = oracle.quantize_pack_last_dim(w.astype(np.float16), G, bits)
            p = p.astype(np.float16)
            got = kv.quantized_gemm(G, t(p), t(c), t(s), t(m), bits).float().cpu().numpy()[:, :, 0].astype(np.float64)
            _check(got, p, c, s, m, bits, G, 2)


@pytest.mark.parametrize("bits,G", [(4, 32), (2, 32), (1, 32), (4, 64), (1, 128)])
@pytest.mark.parametrize("K,N", [(128, 4096), (2048, 128), (300, 256)])
def test_scales_of_many_sizes(cuda, bits, G, K, N):
    """Groups and rows between 1e-4 and 1e3 times the others, inputs between 1e-3 and 300: every column to its own accuracy."""
    import kvmix_b200 as kv
    rng = np.random.default_rng(K + bits)
    w = rng.standard_normal((1, 2, K, N)) * np.repeat(10.0 ** rng.integers(-4, 3, (1, 2, 1, N // G)), G, -1)
    w *= 10.0 ** rng.integers(-1, 2, (1, 2, K, 1))
    x = rng.standard_normal((1, 4, 1, K)) * 10.0 ** rng.integers(-3, 2, (1, 4, 1, K))
    x[..., 7] = 300.0
    c, s, m = oracle.quantize_pack_last_dim(w.astype(np.float16), G, bits)
    x = x.astype(np.float16)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    got = kv.quantized_gemm(G, t(x), t(c), t(s), t(m), bits).float().cpu().numpy()[:, :, 0].astype(np.float64)
    _check(got, x, c, s, m, bits, G, 2)


@pytest.mark.parametrize("bits", [1, 2, 4])
@pytest.mark.parametrize("row", [3, 19, 40])
def test_infinities(cuda, bits, row):
    """An infinite input, scale or zero gives what fp32 products and sums give: infinite, or NaN where 0 meets infinity."""
    import kvmix_b200 as kv
    x, c, s, m = _case(bits, 32, 1, 1, 1, 64, 128, 11 + row)
    s, m, x = np.abs(s), np.abs(m), np.abs(x)                  # non-negative terms: nothing cancels an infinity
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)

    def both(x, s, m):
        f = 32 // bits
        codes = np.stack([(c.view(np.uint32) >> np.uint32(bits * i)) & np.uint32((1 << bits) - 1) for i in range(f)], -1).reshape(1, 1, 64, 128)
        with np.errstate(all="ignore"):
            xs = x[0, 0, 0].astype(np.float32)[:, None] * np.repeat(s[0, 0].astype(np.float32), 32, -1)
            z = x[0, 0, 0].astype(np.float32)[:, None] * np.repeat(m[0, 0].astype(np.float32), 32, -1)
            want = (xs * codes[0, 0].astype(np.float32) + z).sum(0)
        got = kv.quantized_gemm(32, t(x), t(c), t(s), t(m), bits).float().cpu().numpy()[0, 0, 0]
        assert (np.isnan(got) == np.isnan(want)).all() and (np.isinf(got) == np.isinf(want)).all()
        assert (got[np.isinf(got)] == want[np.isinf(want)]).all()
    xi, si, mi = x.copy(), s.copy(), m.copy()
    xi[0, 0, 0, row], si[0, 0, row, 2], mi[0, 0, row, 1] = np.inf, np.inf, np.inf
    both(xi, s, m)
    both(x, si, m)
    both(x, s, mi)

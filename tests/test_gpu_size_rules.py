"""Forms that the kernels take by size, type or alignment, at the edges where one form hands over to the other: against the same
work asked for in the form that the rule does not take, or against the sum in 64 bits."""
import numpy as np
import pytest
import torch

from test_gpu_gemv_tiles import _case, _check
from test_gpu_prefill_projected import rope_tables, rotate_half
from util import REL_TOL

pytestmark = pytest.mark.gpu


def _same(a, b):
    return all((x is None and y is None) or (x.shape == y.shape and torch.equal(x.contiguous().view(torch.int16), y.contiguous().view(torch.int16)))
               for x, y in zip(a, b))


def _gen(cuda, seed):
    return torch.Generator(device=cuda).manual_seed(seed)


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
def test_contiguous_quantizer_units(cuda, bits):
    """From 4096 units a (b, h) slab and 8 waves of CTAs on a thread takes four units: slabs at both sides of the line, ragged ends, rows that
    lie apart -- as the same rows quantized a few heads at a time."""
    from kvmix_b200 import ops
    G, S, H = (11, 121, 240) if bits == 3 else (32, 128, 600)  # a row: 11 units of 11 values, or 4 of 32
    for A, spare in ((1023, 0), (1024, 0), (1025, 0), (1601, 0), (1601, 8), (2047, 1)):
        x = torch.randn((1, H, A, S + spare), generator=_gen(cuda, A), device=cuda, dtype=torch.float16)[..., :S]
        big = ops.quantize_pack_last_dim_cuda(x, G, bits)
        for h in range(0, H, 37):
            assert _same([t[:, h:h + 3] for t in big], ops.quantize_pack_last_dim_cuda(x[:, h:h + 3], G, bits)), (A, spare, h)


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
def test_strided_quantizer_rows(cuda, bits):
    """Tokens 128 elements apart take immediate offsets: as tokens that lie 136 apart, and as keys copied into [.., D, T] order."""
    from kvmix_b200 import ops
    for G in ((11,) if bits == 3 else (32, 64, 128)):
        for groups in (1, 2, 3, 7, 16, 17, 33):
            wide = torch.randn((2, 3, groups * G, 136), generator=_gen(cuda, G + groups), device=cuda, dtype=torch.float16)
            k = wide[..., :128].contiguous()
            want = ops.quantize_pack_last_dim_cuda(wide[..., :128].transpose(2, 3), G, bits)
            assert _same(ops.quantize_pack_last_dim_cuda(k.transpose(2, 3), G, bits), want), (G, groups)
            assert _same(ops.quantize_pack_last_dim_cuda(k.transpose(2, 3).contiguous(), G, bits), want), (G, groups)


@pytest.mark.parametrize("vb", [1, 2, 3, 4])
@pytest.mark.parametrize("kb,G", [(kb, G) for kb in (1, 2, 3, 4) for G in (32, 64, 128)])
def test_prefill_in_one_launch(cuda, kb, vb, G):
    """A prompt that is rotated on the way: as the rotated prompt, whose keys, values and tails are launches of their own."""
    import kvmix_b200 as kv
    for B, H, L, window in ((1, 1, 129 + G, 128), (2, 3, 773, 256), (1, 8, 1025, 128)):
        kp, vp = (torch.randn((B, L, H * 128), generator=_gen(cuda, L + i), device=cuda, dtype=torch.float16) for i in range(2))
        cos, sin = rope_tables(L, 128, cuda)
        k4 = kp.view(B, L, H, 128).transpose(1, 2)
        rot = (k4 * cos[None, None]) + (rotate_half(k4) * sin[None, None])
        one, three = (kv.KVmixLayerCache(B, H, 128, L + 8, kb, vb, G, residual_length=window, device=cuda) for _ in range(2))
        one.prefill_projected(kp, vp, cos, sin)
        three.prefill_projected(rot.transpose(1, 2).contiguous().view(B, L, H * 128), vp)
        assert one.tkq > 0 and one.tvq > 0
        assert _same(one.as_tuple()[:8], three.as_tuple()[:8]), (B, H, L)


@pytest.mark.parametrize("bits,G", [(4, 32), (2, 64), (1, 128), (2, 32)])
@pytest.mark.parametrize("K", [1, 100, 128, 511, 512, 513])
@pytest.mark.parametrize("tiles", [31.5, 32, 33])
def test_mat_vec_tiles_in_a_row(cuda, bits, G, K, tiles):
    """Up to 512 rows a warp takes two or four column tiles in a row where CTAs are many: 148 heads of 32 tiles are 592 CTAs of one tile
    a warp, 300 heads 600 of two; the last tile ragged; and 16-byte rows against rows 4 bytes off."""
    import kvmix_b200 as kv
    N = int(tiles * 128) // G * G
    rng = np.random.default_rng(K)
    for heads in (147, 148, 300):
        x, c, s, m = _case(bits, G, 1, 3, 3, K, N, K + bits)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
        pick = rng.integers(0, 3, heads)
        X, C, S, M = (t(a)[:, torch.from_numpy(pick).to(cuda)] for a in (x, c, s, m))
        got = kv.quantized_gemm(G, X, C, S, M, bits)
        ref = got.float().cpu().numpy()[:, :, 0].astype(np.float64)
        if heads == 300:
            for h in (0, 1, 150, 299):
                i = pick[h:h + 1]
                _check(ref[:, h:h + 1], x[:, i], c[:, i], s[:, i], m[:, i], bits, G, 1)
        for i in range(3):                                     # heads with the same operands
            assert (ref[0, pick == i] == ref[0, pick == i][:1]).all()
        off = torch.empty(C.numel() + 1, dtype=torch.int32, device=cuda)[1:].view(C.shape)
        off.copy_(C)
        assert torch.equal(kv.quantized_gemm(G, X, off, S, M, bits), got)


def _dense(packs, G, bits):
    code, s, m = packs
    f = 11 if bits == 3 else 32 // bits
    n = torch.arange(f, device=code.device, dtype=torch.int32)
    if bits == 3:                                              # ten fields of 3 bits and one of 2
        c = torch.where(n < 10, (code[..., None] >> (3 * n).clamp(max=27)) & 7, (code[..., None] >> 30) & 3)
    else:
        c = (code[..., None] >> (bits * n)) & ((1 << bits) - 1)
    c = c.reshape(*code.shape[:3], -1).double()
    return c * s.double().repeat_interleave(G, -1) + m.double().repeat_interleave(G, -1)


@pytest.mark.parametrize("nh,hkv", [(2, 2), (8, 2), (320, 320)])
@pytest.mark.parametrize("kb,vb", [(kb, vb) for kb in (1, 2, 3, 4) for vb in (1, 2, 4)])
def test_attention_group_sizes(cuda, kb, vb, nh, hkv):
    """Key and value groups of different sizes; packed parts that end inside a tile or fill half of one (3-bit keys: 176 tokens), a lone
    group; short and long fp16 tails -- against the softmax in 64 bits."""
    import kvmix_b200 as kv
    from kvmix_b200 import ops
    for kg in ((11,) if kb == 3 else (32, 64, 128)):
        for vg in (32, 64, 128):
            for nk, T in ((kg, kg + 34), (88 if kb == 3 else 128, 256), (99 if kb == 3 else 384, 431), (187 if kb == 3 else 640, 700), (1056 if kb == 3 else 1024, 1057)):
                nv = (T - 1) // 32 * 32
                if hkv > 2 and (T > 300 or vg == 64):
                    continue
                g = _gen(cuda, kg + T)
                k, v = (torch.randn((1, hkv, T, 128), generator=g, device=cuda, dtype=torch.float16) for _ in range(2))
                k[..., 3] *= 8
                q = torch.randn((1, nh, 1, 128), generator=g, device=cuda, dtype=torch.float16)
                kp = ops.quantize_pack_last_dim_cuda(k[:, :, :nk].transpose(2, 3), kg, kb)
                vp = ops.quantize_pack_last_dim_cuda(v[:, :, :nv].contiguous(), vg, vb)
                # room behind the rows, as a cache has it: rows of 16 bytes and more
                padded = [torch.nn.functional.pad(t, (0, -t.shape[3] % 32 + 32))[..., :t.shape[3]] for t in kp]
                got = kv.decode_attention(q, *padded, k[:, :, nk:].contiguous(), *vp, v[:, :, nv:].contiguous(), kb, kg, vb, vg,
                                          Tkq=nk, Tvq=nv, round_scores=False)
                K = torch.cat((_dense(kp, kg, kb).transpose(2, 3), k[:, :, nk:].double()), 2).repeat_interleave(nh // hkv, 1)
                V = torch.cat((_dense(vp, vg, vb), v[:, :, nv:].double()), 2).repeat_interleave(nh // hkv, 1)
                want = torch.softmax(q.double() @ K.transpose(2, 3) / 128 ** 0.5, -1) @ V
                err = (got.double() - want).norm(dim=-1) / want.norm(dim=-1)
                # p * scale in fp16 (2^-12 a token) and one fp16 rounding of the result, as everywhere in these tests
                assert err.max().item() <= REL_TOL, (kg, vg, nk, T, err.max().item())


@pytest.mark.parametrize("bits", [(2, 2), (3, 4)])
@pytest.mark.parametrize("nh", [74, 75, 148, 149])
def test_whole_heads_alone_on_their_sm(cuda, nh, bits):
    """75 .. 148 short heads stay whole: as the same heads asked for 30 at a time, which are cut."""
    import kvmix_b200 as kv
    g = _gen(cuda, nh)
    k, v = (torch.randn((1, nh, 1023, 128), generator=g, device=cuda, dtype=torch.float16) for _ in range(2))
    q = torch.randn((1, nh, 1, 128), generator=g, device=cuda, dtype=torch.float16)

    def attend(sl):
        c = kv.KVmixLayerCache(1, k[:, sl].shape[1], 128, 1100, *bits, 32, residual_length=128, device=cuda)
        c.prefill(k[:, sl], v[:, sl])
        return c.attend(q[:, sl].contiguous(), round_scores=False).double()
    got = attend(slice(None))
    want = torch.cat([attend(slice(i, min(i + 30, nh))) for i in range(0, nh, 30)], 1)
    # both round p * scale to fp16 (2^-12 a token), relative to another segment's maximum
    assert ((got - want).norm(dim=-1) / want.norm(dim=-1)).max().item() <= REL_TOL


@pytest.mark.parametrize("nh,nk,T", [(2, 352, 400), (64, 5874, 6000), (256, 3960, 4096), (256, 3971, 4003), (320, 693, 700), (320, 1034, 1050), (1024, 5621, 5700)])
def test_three_bit_key_tiles(cuda, nh, nk, T):
    """3-bit keys in tiles of 88 and of 176 tokens: a short segment whose tiles two warps share (88), a long one (176: three passes for five),
    whole heads on eight warps (176: three passes for six; 88: six passes would be seven) and on four (two passes in one; pieces;
    nine for seventeen), with ragged last tiles -- against the softmax in 64 bits, heads with the same operands alike."""
    import kvmix_b200 as kv
    from kvmix_b200 import ops
    g = _gen(cuda, nk)
    k, v = (torch.randn((1, 3, T, 128), generator=g, device=cuda, dtype=torch.float16) for _ in range(2))
    k[..., 3] *= 8
    q = torch.randn((1, 3, 1, 128), generator=g, device=cuda, dtype=torch.float16)
    nv = (T - 1) // 32 * 32
    kp = ops.quantize_pack_last_dim_cuda(k[:, :, :nk].transpose(2, 3), 11, 3)
    vp = ops.quantize_pack_last_dim_cuda(v[:, :, :nv].contiguous(), 32, 2)
    K = torch.cat((_dense(kp, 11, 3).transpose(2, 3), k[:, :, nk:].double()), 2)
    V = torch.cat((_dense(vp, 32, 2), v[:, :, nv:].double()), 2)
    want = torch.softmax(q.double() @ K.transpose(2, 3) / 128 ** 0.5, -1) @ V
    pick = torch.randint(0, 3, (nh,), generator=g, device=cuda)
    padded = [torch.nn.functional.pad(t, (0, -t.shape[3] % 32 + 32))[:, pick][..., :t.shape[3]] for t in kp]
    got = kv.decode_attention(q[:, pick].contiguous(), *padded, k[:, pick, nk:].contiguous(), *(t[:, pick].contiguous() for t in vp),
                              v[:, pick, nv:].contiguous(), 3, 11, 2, 32, Tkq=nk, Tvq=nv, round_scores=False)
    err = (got.double() - want[:, pick]).norm(dim=-1) / want[:, pick].norm(dim=-1)
    # p * scale in fp16 (2^-12 a token) and one fp16 rounding of the result, as everywhere in these tests
    assert err.max().item() <= REL_TOL
    if nh <= 256:                                              # all heads take the same segments
        for i in range(3):
            assert (got[:, pick == i] == got[:, pick == i][:, :1]).all()

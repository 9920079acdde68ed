"""What the framework is measured on: the calls a program makes that keeps its attention state in a mixed-precision KV
cache, over the range of sizes it makes them with.

Four kinds of pass, each through the public entry points:

    decode    one token for a stack of layers: ``KVmixLayerCache.decode_step`` layer by layer, or the whole step replayed
              from a graph (``CapturedDecodeStep``) where the caches keep their state on the device
    prefill   a prompt straight from the projections: ``KVmixLayerCache.prefill_projected`` for a stack of layers
    quantize  the drop-in quantizer on one layer's keys and values: ``quantize_pack_last_dim_cuda``
    gemv      the drop-in mat-vec pair of one decode step: ``quantized_gemm`` for q.K^T and for p.V

Inputs are seeded N(0, 1) tensors; keys carry four channels per head that are eight times larger, as the attention
configurations of ``kvmix_b200.configs`` have them, and the quantizer's inputs four heavy-tailed (Student-t, 3) channels.
"""
import random

import torch

from kvmix_b200 import ops
from kvmix_b200.cache import CapturedDecodeStep, KVmixLayerCache, kv_bytes_per_head, split_point
from kvmix_b200.configs import RESIDUAL_RATIO, synth_kv

D = 128                              # head dimension of every supported model
TOKENS = 8                           # different new tokens a decode loop cycles through
# the largest cases, which drawn ones stay below: (sequence, kv head, token) triples of one layer
DECODE_TRIPLES = 64 * 32 * 4096
QUANT_TRIPLES = 16 * 32 * 8192


def listed():
    decode = dict(kind="decode", masked=False)
    return [
        # the smallest call: one sequence, one layer, short context -- latency of a call from the host
        dict(decode, name="decode one short sequence", captured=False, batch=1, heads=32, kv_heads=32, context=1023,
             group=32, window=128, bits="42", steps=128),
        # a few left-padded sequences of a grouped-query model served from a host loop
        dict(decode, name="decode padded chat batch", captured=False, batch=4, heads=32, kv_heads=8, context=1537, group=64,
             window=128, bits="44 34 22 21", steps=128, masked=True),
        # upstream's own script for a grouped-query model: group 32 and the ratio policy, whose first steps still shrink the
        # prompt's fp16 tail
        dict(decode, name="decode ratio policy group 32", captured=False, batch=4, heads=32, kv_heads=8, context=3001,
             group=32, window=0, bits="44 32 22", steps=256),
        # the headline: 64 sequences of a 32-head model at 4096 tokens, the bit map in its proportions (8 : 12 : 12)
        dict(decode, name="decode batch 64", captured=True, batch=64, heads=32, kv_heads=32, context=4096, group=32,
             window=128, bits="44 32 32 22 22", steps=256),
        # one GPU's share of the same batch on eight GPUs
        dict(decode, name="decode batch 8", captured=True, batch=8, heads=32, kv_heads=32, context=4096, group=32,
             window=128, bits="44 32 32 22 22", steps=256),
        # grouped queries over 32k tokens, the bit map with 1-bit values in it
        dict(decode, name="decode grouped 32k", captured=True, batch=8, heads=32, kv_heads=8, context=32768, group=64,
             window=128, bits="44 34 34 22 21", steps=128),
        # the same map as its configuration writes it, with 3-bit values
        dict(decode, name="decode grouped 32k 3-bit values", captured=False, batch=8, heads=32, kv_heads=8, context=32768,
             group=64, window=128, bits="44 33 33 22 21", steps=128),
        # one very long sequence
        dict(decode, name="decode grouped 131k", captured=True, batch=1, heads=32, kv_heads=8, context=131072, group=128,
             window=256, bits="44 32 32 32 32", steps=64),
        # two long prompts of a grouped-query model, ragged length
        dict(kind="prefill", name="prefill 8k", batch=2, kv_heads=8, length=8191, group=64, window=128, bits="44 34 22"),
        # quantize-on-append: a large cell of the throughput sweep, and the group that falls due in a small decode batch
        # (keys copied into [.., D, T] order first, as the unmodified model files do)
        dict(kind="quantize", name="quantize large", batch=16, heads=32, tokens=8192, group=32, bits="24", copied=False),
        dict(kind="quantize", name="quantize due group", batch=4, heads=32, tokens=32, group=32, bits="42", copied=True),
        # what the unmodified model files call in every decode step
        dict(kind="gemv", name="gemv pair", batch=16, heads=32, kv_heads=32, tokens=4096, group=32, bits="22"),
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "captured", "captured", "captured", "prefill", "quantize", "quantize", "gemv"))
    if kind in ("decode", "captured"):
        captured = kind == "captured"
        heads, kv_heads = rng.choice(((32, 32), (32, 32), (32, 8), (32, 8), (16, 4), (8, 2), (4, 1)))
        batch = _spread(rng, 1, 64)
        context = _spread(rng, 300, max(600, min(131072, DECODE_TRIPLES // (batch * kv_heads))))
        # a captured step needs layouts whose cache update is part of the attention launch: groups of 64 or more for
        # grouped queries, a fixed window, no 3-bit values
        group = rng.choice((32, 64, 128)) if not captured or heads == kv_heads else rng.choice((64, 128))
        pairs = ["44", "32", "22", "34", "21", "42"] + ([] if captured else ["33"])
        return dict(kind="decode", captured=captured, batch=batch, heads=heads, kv_heads=kv_heads, context=context,
                    group=group, window=rng.choice((128, 128, 256)) if captured else rng.choice((0, 128, 256)),
                    bits=" ".join(rng.choice(pairs) for _ in range(rng.randint(1, 5))), steps=64,
                    masked=not captured and rng.random() < 0.3)
    if kind == "prefill":
        kv_heads, batch = rng.choice((8, 32)), _spread(rng, 1, 16)
        length = _spread(rng, 200, max(400, min(32768, QUANT_TRIPLES // (3 * batch * kv_heads))))
        pairs = ("44", "32", "22", "34", "21", "33")
        return dict(kind="prefill", batch=batch, kv_heads=kv_heads, length=length, group=rng.choice((32, 64, 128)),
                    window=rng.choice((0, 128, 256)), bits=" ".join(rng.choice(pairs) for _ in range(rng.randint(1, 3))))
    if kind == "quantize":
        batch, group = _spread(rng, 1, 64), rng.choice((32, 64, 128))
        groups = _spread(rng, 1, max(1, min(32768, QUANT_TRIPLES // (32 * batch)) // group))
        return dict(kind="quantize", batch=batch, heads=32, tokens=groups * group, group=group,
                    bits=rng.choice("1234") + rng.choice("124"), copied=rng.random() < 0.5)
    heads, kv_heads = rng.choice(((32, 32), (32, 8)))
    batch, group = _spread(rng, 1, 16), rng.choice((32, 64, 128))
    groups = _spread(rng, 2, 65536 // batch // group)
    return dict(kind="gemv", batch=batch, heads=heads, kv_heads=kv_heads, tokens=groups * group, group=group,
                bits=rng.choice("1234") + rng.choice("124"))


# ------------------------------------------------------------------------------------------------------
def _bits(case):
    return [(int(p[0]), int(p[1])) for p in case["bits"].split()]


def _key_group(case, k_bits):
    return 11 if k_bits == 3 else case["group"]


def _policy(case, k_bits, v_bits):
    if case["window"]:
        return dict(residual_length=case["window"])
    return dict(k_residual_ratio=RESIDUAL_RATIO[k_bits], v_residual_ratio=RESIDUAL_RATIO[v_bits])


def _caches(case, capacity, device_state=False):
    caches = []
    for kb, vb in _bits(case):
        c = KVmixLayerCache(case["batch"], case["kv_heads"], D, capacity, kb, vb, case["group"], device="cuda",
                            device_state=device_state, **_policy(case, kb, vb))
        for t in _buffers(c):
            t.zero_()                # the buffers are returned whole: spare capacity must hold something definite
        caches.append(c)
    return caches


def _buffers(c):
    return [c.kcode, c.kscale, c.kmn, c.vcode, c.vscale, c.vmn, c.kfull, c.vfull]


def _normal(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16)


def _prepare_decode(case, gen, seed):
    B, nh, hkv, n = case["batch"], case["heads"], case["kv_heads"], len(_bits(case))
    s = dict(case=case, left=case["steps"])
    s["k"], s["v"] = synth_kv(B, hkv, case["context"], D, torch.device("cuda"), seed)
    s["caches"] = _caches(case, case["context"] + case["steps"], device_state=case["captured"])
    for c in s["caches"]:
        c.prefill(s["k"], s["v"])
    if case["captured"]:
        s["q"] = [_normal(gen, B, nh, 1, D) for _ in range(n)]
        s["kn"] = [_normal(gen, B, hkv, 1, D) for _ in range(n)]
        s["vn"] = [_normal(gen, B, hkv, 1, D) for _ in range(n)]
        s["out"] = [torch.zeros_like(q) for q in s["q"]]
        s["step"] = CapturedDecodeStep(s["caches"], s["q"], s["kn"], s["vn"], s["out"], max_replays=case["steps"])
    else:
        s["new"] = [[(_normal(gen, B, nh, 1, D), _normal(gen, B, hkv, 1, D), _normal(gen, B, hkv, 1, D)) for _ in range(n)]
                    for _ in range(TOKENS)]
    s["mask"] = None
    if case["masked"]:
        pads = random.Random(seed)
        s["mask"] = torch.zeros((B, 1, 1, case["context"] + case["steps"]), device="cuda", dtype=torch.float16)
        for b in range(B):
            s["mask"][b, :, :, :pads.randint(0, case["context"] // 2)] = torch.finfo(torch.float16).min
    return s


def _run_decode(s):
    case = s["case"]
    if s["left"] == 0:               # the request is complete: its slot takes the next prompt
        for c in s["caches"]:
            c.reset()
            c.prefill(s["k"], s["v"])
        s["left"] = case["steps"]
        if case["captured"]:
            s["step"].left = case["steps"]
    if case["captured"]:
        s["step"].replay()
        outs = s["out"]
    else:
        new = s["new"][s["left"] % TOKENS]
        mask = None if s["mask"] is None else s["mask"][..., :s["caches"][0].kv_seq_len + 1]
        outs = [c.decode_step(*t, attention_mask=mask) for c, t in zip(s["caches"], new)]
    s["left"] -= 1
    return outs + [t for c in s["caches"] for t in _buffers(c)]


def _prepare_prefill(case, gen, seed):
    B, L, hkv = case["batch"], case["length"], case["kv_heads"]
    s = dict(case=case, caches=_caches(case, L + 64), proj=[])
    for i, _ in enumerate(_bits(case)):
        k, v = synth_kv(B, hkv, L, D, torch.device("cuda"), 16 * seed + i)
        s["proj"].append(tuple(t.transpose(1, 2).reshape(B, L, hkv * D) for t in (k, v)))    # as a projection writes them
    angle = torch.arange(L, device="cuda").float()[:, None] / 10000.0 ** (torch.arange(0, D, 2, device="cuda").float() / D)
    s["cos"], s["sin"] = (f(torch.cat((angle, angle), 1)).half() for f in (torch.cos, torch.sin))
    return s


def _run_prefill(s):
    for c, (k, v) in zip(s["caches"], s["proj"]):
        c.reset()
        c.prefill_projected(k, v, s["cos"], s["sin"])
    return [t for c in s["caches"] for t in _buffers(c)]


def _heavy_tailed(gen, *shape):
    x = _normal(gen, *shape)
    chi = torch.randn(shape[:-1] + (4, 3), generator=gen, device="cuda").square().sum(-1).div(3.0).sqrt()
    x[..., :4] = (x[..., :4].float() / chi).half()
    return x


def _prepare_quantize(case, gen, seed):
    B, H, T = case["batch"], case["heads"], case["tokens"]
    (kb, vb), = _bits(case)
    nk = T // 11 * 11 if kb == 3 else T
    k = _heavy_tailed(gen, B, H, T, D)[:, :, :nk].transpose(2, 3)
    return dict(case=case, k=k.contiguous() if case["copied"] else k, v=_heavy_tailed(gen, B, H, T, D))


def _run_quantize(s):
    case = s["case"]
    (kb, vb), = _bits(case)
    return (ops.quantize_pack_last_dim_cuda(s["k"], _key_group(case, kb), kb) +
            ops.quantize_pack_last_dim_cuda(s["v"], case["group"], vb))


def _prepare_gemv(case, gen, seed):
    B, nh, hkv, T = case["batch"], case["heads"], case["kv_heads"], case["tokens"]
    (kb, vb), = _bits(case)
    k, v = synth_kv(B, hkv, T, D, torch.device("cuda"), seed)
    if kb == 3:
        k = k[:, :, :T // 11 * 11]
    p = torch.softmax(torch.randn((B, nh, 1, T), generator=gen, device="cuda") * 2, -1).half()
    return dict(case=case, q=_normal(gen, B, nh, 1, D), p=p,
                keys=ops.quantize_pack_last_dim_cuda(k.transpose(2, 3), _key_group(case, kb), kb),
                values=ops.quantize_pack_last_dim_cuda(v, case["group"], vb))


def _run_gemv(s):
    case = s["case"]
    (kb, vb), = _bits(case)
    return (ops.quantized_gemm(_key_group(case, kb), s["q"], *s["keys"], kb),
            ops.quantized_gemm(case["group"], s["p"], *s["values"], vb))


_PREPARE = dict(decode=_prepare_decode, prefill=_prepare_prefill, quantize=_prepare_quantize, gemv=_prepare_gemv)
_RUN = dict(decode=_run_decode, prefill=_run_prefill, quantize=_run_quantize, gemv=_run_gemv)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return _PREPARE[case["kind"]](case, gen, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------------
def _tails(case, tokens, kb, vb):
    """Packed tokens of the keys and of the values once `tokens` are cached and the window policy has settled."""
    pol = dict(ratio=None, residual_length=case["window"])
    gk, gv = _key_group(case, kb), case["group"]
    if case["window"]:
        return split_point(tokens, gk, **pol), split_point(tokens, gv, **pol)
    # the ratio policy keeps less than a group and its share of it
    return (tokens - gk) // gk * gk, (tokens - gv) // gv * gv


def _cache_bytes(case, nk, nv, tokens, kb, vb):
    per_head = kv_bytes_per_head(nk, nv, tokens - nk, tokens - nv, D, kb, _key_group(case, kb), vb, 11 if vb == 3 else case["group"])
    return per_head * case["batch"] * case["kv_heads"]


def work(case):
    total = flops = 0
    kind = case["kind"]
    if kind == "decode":
        T = case["context"] + case["steps"] // 2
        for kb, vb in _bits(case):
            total += _cache_bytes(case, *_tails(case, T, kb, vb), T, kb, vb)
            total += 2 * case["batch"] * (case["heads"] + case["kv_heads"]) * D * 2              # q, k, v in, output out
            total += case["batch"] * T * 2 if case["masked"] else 0
            flops += 4 * case["batch"] * case["heads"] * T * D
    elif kind == "prefill":
        L, n = case["length"], case["batch"] * case["kv_heads"] * D
        for kb, vb in _bits(case):
            nk, nv = (split_point(L, g, residual_length=case["window"]) if case["window"] else
                      split_point(L, g, ratio=RESIDUAL_RATIO[b]) for g, b in ((_key_group(case, kb), kb), (case["group"], vb)))
            total += 2 * n * L * 2 + _cache_bytes(case, nk, nv, L, kb, vb)
        total += 2 * L * D * 2                                                                  # rotary tables
    elif kind == "quantize":
        (kb, vb), = _bits(case)
        T = case["tokens"]
        nk = T // 11 * 11 if kb == 3 else T
        as_cache = dict(case, kv_heads=case["heads"], window=0)
        n = case["batch"] * case["heads"] * D
        total = n * (nk + T) * 2 + _cache_bytes(as_cache, nk, T, T, kb, vb) - n * (T - nk) * 2
    else:
        (kb, vb), = _bits(case)
        T = case["tokens"]
        nk = T // 11 * 11 if kb == 3 else T
        total = _cache_bytes(case, nk, T, T, kb, vb) - case["batch"] * case["kv_heads"] * D * (T - nk) * 2
        total += case["batch"] * case["heads"] * (2 * D + nk + T) * 2                            # q, p in; scores, output out
        flops = 2 * case["batch"] * case["heads"] * (nk + T) * D
    return {"bytes": total, "flops": flops}


def tolerance(case):
    # Codes, scales, minima and fp16 tails have one right answer (whole values are compared exactly under every tolerance).
    if case["kind"] in ("prefill", "quantize"):
        return "exact"
    # fp16 outputs of fp32 sums: another order of the sums flips last bits only (against sums in 64 bits: 0.5e-5 .. 3.3e-5,
    # the largest difference one unit in the last place, 9.7e-4)
    if case["kind"] == "gemv":
        return {"rel": 1.4e-4, "max": 4e-3}
    # Attention carries probability * scale in fp16 once per token; two ways of cutting the tokens into segments are two
    # draws of that rounding (4.0e-4 .. 4.9e-4 between them)
    return {"rel": 2e-3}

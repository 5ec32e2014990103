"""What this framework is timed on: the calls a user makes, over the sizes they are made at.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw(rng)`` gives others of the same ranges,
``prepare`` makes what a user's program has in hand before the call and ``run`` makes the call through the public entry
points (``NSAAttention``, ``nsa_decode`` and its compressed cache, ``selection_attention``, ``flash_attn_func``,
``KVCompressorVarlen``).  Shapes are those of BASELINE.json and of the tests: 16 query heads per KV head, bf16,
compression block 32 / stride 16, selection block 64, top-16, window 512; inputs ~ N(0,1), weights ~ N(0,0.02).

Kinds of case
  train       NSAAttention forward + backward on ``batch`` sequences of ``tokens`` tokens (every gradient)
  packed      the same on ``nseq`` packed sequences of unequal length (cu_seqlens)
  prefill     NSAAttention forward without gradients
  decode      one new token for each of ``nseq`` cached sequences; with ``extend`` the compressed cache is first brought
              up to the token appended since the step before, as a generation loop does
  compress    KVCompressorVarlen forward + backward on packed sequences of unequal length
  select      selection_attention forward on given block indices (BASELINE.json's microbenchmark)
  compressed  flash_attn_func forward + backward: compressed attention and block selection alone
"""
import random

import torch

import nsa_b200
from nsa_b200.compression_kv import KVCompressorVarlen
from nsa_b200.decode import compress_cache, extend_compress_cache, nsa_decode
from nsa_b200.triton_attention import flash_attn_func

BLOCK, STRIDE, SEL_BLOCK, N_SEL, WINDOW = 32, 16, 64, 16, 512


def listed():
    return [
        # the smallest training step: BASELINE.json's first configuration (head_dim 64); launches and host work count
        dict(name="train_1k_d64", kind="train", batch=1, tokens=1024, heads=16, dim=64),
        # a small step at the usual head_dim; length as in the tests, not a multiple of the 64-key selection block
        dict(name="train_2k", kind="train", batch=2, tokens=2080, heads=32, dim=128),
        # the headline configuration
        dict(name="train_8k", kind="train", batch=8, tokens=8192, heads=64, dim=128),
        # long context on one GPU; the largest case
        dict(name="train_64k", kind="train", batch=1, tokens=65536, heads=64, dim=128),
        # fine-tuning on packed documents of unequal length
        dict(name="train_packed", kind="packed", nseq=6, shortest=1024, longest=4096, lengths=11, heads=64, dim=128),
        # a prompt of arbitrary (odd) length through an inference-only forward
        dict(name="prefill_5k", kind="prefill", batch=1, tokens=5003, heads=64, dim=128),
        # one user's next token: the smallest call, all latency
        dict(name="decode_1", kind="decode", nseq=1, shortest=4096, longest=4096, lengths=1, heads=64, dim=128, extend=False),
        # a serving batch: BASELINE.json's decode configuration
        dict(name="decode_128", kind="decode", nseq=128, shortest=4096, longest=32768, lengths=4, heads=64, dim=128,
             extend=False),
        # a whole generation step of a serving batch: extend the compressed cache by the appended token, then decode
        dict(name="generate_32", kind="decode", nseq=32, shortest=2048, longest=16384, lengths=7, heads=64, dim=128,
             extend=True),
        # the trainable compression alone on packed sequences
        dict(name="compress_packed", kind="compress", nseq=8, shortest=500, longest=9000, lengths=3, heads=64, dim=128),
        # BASELINE.json's selection microbenchmark
        dict(name="select_8k", kind="select", batch=4, tokens=8192, heads=64, dim=128),
        # compressed attention + block selection as a building block of a user's own module
        dict(name="compressed_4k", kind="compressed", batch=2, tokens=4096, heads=64, dim=128),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, evenly spread over the logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["train", "train", "packed", "prefill", "decode", "decode", "generate", "compress", "select",
                       "compressed"])
    heads = rng.choice([16, 32, 64])
    dim = 128
    if kind in ("train", "prefill", "compressed", "select"):
        tokens = _log(rng, 1024, {"train": 32768, "prefill": 65536}.get(kind, 16384))
        batch = rng.randint(1, max(1, min(8, 32768 // tokens)))
        if kind != "select" and tokens <= 4096 and rng.random() < 0.25:
            dim = 64
        return dict(kind=kind, batch=batch, tokens=tokens, heads=heads, dim=dim)
    if kind == "packed":
        shortest = _log(rng, 1024, 2048)
        return dict(kind=kind, nseq=rng.randint(2, 8), shortest=shortest, longest=_log(rng, shortest, 8192),
                    lengths=rng.randrange(1 << 20), heads=heads, dim=dim)
    if kind == "compress":
        shortest = _log(rng, 100, 2000)
        return dict(kind=kind, nseq=rng.randint(1, 16), shortest=shortest, longest=_log(rng, shortest, 16384),
                    lengths=rng.randrange(1 << 20), heads=heads, dim=rng.choice([64, 128, 128]))
    shortest = _log(rng, 1024, 8192)
    return dict(kind="decode", nseq=_log(rng, 1, 128), shortest=shortest, longest=_log(rng, shortest, 32768),
                lengths=rng.randrange(1 << 20), heads=heads, dim=dim, extend=kind == "generate")


def _lengths(case):
    rng = random.Random(case["lengths"])
    return [rng.randint(case["shortest"], case["longest"]) for _ in range(case["nseq"])]


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


def _module(case, gen):
    mod = nsa_b200.NSAAttention(case["dim"], True, None, 0.0, compression_stride=STRIDE, compression_block=BLOCK,
                                selection_block=SEL_BLOCK, selected_block_count=N_SEL, sliding_window=WINDOW,
                                device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0.0, 0.02, generator=gen)
    return mod


def _block_indices(B, T, H, gen):
    """Per (token, KV head) up to 16 distinct blocks drawn evenly from the causally valid ones, always with the first
    and the token's own; unused slots hold -1."""
    nb = (T + SEL_BLOCK - 1) // SEL_BLOCK
    own = (torch.arange(T, device="cuda") // SEL_BLOCK).view(T, 1, 1)
    blk = torch.arange(nb, device="cuda").view(1, 1, nb)
    out = torch.full((B, T, H, N_SEL), -1, dtype=torch.int64, device="cuda")
    for b in range(B):
        r = torch.rand(T, H, nb, generator=gen, device="cuda")
        r = torch.where((blk == 0) | (blk == own), 2.0, torch.where(blk < own, r, -1.0))
        top = torch.topk(r, min(N_SEL, nb), dim=-1)
        out[b, :, :, :top.indices.shape[-1]] = torch.where(top.values >= 0, top.indices, -1)
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, Hq, D = case["kind"], case["heads"], case["dim"]
    Hkv = Hq // 16

    def normal(*shape, grad=False):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.bfloat16).requires_grad_(grad)

    if kind in ("train", "packed", "prefill"):
        lens = [case["tokens"]] * case["batch"] if kind != "packed" else _lengths(case)
        n, grad = sum(lens), kind != "prefill"
        s = dict(module=_module(case, gen), q=normal(n, Hq, D, grad=grad), k=normal(n, Hkv, D, grad=grad),
                 v=normal(n, Hkv, D, grad=grad), cu=torch.tensor(_cu(lens), dtype=torch.int32, device="cuda"),
                 longest=max(lens))
        if grad:
            s["do"] = normal(n, Hq, D)
            s["names"] = [name for name, _ in s["module"].named_parameters()]
        else:
            s["module"].requires_grad_(False)
    elif kind == "decode":
        lens = _lengths(case)
        cu = _cu(lens)
        s = dict(module=_module(case, gen).requires_grad_(False), q=normal(len(lens), Hq, D), k=normal(cu[-1], Hkv, D),
                 v=normal(cu[-1], Hkv, D), cu=cu)
        if case["extend"]:   # the cache as the step before left it: one token shorter everywhere
            keep = torch.ones(cu[-1], dtype=torch.bool, device="cuda")
            keep[torch.tensor(cu[1:], device="cuda") - 1] = False
            s["cache"] = compress_cache(s["module"], s["k"][keep], s["v"][keep], _cu([n - 1 for n in lens]))
        else:
            s["cache"] = compress_cache(s["module"], s["k"], s["v"], cu)
    elif kind == "compress":
        lens = _lengths(case)
        comp = KVCompressorVarlen(STRIDE, BLOCK, D, "cuda", torch.bfloat16)
        with torch.no_grad():
            for p in comp.parameters():
                p.normal_(0.0, 0.02, generator=gen)
        outs = sum(max((n - BLOCK) // STRIDE, 0) for n in lens)
        s = dict(module=comp, k=normal(sum(lens), Hkv, D, grad=True), v=normal(sum(lens), Hkv, D, grad=True), cu=_cu(lens),
                 dck=normal(outs, Hkv, D), dcv=normal(outs, Hkv, D))
    elif kind == "select":
        B, T = case["batch"], case["tokens"]
        s = dict(q=normal(B, T, Hq, D), k=normal(B, T, Hkv, D), v=normal(B, T, Hkv, D), g=normal(B, T, Hq).sigmoid(),
                 idx=_block_indices(B, T, Hkv, gen))
    else:
        B, T = case["batch"], case["tokens"]
        Tc = (T - BLOCK) // STRIDE + 1
        s = dict(q=normal(B, T, Hq, D, grad=True), ck=normal(B, Tc, Hkv, D, grad=True), cv=normal(B, Tc, Hkv, D, grad=True),
                 do=normal(B, T, Hq, D), kv_heads=Hkv)
    s["case"] = case
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind in ("train", "packed"):
        m = s["module"]
        o = m(s["q"], s["k"], s["v"], s["cu"], s["longest"])
        grads = torch.autograd.grad(o, [s["q"], s["k"], s["v"], *m.parameters()], s["do"])
        out = dict(zip(["o", "dq", "dk", "dv", *s["names"]], [o, *grads]))
        # A key bias of the compression adds the same amount to every logit of a row, so its gradient is zero: what is
        # computed for it is what the roundings leave, and is not compared.
        del out["compressor.compressor_k.bias"]
        return out
    if kind == "prefill":
        with torch.no_grad():
            return s["module"](s["q"], s["k"], s["v"], s["cu"], s["longest"])
    if kind == "decode":
        if not s["case"]["extend"]:
            return nsa_decode(s["module"], s["q"], s["k"], s["v"], s["cu"], s["cache"])
        cache = extend_compress_cache(s["module"], s["cache"], s["k"], s["v"], s["cu"])
        o = nsa_decode(s["module"], s["q"], s["k"], s["v"], s["cu"], cache)
        return dict(o=o, ck=cache.ck, cv=cache.cv)
    if kind == "compress":
        ck, cv, cu_out = s["module"](s["k"], s["v"], s["cu"])
        dk, dv, dwk, dwv = torch.autograd.grad([ck, cv], [s["k"], s["v"], *s["module"].parameters()], [s["dck"], s["dcv"]])
        return dict(ck=ck, cv=cv, cu_out=cu_out, dk=dk, dv=dv, dwk=dwk, dwv=dwv)
    if kind == "select":
        with torch.no_grad():
            return nsa_b200.selection_attention(s["q"], s["k"], s["v"], s["g"], s["g"], s["idx"])
    o, idx = flash_attn_func(s["q"], s["ck"], s["cv"], STRIDE, BLOCK, True, None, s["kv_heads"],
                             SEL_BLOCK // STRIDE + 1, SEL_BLOCK // STRIDE, BLOCK // STRIDE - 2, N_SEL)
    dq, dck, dcv = torch.autograd.grad(o, [s["q"], s["ck"], s["cv"]], s["do"])
    return dict(o=o, idx=idx, dq=dq, dck=dck, dcv=dcv)


def _attention_flops(T, Hq, D, parts, backward):
    """(key, query head) pairs that one sequence of T tokens visits, times 4 D for the two products of the forward and
    10 D for the five of the backward.  The selection follows the reference's unmasked scores, for which blocks of the
    future are as likely as others and are skipped; its scores cost one more product over all compressed keys."""
    Tc, nb = (T - BLOCK) // STRIDE + 1, (T + SEL_BLOCK - 1) // SEL_BLOCK
    pairs, score = 0.0, 0.0
    if "cmp" in parts:
        pairs += sum(min(max((t - BLOCK) // STRIDE + 1, 0), Tc) for t in range(T))
        score = 2.0 * D * T * Tc
    if "own" in parts:    # the module's own selection
        pairs += sum(SEL_BLOCK * N_SEL * min(1.0, (t // SEL_BLOCK + 1) / nb) for t in range(T))
    if "given" in parts:  # indices that are all causally valid
        pairs += sum(SEL_BLOCK * min(N_SEL, t // SEL_BLOCK + 1) for t in range(T))
    if "win" in parts:
        pairs += sum(min(t + 1, WINDOW) for t in range(T))
    return Hq * (pairs * D * (14.0 if backward else 4.0) + score)


def work(case):
    kind, Hq, D = case["kind"], case["heads"], case["dim"]
    Hkv = Hq // 16
    lens = [case["tokens"]] * case["batch"] if "tokens" in case else _lengths(case)
    n, comp = sum(lens), 2.0 * BLOCK * D * D
    row, kvrow, weights = 2.0 * Hq * D, 2.0 * Hkv * D, 2.0 * 2 * BLOCK * D * D
    outs = sum(max((t - BLOCK) // STRIDE + 1, 0) for t in lens)
    if kind in ("train", "packed", "prefill"):
        grad = kind != "prefill"
        per = {t: _attention_flops(t, Hq, D, ("cmp", "own", "win"), grad) for t in set(lens)}
        flops = sum(per[t] for t in lens) + (3 if grad else 1) * (2 * outs * Hkv * comp + 6.0 * D * n * Hq)
        # forward: q, k, v -> o; backward: dO as well, dq, dk, dv and the weights' gradients
        return dict(bytes=n * (row * (4 if grad else 2) + kvrow * (4 if grad else 2)) + weights * (2 if grad else 1), flops=flops)
    if kind == "decode":
        tc = [(t - BLOCK) // STRIDE + 1 for t in lens]
        seen = sum(min(N_SEL * SEL_BLOCK, t) + min(WINDOW, t) for t in lens)
        # q and o; the compressed cache, the selected blocks and the window, each key with its value
        b = 2 * len(lens) * row + 2 * kvrow * (sum(tc) + seen)
        if case["extend"]:   # the caches are packed: the grown one is written whole
            b += 2 * kvrow * sum(tc)
        return dict(bytes=b, flops=Hq * D * (4.0 * seen + 6.0 * sum(tc)))
    if kind == "compress":
        return dict(bytes=2 * kvrow * (2 * n + 2 * outs) + 2 * weights, flops=3 * 2 * outs * Hkv * comp)
    T, B = case["tokens"], case["batch"]
    if kind == "select":
        return dict(bytes=n * (2 * row + 2 * kvrow + 2 * Hq + 8 * Hkv * N_SEL),
                    flops=B * _attention_flops(T, Hq, D, ("given",), False))
    return dict(bytes=n * (4 * row + 8 * Hkv * N_SEL) + 4 * kvrow * outs, flops=B * _attention_flops(T, Hq, D, ("cmp",), True))


def tolerance(case):
    kind = case["kind"]
    if kind == "select":
        return dict(rel=1e-2, max=0.2)
    if kind == "compress":
        return dict(rel=1e-2, max=0.1)
    # bf16 results of bf16 products.  A block whose score ties with the last one chosen, to within the roundings of a
    # 32-bit sum, may be exchanged for it: a few rows then change as a whole, and a few indices differ.
    return dict(rel=1e-2, max=0.9, differ=1e-3)

"""Batched decode with 1, 2, 4 and 8 CTAs per (sequence, KV head), which depends on how many there are: the same sequences
decoded in one batch of 40 and in smaller ones, from a few tokens to several tiles of every phase."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("Hkv,parts", [(4, (1, 2, 5, 10)), (1, (3, 20, 40))])
def test_decode_batches_agree(Hkv, parts, seed):
    """The blocks are the same ones whatever the batch: the caches and the scores do not depend on it.  What a branch adds up in another
    order differs by roundings."""
    import nsa_b200 as nsa
    from nsa_b200.decode import nsa_decode
    torch.manual_seed(seed)   # the module's weights
    gen = torch.Generator(device=DEV).manual_seed(100 * seed + Hkv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    lens = [40, 5000, 1, 33, 700, 64, 2047, 9000, 513, 1100] + [100 + 37 * i for i in range(150 // Hkv)]
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    k, v, q = rnd(cu[-1], Hkv, 128), rnd(cu[-1], Hkv, 128), rnd(len(lens), 16 * Hkv, 128)
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)

    def run(a, b):
        c = [x - cu[a] for x in cu[a:b + 1]]
        return nsa_decode(mod, q[a:b], k[cu[a]:cu[b]], v[cu[a]:cu[b]], torch.tensor(c, dtype=torch.int32, device=DEV), return_parts=True)

    o, (o_cmp, o_slc, o_swa, lse, idx) = run(0, len(lens))
    at = 0
    for n in parts:
        got, got_parts = run(at, at + n)
        sl = slice(at, at + n)
        assert torch.equal(got_parts[4], idx[sl])
        for name, x, ref in (("o", got, o), ("cmp", got_parts[0], o_cmp), ("slc", got_parts[1], o_slc), ("swa", got_parts[2], o_swa)):
            _close("decode %s, %d at %d" % (name, n, at), x, ref[sl])
        assert torch.allclose(got_parts[3].nan_to_num(neginf=-1e4), lse[:, sl].nan_to_num(neginf=-1e4), atol=1e-4)
        at = min(at + n, len(lens) - 40)
    nsa._lib.device_status()


@pytest.mark.parametrize("nseq", [2, 30, 40])   # clusters, an SM an item, a CTA of half of an SM's warps an item
def test_decode_passes_nan_on(nseq):
    """A NaN in a key, a value or the query makes the outputs that see it NaN, and no others."""
    import nsa_b200 as nsa
    from nsa_b200.decode import compress_cache, nsa_decode
    gen = torch.Generator(device=DEV).manual_seed(nseq)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    L, H = 3000, 4
    cu = [L * i for i in range(nseq + 1)]
    q, k, v = rnd(nseq, 16 * H, 128), rnd(nseq * L, H, 128), rnd(nseq * L, H, 128)
    cache = compress_cache(mod, k, v, cu)

    def run(q=q, k=k, v=v, ck=cache.ck, cv=cache.cv):
        cache.ck, cache.cv = ck, cv
        o, (o_cmp, o_slc, o_swa, _, _) = nsa_decode(mod, q, k, v, cu, cache, return_parts=True)
        return dict(o=o, cmp=o_cmp, slc=o_slc, swa=o_swa)

    def spoiled(x, row):   # head 1 of sequence 1's row, in one channel or (two heads of q) all
        y = x.clone()
        y[row, 1 if x is not q else 16, 5] = float("nan")
        return y

    base, tc = run(), cache.cu_c[1]
    for change, branches in ((dict(k=spoiled(k, 2 * L - 100)), ("swa",)), (dict(v=spoiled(v, 2 * L - 100)), ("swa",)),
                             (dict(ck=spoiled(cache.ck, tc + 50)), ("cmp",)), (dict(cv=spoiled(cache.cv, tc + 50)), ("cmp",)),
                             (dict(q=spoiled(q, 1)), ("cmp", "swa"))):
        got = run(**change)
        for name in ("o", "cmp", "swa"):
            nan = torch.isnan(got[name])
            hit = torch.zeros_like(nan)
            if name == "o" or name in branches:
                rows = slice(16, 17) if "q" in change else slice(16, 32)      # the query heads of KV head 1
                chan = slice(5, 6) if "v" in change or "cv" in change else slice(0, 128)
                hit[1, rows, chan] = True
            if "ck" in change:   # the scores of that group are spoiled as well: its blocks may be others
                assert nan[hit].all() and not nan[0].any()
                continue
            assert torch.equal(nan, hit), (list(change), name)
            assert torch.equal(got[name][0], base[name][0])

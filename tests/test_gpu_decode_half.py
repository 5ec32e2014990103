"""Decode with two CTAs of three warps per SM (more items than SMs) and with one of six: every sum is the same six chains in
either, so the blocks and the outputs are the same bit for bit.  Batches on both sides of the rule that chooses between them."""
import pytest
import torch

from oracle import nsa_oracle as O
from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


# items (sequences x KV heads): 148 SMs; two CTAs per SM from 149 items on, but below 296 only up to 12 K (22 K with 295) keys, and up
# to 444 only where lengths differ (test_equal_lengths)
@pytest.mark.parametrize("nseq,Hkv,longest", [(150, 1, 700), (74, 2, 12000), (75, 2, 14000), (150, 2, 3000), (40, 4, 1), (300, 1, 1), (300, 1, 2100)])
def test_blocks_do_not_depend_on_the_spread(nseq, Hkv, longest):
    import nsa_b200 as nsa
    from nsa_b200.decode import nsa_decode
    torch.manual_seed(nseq)
    gen = torch.Generator(device=DEV).manual_seed(nseq + Hkv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    # around the chains' tile pairs of 128 positions (2048 keys) and the first block; one long sequence decides the rule
    lens = [longest] + [(1, 31, 32, 2063, 2064, 2080, 4111, 4112, 700)[i % 9] if longest > 1 else 40 + i for i in range(nseq - 1)]
    cu = [sum(lens[:i]) for i in range(nseq + 1)]
    k, v, q = rnd(cu[-1], Hkv, 128), rnd(cu[-1], Hkv, 128), rnd(nseq, 16 * Hkv, 128)
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)

    def run(a, b):
        c = [x - cu[a] for x in cu[a:b + 1]]
        return nsa_decode(mod, q[a:b], k[cu[a]:cu[b]], v[cu[a]:cu[b]], torch.tensor(c, dtype=torch.int32, device=DEV), return_parts=True)

    o, (_, _, _, lse, idx) = run(0, nseq)
    for a in range(0, nseq, 30):   # clusters, or a CTA per item
        b = min(a + 30, nseq)
        got, parts = run(a, b)
        assert torch.equal(parts[4], idx[a:b])
        _close("decode o, %d of %d" % (b - a, nseq), got, o[a:b])
        assert torch.allclose(parts[3].nan_to_num(neginf=-1e4), lse[:, a:b].nan_to_num(neginf=-1e4), atol=1e-4)
    nsa._lib.device_status()


# below 296 items the longest sequence decides: 150 items up to 12.3 K keys in pairs of CTAs, 290 up to 22.1 K
@pytest.mark.parametrize("nseq,short,long", [(150, 6000, 14000), (290, 1200, 24000), (212, 700, 18000)])
def test_outputs_do_not_depend_on_the_form(nseq, short, long):
    """The same batch but for its longest sequence, whose length decides between the two forms: every other sequence gets the same bits in
    the output, the branches and their statistics, wherever it stands among the items of a CTA."""
    import nsa_b200 as nsa
    from nsa_b200.decode import nsa_decode
    torch.manual_seed(nseq)
    gen = torch.Generator(device=DEV).manual_seed(nseq)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    lens = [short] + [(1, 31, 32, 63, 64, 65, 129, 500, 513, 577, 640, 3 * short // 4, short - 1)[i % 13] for i in range(nseq - 1)]
    n = sum(lens)
    k, v, q = rnd(n - short + long, 1, 128), rnd(n - short + long, 1, 128), rnd(nseq, 16, 128)
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)

    def run(first):
        a = long - first     # the sequences behind the first one keep their keys
        cu = [0, first]
        for x in lens[1:]:
            cu.append(cu[-1] + x)
        o, (o_cmp, o_slc, o_swa, lse, idx) = nsa_decode(mod, q, k[a:], v[a:], cu, return_parts=True)
        return dict(o=o, cmp=o_cmp, slc=o_slc, swa=o_swa, lse=lse.transpose(0, 1), idx=idx)

    pair, one = run(short), run(long)
    for name in pair:
        assert torch.equal(pair[name][1:], one[name][1:]), name
    nsa._lib.device_status()


@pytest.mark.parametrize("nseq,Hkv,L", [(160, 1, 2100), (75, 4, 2100), (150, 3, 1000)])   # 160 items: pairs; 300: one CTA per SM; 450: pairs
def test_equal_lengths(nseq, Hkv, L):
    """Sequences of one length, up to three items per SM of which are not dealt to pairs of CTAs: the blocks of small batches."""
    import nsa_b200 as nsa
    from nsa_b200.decode import nsa_decode
    torch.manual_seed(nseq)
    gen = torch.Generator(device=DEV).manual_seed(nseq)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    k, v, q = rnd(nseq * L, Hkv, 128), rnd(nseq * L, Hkv, 128), rnd(nseq, 16 * Hkv, 128)
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    run = lambda a, b: nsa_decode(mod, q[a:b], k[a * L:b * L], v[a * L:b * L], [L * i for i in range(b - a + 1)], return_parts=True)
    o, parts = run(0, nseq)
    for a in range(0, nseq, 30):
        b = min(a + 30, nseq)
        got, got_parts = run(a, b)
        assert torch.equal(got_parts[4], parts[4][a:b])
        _close("decode o, %d equal of %d" % (b - a, nseq), got, o[a:b])
    nsa._lib.device_status()


def test_rows_match_the_oracle():
    """Rows of a batch that is dealt to pairs of CTAs (160 items) against the fp32 oracle on the kernel's compressed cache."""
    import nsa_b200 as nsa
    from nsa_b200.decode import compress_cache, nsa_decode
    gen = torch.Generator().manual_seed(160)
    r = lambda *s, m=1.0: (torch.randn(*s, generator=gen) * m).bfloat16().float()
    lens = [(20, 40, 95, 300, 517, 700, 1061, 2048)[i % 8] for i in range(160)]
    cu = [sum(lens[:i]) for i in range(161)]
    q, k, v = r(160, 16, 128), r(cu[-1], 1, 128), r(cu[-1], 1, 128)
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    for p in mod.parameters():
        p.copy_(r(*p.shape, m=0.02))
    d = lambda x: x.to(DEV, torch.bfloat16)
    cache = compress_cache(mod, d(k), d(v), cu)
    o = nsa_decode(mod, d(q), d(k), d(v), cu, cache)
    nsa._lib.device_status()
    ck, cv, _, cu_c = cache
    weights = [t.detach().float().cpu() for c in (mod.compressor.compressor_k, mod.compressor.compressor_v) for t in (c.weight, c.bias)]
    gate = [t.detach().float().cpu() for t in (mod.gating.weight, mod.gating.bias)]
    for i in [*range(8), *range(152, 160)]:
        s, c = slice(cu[i], cu[i + 1]), slice(cu_c[i], cu_c[i + 1])
        ref, _ = O.nsa_decode_row(q[i], k[s], v[s], *weights, *gate, n_sel=16, window=512, ck=ck[c].cpu(), cv=cv[c].cpu())
        _close("decode row %d of 160 (%d keys)" % (i, lens[i]), o[i], ref, atol=3e-2)   # (as for the rows of small batches)

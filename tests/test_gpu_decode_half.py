"""Decode with two CTAs of three warps per SM (more items than SMs) and with one of six: every sum is the same six chains in
either, so the blocks and the outputs are the same bit for bit.  Batches on both sides of the rule that chooses between them."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


# items (sequences x KV heads): 148 SMs; two CTAs per SM from 149 items on, but below 296 only up to 12 K (22 K with 295) keys, and up
# to 444 only where lengths differ
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

"""Decode with two CTAs of three warps per SM (more items than SMs) and with one of six: the soft-max statistics are six chains in
either, so the blocks are the same bit for bit.  Batches on both sides of the rule that chooses between them."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


# items (sequences x KV heads): 148 SMs; two CTAs per SM from 149 items on, but below 296 only up to some 12 K keys, and up to 444 only
# where lengths differ
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

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

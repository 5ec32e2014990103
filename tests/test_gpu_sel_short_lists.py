"""The key-major selected forward where a CTA has one to four batches of eight tokens: its drain warps pass from one staging tile to the
other before any hand-over between them, and every row of every tile has to be there when the tile is stored."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,NB,Hkv,G", [(4, 111, 2, 16), (1, 5, 1, 16), (2, 111, 4, 32)])   # a list per CTA; shared lists; two head groups
def test_short_lists(B, NB, Hkv, G):
    import nsa_b200
    gen = torch.Generator(device=DEV).manual_seed(NB + G)
    T, D = 64 * NB - 3, 128
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    q, k, v, g = rnd(B, T, Hkv * G, D), rnd(B, T, Hkv, D), rnd(B, T, Hkv, D), rnd(B, T, Hkv * G).sigmoid()
    # block b is selected by this many of its own tokens: 0 to 4 batches, whole ones and remainders
    count = torch.tensor([1, 7, 8, 9, 15, 16, 17, 23, 24, 25, 32, 0], device=DEV)
    t = torch.arange(T, device=DEV)
    blk = t // 64
    idx = torch.where(63 - t % 64 < count[(blk + 5) % 12], blk, -1)   # (the last tokens of a block: up to all of its keys are visible)
    with torch.no_grad():
        o = nsa_b200.selection_attention(q, k, v, g, g, idx.view(1, T, 1, 1).expand(B, T, Hkv, 1).contiguous())
        for _ in range(10):
            assert torch.equal(o, nsa_b200.selection_attention(q, k, v, g, g, idx.view(1, T, 1, 1).expand(B, T, Hkv, 1).contiguous()))
    nsa_b200._lib.device_status()
    pad = lambda x: torch.nn.functional.pad(x.float(), (0, 0, 0, 3))
    key = torch.arange(64, device=DEV) + 64 * blk[:, None]
    for b in range(B):
        for h in range(Hkv):
            kb, vb = (pad(x[b, :, h]).view(NB, 64, D)[blk] for x in (k, v))      # [T, 64, D]
            s = torch.einsum("tgd,tkd->tgk", q[b, :, h * G:(h + 1) * G].float(), kb) * D ** -0.5
            p = s.masked_fill((key > t[:, None])[:, None], float("-inf")).softmax(-1)
            ref = torch.einsum("tgk,tkd->tgd", p, vb) * g[b, :, h * G:(h + 1) * G].float()[..., None] * (idx >= 0)[:, None, None]
            _close("short lists %d %d" % (b, h), o[b, :, h * G:(h + 1) * G], ref)

"""The key-major selected forward where the first block's list has shares of its own (many blocks in all, more than twice as many as a
token selects): every batch gets the bits that it gets alone, where all lists are shared otherwise."""
import pytest
import torch

from parity_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,Hkv,G,S", [(4, 3584, 4, 16, 4), (5, 3001, 4, 16, 3), (2, 3600, 8, 32, 2), (4, 3584, 4, 16, 28)])
def test_shares_of_the_first_block(B, T, Hkv, G, S):
    import nsa_b200
    gen = torch.Generator(device=DEV).manual_seed(T + S)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    q, k, v, g = rnd(B, T, Hkv * G, 128), rnd(B, T, Hkv, 128), rnd(B, T, Hkv, 128), rnd(B, T, Hkv * G).sigmoid()
    # distinct blocks per token, future ones among them; the first one always, but in the last head of the last batch never
    order = torch.rand(B, T, Hkv, (T + 63) // 64, generator=gen, device=DEV)
    order[..., 0] = 2.0
    order[-1, :, -1, 0] = -1.0
    idx = order.topk(S, dim=-1).indices
    with torch.no_grad():
        both = nsa_b200.selection_attention(q, k, v, g, g, idx)
        for b in range(B):
            alone = nsa_b200.selection_attention(q[b:b + 1], k[b:b + 1], v[b:b + 1], g[b:b + 1], g[b:b + 1], idx[b:b + 1])
            assert torch.equal(both[b:b + 1], alone)
    nsa_b200._lib.device_status()

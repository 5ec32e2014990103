"""Selection scores of the tcgen05 kernel against fp32 torch at lengths of several tiles of 128 compressed keys, with more
items of 16 tokens x 16 heads than SMs, so that a CTA uses its score vectors again."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("score_mode", [0, 1])
@pytest.mark.parametrize("B,T", [(1, 2064), (1, 4200), (2, 8200)])
def test_pooled_scores_and_indices(score_mode, B, T):
    from nsa_b200 import _lib
    Hq, Hkv, D, block, stride, n = 32, 2, 128, 32, 16, 16
    Tc = (T - block) // stride + 1
    gen = torch.Generator(device=DEV).manual_seed(T)
    q, ck, cv = (torch.randn(B, *s, D, generator=gen, device=DEV).bfloat16() for s in ((T, Hq), (Tc, Hkv), (Tc, Hkv)))
    L, P = _lib.lib(), _lib.ptr
    n_pool = L.nsa_pool_out_len(Tc, 5, 4, 0)
    o, lse = torch.empty_like(q), torch.empty(B, T, Hq, device=DEV)
    idx = torch.empty(B, T, Hkv, n, dtype=torch.int32, device=DEV)
    scores = torch.empty(B, Hkv, T, n_pool, device=DEV)
    _lib.check(L.nsa_cmp_attn_fwd_gated(P(q), P(ck), P(cv), P(o), P(lse), P(idx), P(scores), None, None, None, None, None, B, T, Tc,
                                        Hq, Hkv, D, block, stride, 1, D ** -0.5, n, 5, 4, 0, score_mode, T, 0, _lib.stream()),
               "nsa_cmp_attn_fwd_gated")
    hidden = torch.arange(Tc, device=DEV)[None] * stride + block > torch.arange(T, device=DEV)[:, None]
    scale = D ** -0.5 if score_mode else 1.0
    for b in range(B):
        for h in range(Hkv):
            s = torch.einsum("thd,sd->hts", q[b, :, 16 * h:16 * h + 16].float(), ck[b, :, h].float()) * scale
            if score_mode:
                s = s.masked_fill(hidden, float("-inf"))
            p = torch.softmax(s, -1).nan_to_num(0.0).sum(0)      # (a row that sees nothing scores 0)
            ref = torch.nn.functional.avg_pool1d(p, 5, 4, 0, ceil_mode=True)
            _close("pooled scores, mode %d, T=%d" % (score_mode, T), scores[b, h], ref, atol=2e-3, rtol=1e-2)
            # the indices follow from the kernel's own scores: highest first, ties to the lower block
            want = torch.argsort(scores[b, h], dim=-1, descending=True, stable=True)[:, :n]
            assert torch.equal(idx[b, :, h].long(), want)
    _lib.device_status()

"""The tcgen05 kernels of the dense branches' backward (sliding window, compressed) against fp32 torch autograd on the same
bf16 inputs: sequences shorter than a tile of 8 tokens and around its edges, windows shorter and longer than the sequence and
than a tile of 128 keys, tokens that see no compressed position, accumulation."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    import nsa_b200
    yield nsa_b200
    nsa_b200._lib.device_status()


def _attend(q, k, v, mask, scale):
    """fp32; q [B,T,Hq,D], k, v [B,L,Hk,D], mask [T,L]: output and lse, 0 and -inf where no key is visible."""
    g = q.shape[2] // k.shape[2]
    s = torch.einsum("bthd,blhd->bthl", q, k.repeat_interleave(g, 2)) * scale
    s = s.masked_fill(~mask[:, None], float("-inf"))
    lse = torch.logsumexp(s, -1)
    p = torch.exp(s - lse.masked_fill(lse == float("-inf"), 0.0)[..., None])
    return torch.einsum("bthl,blhd->bthd", p, v.repeat_interleave(g, 2)), lse


@pytest.mark.parametrize("B,T,Hq,Hk,D,window", [(1, 1, 16, 1, 128, 512), (2, 7, 32, 1, 64, 3), (1, 129, 64, 4, 128, 128),
                                                 (2, 333, 16, 1, 64, 100), (1, 1100, 32, 2, 128, 512), (3, 257, 16, 1, 128, 1000),
                                                 (1, 4100, 32, 1, 128, 200)])
def test_dense_backward(nsa, B, T, Hq, Hk, D, window):
    L, P = nsa._lib.lib(), lambda t: t.data_ptr()
    gen = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    block, stride, scale = 32, 16, D ** -0.5
    Tc = max((T - block) // stride + 1, 1)
    q, do, g, k, v, ck, cv = rnd(B, T, Hq, D), rnd(B, T, Hq, D), rnd(B, T, Hq), *(rnd(B, T, Hk, D) for _ in range(2)), *(
        rnd(B, Tc, Hk, D) for _ in range(2))
    t, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
    masks = ((j <= t) & (j > t - window), t >= torch.arange(Tc, device=DEV)[None] * stride + block)
    want, lse, delta = [], [], []
    for (kk, vv), mask in zip(((k, v), (ck, cv)), masks):
        leaf = [x.float().requires_grad_(True) for x in (q, kk, vv)]
        o, l = _attend(*leaf, mask, scale)
        want.append(torch.autograd.grad(o, leaf, do.float() * g.float()[..., None]))
        lse.append(l.detach().contiguous())
        delta.append((g.float() * (o.detach() * do.float()).sum(-1)).contiguous())
    dq_w, dq_c, both, dk, dv, dck, dcv = (torch.empty_like(x) for x in (q, q, q, k, v, ck, cv))
    nws = L.nsa_cmp_attn_bwd_workspace_bytes(B, T, Tc, Hk, D)
    ws = torch.full((nws,), 0x7f, dtype=torch.uint8, device=DEV)
    opt = lambda *ts: [P(x) if x is not None else None for x in ts]
    win = lambda dq, acc, dk, dv: L.nsa_sel_swa_bwd(
        P(q), P(k), P(v), None, 0, None, None, None, None, None, P(do), P(lse[0]), P(delta[0]), P(g), P(dq), acc, *opt(dk, dv),
        None, 0, B, T, Hq, Hk, D, 16, 64, window, scale, None)
    cmp = lambda dq, acc, dk, dv: L.nsa_cmp_attn_bwd(
        P(q), P(ck), P(cv), P(lse[1]), P(do), P(delta[1]), P(g), P(dq), acc, *opt(dk, dv), P(ws), nws, B, T, Tc, Hq, Hk, D, block,
        stride, 1, scale, None)
    for rc in (win(dq_w, 0, dk, dv), cmp(dq_c, 0, dck, dcv), win(both, 0, None, None), cmp(both, 1, None, None)):
        nsa._lib.check(rc, "dense backward")
    _close("dq window", dq_w, want[0][0])
    _close("dq compressed", dq_c, want[1][0])
    _close("dq accumulated", both, want[0][0] + want[1][0])
    for name, x, ref in (("dk", dk, want[0][1]), ("dv", dv, want[0][2]), ("dck", dck, want[1][1]), ("dcv", dcv, want[1][2])):
        _close(name, x, ref, scaled=True)
    nsa._lib.device_status()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_sequence_keeps_its_nan_to_itself(nsa, D, bad):
    """NaN or infinity in dO or q of the second sequence: the first one's gradients are the same bits as without (its last tile of 8 tokens
    reaches into the second)."""
    gen = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    T, H = 1037, 16
    mod = nsa.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    q, k, v, do = rnd(2 * T, H, D), rnd(2 * T, 1, D), rnd(2 * T, 1, D), rnd(2 * T, H, D)
    cu = torch.tensor([0, T, 2 * T], dtype=torch.int32, device=DEV)

    def grads(q, do):
        leaf = [x.clone().requires_grad_(True) for x in (q, k, v)]
        return [g[:T] for g in torch.autograd.grad(mod(*leaf, cu, T), leaf, do)]

    want = grads(q, do)
    for i in range(2):
        x = [q.clone(), do.clone()]
        x[i][T + 2, 0, 3] = bad
        assert all(torch.equal(a, b) for a, b in zip(grads(*x), want)), ("q", "do")[i]

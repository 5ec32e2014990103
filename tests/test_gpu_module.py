"""NSAAttention as a whole: precision of its gradients against fp64."""
import pytest
import torch

from parity_util import DEV

pytestmark = pytest.mark.gpu


def _attend64(q, k, v, mask):
    """fp64 attention of one sequence, q [T,H,D], k, v [S,Hk,D], mask [T,S]; rows that see nothing give 0."""
    g = q.shape[1] // k.shape[1]
    s = torch.einsum("thd,shd->hts", q, k.repeat_interleave(g, 1)) * q.shape[2] ** -0.5
    live = mask.any(-1, keepdim=True)
    p = torch.softmax(torch.where(live, s.masked_fill(~mask, float("-inf")), torch.zeros_like(s)), -1) * live
    return torch.einsum("hts,shd->thd", p, v.repeat_interleave(g, 1))


def test_dq_is_rounded_once_where_the_selected_branch_is_small():
    """Constant gates 1/16 (selected), 1, 1: dq is the window's and the compressed branch's but for a sixteenth, so its error is that of
    one rounding to bf16 (1.66e-3 of its norm: 2^-8 / sqrt(12) averaged over a binade) and of dS in bf16, 1.85e-3 alone (the window by
    itself, 2.48e-3 with the rounding).  Another rounding at full size makes it 3.0e-3.  (head_dim 64, where the selected branch's dQ is a
    kernel of its own.)"""
    import nsa_b200
    T, H, D = 1024, 16, 64
    gen = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa_b200.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16)
    with torch.no_grad():
        for p in mod.compressor.parameters():
            p.normal_(0.0, 0.02, generator=gen)
        mod.gating.weight.zero_()
        mod.gating.bias.copy_(torch.tensor([1 / 16, 1.0, 1.0]))
    q, k, v, do = rnd(T, H, D).requires_grad_(True), rnd(T, 1, D), rnd(T, 1, D), rnd(T, H, D)
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    dq, = torch.autograd.grad(mod(q, k, v, cu, T), q, do)
    ck, cv, _ = mod.compressor(k, v, cu, None)
    x = [a.detach().double() for a in (q, k, v, ck[0], cv[0])]
    x[0].requires_grad_(True)
    t, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
    seen = t >= 16 * torch.arange(ck.shape[1], device=DEV)[None] + 32
    # 16 of 16 blocks are selected: that branch is causal attention over everything
    o = _attend64(x[0], x[1], x[2], j <= t) / 16 + _attend64(x[0], x[1], x[2], (j <= t) & (j > t - 512)) + _attend64(x[0], x[3], x[4], seen)
    want, = torch.autograd.grad(o, x[0], do.double())
    err = float((dq.double() - want).norm() / want.norm())
    assert err < 2.7e-3, "relative error %.2e" % err


def test_shapes_that_do_not_fit_are_refused():
    """A module of another head_dim, keys of another head_dim: an error on the host."""
    import nsa_b200
    cu = torch.tensor([0, 1024], dtype=torch.int32, device=DEV)
    x = {(h, d): torch.zeros(1024, h, d, device=DEV, dtype=torch.bfloat16) for h in (1, 16) for d in (64, 128)}
    for D in (64, 128):
        mod = nsa_b200.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16)
        for q, k in ((x[16, 192 - D], x[1, 192 - D]), (x[16, D], x[1, 192 - D]), (x[16, 192 - D], x[1, D])):
            with pytest.raises(RuntimeError, match="does not fit"):
                mod(q, k, k, cu, 1024)


class _Scaled(torch.nn.Module):
    """A stand-in for the compressor that doubles the compressed values."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, k, v, cu, group=None):
        ck, cv, cu = self.inner(k, v, cu, group)
        return ck, 2 * cv, cu


@pytest.mark.parametrize("mode", ["reference", "causal"])
@pytest.mark.parametrize("lens", [(1100, 1100), (1100, 1037)])
def test_the_compressor_is_called_where_that_shows(lens, mode):
    """Forward hooks on it run (and give the same results as without), a substitute is used: twice the compressed values with half their
    gate is the module itself."""
    import nsa_b200
    D, H, n = 128, 32, sum(lens)
    gen = torch.Generator(device=DEV).manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa_b200.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16)
    mod.score_mode = mode
    with torch.no_grad():
        for p in mod.parameters():
            p.normal_(0.0, 0.05, generator=gen)
    q, k, v, do = rnd(n, H, D).requires_grad_(True), rnd(n, 2, D).requires_grad_(True), rnd(n, 2, D).requires_grad_(True), rnd(n, H, D)
    cu = torch.tensor([0, lens[0], n], dtype=torch.int32, device=DEV)

    def run():
        o = mod(q, k, v, cu)
        return [o, *torch.autograd.grad(o, [q, k, v, *mod.parameters()], do)]

    plain = run()
    seen = []
    handle = mod.compressor.register_forward_hook(lambda m, args, out: seen.append(tuple(out[0].shape)))
    hooked = run()
    handle.remove()
    assert seen == ([(2, 67, 2, D)] if lens[0] == lens[1] else [(1, 67, 2, D), (1, 63, 2, D)])
    names = ["o", "dq", "dk", "dv"] + [name for name, _ in mod.named_parameters()]
    for name, a, b in zip(names, hooked, plain):
        if name != "compressor.compressor_k.bias":   # zero but for roundings
            # both round to bf16 on the way, the composed form up to twice as often: 2e-3 apart, the gates' bias (a sum that nearly cancels) 2e-2
            assert float((a - b).detach().float().norm() / b.detach().float().norm()) < (3e-2 if name == "gating.bias" else 8e-3), name
    mod.compressor = _Scaled(mod.compressor)
    with torch.no_grad():
        mod.gating.weight[2] /= 2
        mod.gating.bias[2] /= 2
    doubled = run()
    assert float((doubled[0] - plain[0]).detach().float().norm() / plain[0].detach().float().norm()) < 8e-3


@pytest.mark.parametrize("D", [64, 128])
def test_a_forward_without_gradients_does_no_work_for_a_backward(D):
    """Under no_grad a module (and gates) with trainable parameters launch the same kernels, take the same memory and give the same bits
    as frozen ones."""
    import nsa_b200
    T, H = 2048, 32
    gen = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa_b200.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16)
    q, k, v, cu = rnd(T, H, D), rnd(T, 2, D), rnd(T, 2, D), torch.tensor([0, T], dtype=torch.int32, device=DEV)
    g = rnd(1, T, H).sigmoid()
    idx = torch.arange(16, device=DEV).expand(1, T, 2, 16).contiguous()
    calls = (lambda: mod(q, k, v, cu, T),
             lambda: nsa_b200.selection_attention(q[None], k[None], v[None], g, g, idx, window_size=128))

    def measure(call):
        launches = nsa_b200._lib.lib().nsa_kernel_launch_count()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        with torch.no_grad():
            o = call()
        return nsa_b200._lib.lib().nsa_kernel_launch_count() - launches, torch.cuda.max_memory_allocated() - before, o

    for call in calls:
        res = []
        for train in (True, False):
            mod.requires_grad_(train)
            g.requires_grad_(train)
            res.append(measure(call))
        assert res[0][:2] == res[1][:2] and torch.equal(res[0][2], res[1][2])
        mod.requires_grad_(True)
        g.requires_grad_(True)
        assert torch.equal(call().detach(), res[0][2])


def _odd(x):
    """x at an address two bytes behind a 16-byte boundary, as a piece of a flat buffer of parameters may be."""
    y = torch.empty(x.numel() + 8, dtype=x.dtype, device=x.device)[1:x.numel() + 1].view(x.shape)
    return y.copy_(x)


def test_gates_and_their_weights_at_any_address():
    import nsa_b200
    from nsa_b200.decode import compress_cache, nsa_decode
    gen = torch.Generator(device=DEV).manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    # the gates of selection_attention, at the head_dim whose backward copies them in pieces of 32 bytes
    q, k, v, do = rnd(1, 300, 16, 64).requires_grad_(True), rnd(1, 300, 1, 64), rnd(1, 300, 1, 64), rnd(1, 300, 16, 64)
    idx = torch.tensor([0, 2, 4], device=DEV).expand(1, 300, 1, 3).contiguous()
    g = rnd(1, 300, 16)
    res = []
    for gates in (g, _odd(g)):
        gates = gates.detach().requires_grad_(True)
        o = nsa_b200.selection_attention(q, k, v, gates, gates, idx, window_size=100)
        res.append([o.detach(), *torch.autograd.grad(o, [q, gates], do)])
    assert all(torch.equal(a, b) for a, b in zip(*res))
    # the module's weights: gates, and the compression's (element by element)
    mod = nsa_b200.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    q, k, v = rnd(1100, 16, 128), rnd(1100, 1, 128), rnd(1100, 1, 128)
    cu = torch.tensor([0, 1100], dtype=torch.int32, device=DEV)
    res = []
    for move in (lambda x: x, _odd):
        for p in mod.parameters():
            p.data = move(p.data)
        cache = compress_cache(mod, k, v, [0, 1100])
        res.append([mod(q, k, v, cu, 1100), cache.ck, cache.cv, nsa_decode(mod, q[-1:], k, v, [0, 1100], cache)])
    assert mod.gating.weight.data_ptr() % 16 == 2 and all(torch.equal(a, b) for a, b in zip(*res))


def test_compression_biases_at_any_address():
    """Also where the contraction is split, which reads four of them at a time."""
    from nsa_b200.compression_kv import _CompressPair
    gen = torch.Generator(device=DEV).manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    k, v, w, b = rnd(64, 1, 128), rnd(64, 1, 128), rnd(4096, 128), rnd(128)
    with torch.no_grad():
        for split in (True, False):
            want, got = (_CompressPair.apply(k, v, w, w, bias, bias, [0, 64], [0, 3], 32, 16, split) for bias in (b, _odd(b)))
            assert torch.equal(want[0], got[0]) and torch.equal(want[1], got[1])


def test_queries_of_the_first_tokens_alone():
    """q may hold the first tokens of every (equally long) sequence: their rows of the whole result."""
    import nsa_b200
    T, Tq, H, D = 1100, 700, 32, 128
    gen = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa_b200.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    q, k, v = rnd(2, T, H, D), rnd(2 * T, 2, D), rnd(2 * T, 2, D)
    cu = torch.tensor([0, T, 2 * T], dtype=torch.int32, device=DEV)
    whole = mod(q.reshape(2 * T, H, D), k, v, cu, T).view(2, T, H, D)
    part = mod(q[:, :Tq].reshape(2 * Tq, H, D), k, v, cu, T).view(2, Tq, H, D)
    assert torch.equal(part, whole[:, :Tq])
    for bad in (q.reshape(2 * T, H, D)[:-1], torch.cat([q, q[:, :2]], 1).reshape(-1, H, D)):
        with pytest.raises((ValueError, RuntimeError)):
            mod(bad, k, v, cu, T)


@pytest.mark.parametrize("block", [32, 48])   # the tcgen05 backward of the compression and the other one
@pytest.mark.parametrize("without", [("k",), ("v",), ("k", "v")])
def test_biases_of_the_compression_are_independent(without, block):
    """A compressor with one bias only: the other's gradient is that of a module whose missing bias is zero."""
    import nsa_b200
    T, H, D = 1100, 16, 64
    gen = torch.Generator(device=DEV).manual_seed(block)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa_b200.NSAAttention(D, True, compression_block=block, selected_block_count=8, device=DEV, dtype=torch.bfloat16)
    conv = dict(k=mod.compressor.compressor_k, v=mod.compressor.compressor_v)
    with torch.no_grad():
        for name in without:
            conv[name].bias.zero_()
    q, k, v, do = rnd(T, H, D), rnd(T, 1, D), rnd(T, 1, D), rnd(T, H, D)
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    grads = lambda: dict(zip([n for n, _ in mod.named_parameters()], torch.autograd.grad(mod(q, k, v, cu, T), list(mod.parameters()), do)))
    want = grads()
    for name in without:
        conv[name].bias = None
    got = grads()
    assert len(got) == 6 - len(without) and all(torch.equal(g, want[n]) for n, g in got.items())

"""The kernels wait for the one before them themselves (programmatic dependent launch): the same chains captured in a CUDA graph and
replayed on new inputs, which overwrite the ones before while nothing else separates the steps."""
import pytest
import torch

from parity_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["prefill", "select", "decode", "generate"])
def test_captured_steps_equal_eager_ones(kind):
    import nsa_b200 as nsa
    from nsa_b200.decode import compress_cache, extend_compress_cache, nsa_decode
    torch.manual_seed(0)
    gen = torch.Generator(device=DEV).manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    T, H = 1500, 2
    if kind in ("prefill", "select"):
        q, k, v = rnd(T, 16 * H, 128), rnd(T, H, 128), rnd(T, H, 128)
        cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
        own = (torch.arange(T, device=DEV) // 64).view(1, T, 1, 1)
        idx = (own - torch.arange(4, device=DEV).view(1, 1, 1, 4)).expand(1, T, H, 4).contiguous()   # (before the first: skipped)
        g = rnd(1, T, 16 * H)
        step = (lambda: mod(q, k, v, cu, T)) if kind == "prefill" else (lambda: nsa.selection_attention(q[None], k[None], v[None], g, g, idx))
    else:
        lens = [2000, 700, 33, 1300]
        cu = [sum(lens[:i]) for i in range(5)]
        q, k, v = rnd(4, 16 * H, 128), rnd(cu[-1], H, 128), rnd(cu[-1], H, 128)
        keep = torch.ones(cu[-1], dtype=torch.bool, device=DEV)
        keep[torch.tensor(cu[1:], device=DEV) - 1] = False
        cache = compress_cache(mod, k, v, cu) if kind == "decode" else compress_cache(mod, k[keep], v[keep], [c - i for i, c in enumerate(cu)])

        def step():
            c = cache if kind == "decode" else extend_compress_cache(mod, cache, k, v, cu)
            return nsa_decode(mod, q, k, v, cu, c)
    with torch.no_grad():
        for _ in range(2):
            step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = step()
        got, want = [], []
        news = [rnd(*q.shape) for _ in range(4)]
        for x in news:
            q.copy_(x)
            graph.replay()
            got.append(out.clone())
        for x in news:
            q.copy_(x)
            want.append(step().clone())
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    nsa._lib.device_status()


@pytest.mark.parametrize("kind", ["module", "module64", "select", "compressed", "compress"])
def test_captured_training_steps_equal_eager_ones(kind):
    """Forward and backward, every gradient: captured and replayed on new inputs, and eager on a stream of their own."""
    import nsa_b200 as nsa
    from nsa_b200.compression_kv import KVCompressorVarlen
    from nsa_b200.triton_attention import flash_attn_func
    torch.manual_seed(1)
    gen = torch.Generator(device=DEV).manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    D, H, T = 64 if kind == "module64" else 128, 2, 1500
    leaf = lambda *s: rnd(*s).requires_grad_(True)
    if kind in ("module", "module64"):
        mod = nsa.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16)
        cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
        inputs, params, douts = [leaf(T, 16 * H, D), leaf(T, H, D), leaf(T, H, D)], list(mod.parameters()), [rnd(T, 16 * H, D)]
        forward = lambda: [mod(*inputs, cu, T)]
    elif kind == "select":
        own = (torch.arange(T, device=DEV) // 64).view(1, T, 1, 1)
        idx = (own - torch.arange(4, device=DEV).view(1, 1, 1, 4)).expand(1, T, H, 4).contiguous()
        inputs, params, douts = [leaf(1, T, 16 * H, D), leaf(1, T, H, D), leaf(1, T, H, D), leaf(1, T, 16 * H), leaf(1, T, 16 * H)], [], [rnd(1, T, 16 * H, D)]
        forward = lambda: [nsa.selection_attention(*inputs, idx, None, 64, 100)]
    elif kind == "compressed":
        Tc = (T - 32) // 16 + 1
        inputs, params, douts = [leaf(1, T, 16 * H, D), leaf(1, Tc, H, D), leaf(1, Tc, H, D)], [], [rnd(1, T, 16 * H, D)]
        forward = lambda: [flash_attn_func(*inputs, 16, 32, True, None, H, 5, 4, 0, 8)[0]]
    else:
        lens = [700, 33, 767]
        cu = [0, 700, 733, T]
        comp = KVCompressorVarlen(16, 32, D, DEV, torch.bfloat16)
        outs = sum((n - 32) // 16 for n in lens)
        inputs, params, douts = [leaf(T, H, D), leaf(T, H, D)], list(comp.parameters()), [rnd(outs, H, D), rnd(outs, H, D)]
        forward = lambda: list(comp(*inputs, cu)[:2])

    def step():
        outs = forward()
        return [*outs, *torch.autograd.grad(outs, inputs + params, douts)]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = step()
    news = [[rnd(*x.shape) for x in inputs + douts] for _ in range(3)]

    def load(new):
        with torch.no_grad():
            for x, y in zip(inputs + douts, new):
                x.copy_(y)

    got, want = [], []
    for new in news:
        load(new)
        graph.replay()
        got.append([x.clone() for x in out])
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for new in news:
            load(new)
            want.append([x.clone() for x in step()])
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))
    nsa._lib.device_status()

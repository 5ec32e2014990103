"""The tcgen05 compression GEMMs (forward and backward, both tensors per launch) against fp32 torch on the same bf16
inputs, at the edges of their tiles: 128-row tiles of (positions x heads), sequences that start off the stride grid, tails,
sequences without a position, head counts that do not divide the tile, one to many splits."""
import pytest
import torch

from parity_util import DEV, close as _close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    import nsa_b200
    yield nsa_b200
    nsa_b200._lib.device_status()


def _ref(x, w, b, cu, block, stride, n_out):
    """fp32, one sequence after the other: windows unfolded, one matmul."""
    outs = []
    for i, n in enumerate(n_out):
        s = x[cu[i]:cu[i + 1]]
        if n:
            win = torch.stack([s[j * stride:j * stride + block] for j in range(n)])          # [n, l, H, D]
            outs.append(torch.einsum("nlhd,lde->nhe", win, w.view(block, x.shape[-1], -1)) + (0 if b is None else b))
    return torch.cat(outs)


@pytest.mark.parametrize("D,H,block,stride,lens", [
    (128, 4, 32, 16, [5003]), (128, 4, 32, 16, [33, 1000, 31, 48, 2001, 700]), (128, 1, 32, 16, [2111, 2049]),
    (128, 3, 32, 16, [700, 45]), (64, 4, 32, 16, [1024, 1037]), (64, 2, 64, 32, [3000, 65, 64]), (128, 4, 16, 16, [640, 17]),
    (128, 4, 64, 16, [900, 77])])
@pytest.mark.parametrize("split", [True, False])
def test_compress_pair_fwd_bwd(nsa, D, H, block, stride, lens, split):
    gen = torch.Generator(device=DEV).manual_seed(D + H + len(lens))
    rnd = lambda *s, m=1.0: (torch.randn(*s, generator=gen, device=DEV) * m).bfloat16()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    n_out = [(n - block) // stride + 1 if n >= block else 0 for n in lens]
    cu_out = [sum(n_out[:i]) for i in range(len(n_out) + 1)]
    args = [rnd(cu[-1], H, D), rnd(cu[-1], H, D), rnd(block * D, D, m=0.03), rnd(block * D, D, m=0.03), rnd(D), rnd(D)]
    dck, dcv = rnd(cu_out[-1], H, D), rnd(cu_out[-1], H, D)
    ours = [a.clone().requires_grad_(True) for a in args]
    ck, cv = nsa.compression_kv._CompressPair.apply(*ours, cu, cu_out, block, stride, split)
    got = torch.autograd.grad([ck, cv], ours, [dck, dcv])
    ref = [a.float().requires_grad_(True) for a in args]
    rk, rv = _ref(ref[0], ref[2], ref[4], cu, block, stride, n_out), _ref(ref[1], ref[3], ref[5], cu, block, stride, n_out)
    want = torch.autograd.grad([rk, rv], ref, [dck.float(), dcv.float()])
    _close("ck", ck, rk)
    _close("cv", cv, rv)
    for name, g, w in zip(("dk", "dv", "dw_k", "dw_v", "db_k", "db_v"), got, want):
        _close(name, g, w, scaled=name[:2] != "dk" and name[:2] != "dv")
    nsa._lib.device_status()


@pytest.mark.parametrize("D,H,lens", [(128, 4, [13007, 12999, 12100]), (128, 4, [15001, 16010]), (64, 4, [13007, 12999, 12100]),
                                      (128, 130, [640, 523])])
def test_forward_tile_of_a_call_keeps_the_bits(nsa, D, H, lens):
    """Few rows: half of the columns per CTA; a little more than one CTA per SM: two row tiles; else one.  A sequence gets the same
    bits from the tile that it gets alone and from the packed call's."""
    gen = torch.Generator(device=DEV).manual_seed(D + H)
    rnd = lambda *s, m=1.0: (torch.randn(*s, generator=gen, device=DEV) * m).bfloat16()
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    n_out = [(n - 32) // 16 + 1 for n in lens]
    cu_out = [sum(n_out[:i]) for i in range(len(n_out) + 1)]
    k, v, w_k, w_v, b = rnd(cu[-1], H, D), rnd(cu[-1], H, D), rnd(32 * D, D, m=0.03), rnd(32 * D, D, m=0.03), rnd(D)
    run = lambda i, j: nsa.compression_kv._CompressPair.apply(k[cu[i]:cu[j]], v[cu[i]:cu[j]], w_k, w_v, b, b, [c - cu[i] for c in cu[i:j + 1]],
                                                              [c - cu_out[i] for c in cu_out[i:j + 1]], 32, 16, False)
    packed = run(0, len(lens))
    for i in range(len(lens)):
        for alone, both in zip(run(i, i + 1), packed):
            assert torch.equal(alone, both[cu_out[i]:cu_out[i + 1]])
    _close("ck", packed[0][:n_out[0]], _ref(k[:lens[0]].float(), w_k.float(), b.float(), [0, lens[0]], 32, 16, n_out[:1]))
    nsa._lib.device_status()


@pytest.mark.parametrize("D,block,stride", [(128, 32, 16), (64, 64, 32)])
def test_conv_weight_layout(nsa, D, block, stride):
    w = torch.randn(D, D, block, device=DEV).bfloat16().requires_grad_(True)
    a, b = nsa.compression_kv._ConvLayout.apply(w, w)
    assert torch.equal(a, w.permute(2, 1, 0).reshape(block * D, D)) and torch.equal(a, b)


@pytest.mark.parametrize("grow", [[1] * 5, [0, 16, 3, 700, 40]])
def test_extended_cache_equals_a_new_one(nsa, grow):
    from nsa_b200.decode import compress_cache, extend_compress_cache
    old = [2048, 1000, 20, 47, 31]
    new = [a + b for a, b in zip(old, grow)]
    mod = nsa.NSAAttention(128, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    k, v = (torch.randn(sum(new), 4, 128, device=DEV).bfloat16() for _ in range(2))
    keep = torch.cat([torch.arange(n, device=DEV) < o for n, o in zip(new, old)])
    cum = lambda ls: [sum(ls[:i]) for i in range(len(ls) + 1)]
    before = compress_cache(mod, k[keep], v[keep], cum(old))
    got, want = extend_compress_cache(mod, before, k, v, cum(new)), compress_cache(mod, k, v, cum(new))
    assert got.cu == want.cu and got.cu_c == want.cu_c and torch.equal(got.table_dev[:12], want.table_dev[:12])
    _close("extended ck", got.ck, want.ck)
    _close("extended cv", got.cv, want.cv)
    with pytest.raises(ValueError):
        extend_compress_cache(mod, want, k, v, cum([n - 1 for n in new]))
    nsa._lib.device_status()


@pytest.mark.parametrize("block,stride", [(32, 16), (64, 16)])   # the tcgen05 backward and the other one
def test_an_unused_output_gives_no_gradient(nsa, block, stride):
    """Gradients of the used output alone are those of both, the other tensor's are None."""
    gen = torch.Generator(device=DEV).manual_seed(1)
    comp = nsa.compression_kv.KVCompressorVarlen(stride, block, 128, DEV, torch.bfloat16)
    k, v = (torch.randn(500, 2, 128, generator=gen, device=DEV).bfloat16().requires_grad_(True) for _ in range(2))
    leaves = [k, v, comp.k_weight, comp.v_weight]
    ck, cv, _ = comp(k, v, [0, 300, 500])
    dck, dcv = (torch.randn(ck.shape, generator=gen, device=DEV).bfloat16() for _ in range(2))
    both = torch.autograd.grad([ck, cv], leaves, [dck, dcv], retain_graph=True)
    for out, dy, mine in ((ck, dck, (0, 2)), (cv, dcv, (1, 3))):
        got = torch.autograd.grad(out, leaves, dy, retain_graph=True, allow_unused=True)
        for i in range(4):
            assert (torch.equal(got[i], both[i]) if i in mine else got[i] is None)


def test_keys_and_values_of_different_shapes(nsa):
    """Other head counts, head_dims and lengths of the two: each is compressed as it would be beside a tensor like itself."""
    gen = torch.Generator(device=DEV).manual_seed(2)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16().requires_grad_(True)
    compress_kv, cu = nsa.compression_kv.compress_kv, [0, 300, 480]
    for v_shape in ((480, 4, 128), (500, 2, 128), (480, 2, 64)):
        k, v = rnd(480, 2, 128), rnd(*v_shape)
        w_k, w_v = (rnd(32 * x.shape[2], x.shape[2]) for x in (k, v))
        ck, cv, cu_out = compress_kv(k, v, w_k, w_v, cu, 16, 32)
        dck, dcv = rnd(*ck.shape).detach(), rnd(*cv.shape).detach()
        got = torch.autograd.grad([ck, cv], [k, v, w_k, w_v], [dck, dcv])
        for x, w, c, dc, i in ((k, w_k, ck, dck, 0), (v, w_v, cv, dcv, 1)):
            alone, _, cu_alone = compress_kv(x, x.detach(), w, w.detach(), cu, 16, 32)
            assert torch.equal(alone, c) and torch.equal(cu_alone, cu_out)
            dx, dw = torch.autograd.grad(alone, [x, w], dc)
            assert torch.equal(dx[:480], got[i][:480]) and torch.equal(dw, got[2 + i])
    comp = nsa.compression_kv.KVCompressor(16, 32, 128, DEV, torch.bfloat16)
    k, v = rnd(600, 2, 128), rnd(600, 4, 128)
    cu = torch.tensor([0, 300, 600], dtype=torch.int32)
    ck, cv, _ = comp(k, v, cu)
    assert torch.equal(ck, comp(k, k, cu)[0]) and torch.equal(cv, comp(v, v, cu)[1])


@pytest.mark.parametrize("D,H,block,stride,lens", [(128, 4, 32, 16, [33, 1000, 31, 700]), (64, 3, 64, 16, [200, 64, 1037]), (128, 1, 16, 16, [640, 17])])
def test_single_tensor_entry_point(nsa, D, H, block, stride, lens):
    """nsa_compress_fwd (mma.sync, one tensor) against nsa_compress_fwd_kv without split: one chain of the same products each, so the same
    bits."""
    gen = torch.Generator(device=DEV).manual_seed(D)
    rnd = lambda *s, m=1.0: (torch.randn(*s, generator=gen, device=DEV) * m).bfloat16()
    cum = lambda ls: [sum(ls[:i]) for i in range(len(ls) + 1)]
    n_out = [(n - block) // stride + 1 if n >= block else 0 for n in lens]
    cu, cu_out = cum(lens), cum(n_out)
    x, w, b = rnd(cu[-1], H, D), rnd(block * D, D, m=0.03), rnd(D)
    L, P = nsa._lib.lib(), nsa._lib.ptr
    cin, cout = (torch.tensor(c, dtype=torch.int32, device=DEV) for c in (cu, cu_out))
    one, pair = (torch.empty(cu_out[-1], H, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    nsa._lib.check(L.nsa_compress_fwd(P(x), P(w), P(b), P(one), P(cin), P(cout), len(lens), H, D, block, stride, max(n_out),
                                      nsa._lib.stream()), "nsa_compress_fwd")
    nsa._lib.check(L.nsa_compress_fwd_kv(P(x), P(x), P(w), P(w), P(b), P(b), P(pair), P(pair), P(cin), P(cout), len(lens), 0, 0, cu[-1],
                                         cu_out[-1], H, D, block, stride, 0, nsa._lib.stream()), "nsa_compress_fwd_kv")
    _close("nsa_compress_fwd", one, _ref(x.float(), w.float(), b.float(), cu, block, stride, n_out))
    assert torch.equal(one, pair)

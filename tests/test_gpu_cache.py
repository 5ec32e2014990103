"""The compressed cache of a generation loop (compress_cache, extend_compress_cache): its values depend on the sequence alone."""
import pytest
import torch

from parity_util import DEV

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nsa():
    import nsa_b200
    yield nsa_b200
    nsa_b200._lib.device_status()


def _cum(lens):
    return [sum(lens[:i]) for i in range(len(lens) + 1)]


def _module(nsa, gen, D=128):
    mod = nsa.NSAAttention(D, True, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    for p in mod.parameters():
        p.normal_(0.0, 0.02, generator=gen)
    return mod


@pytest.mark.parametrize("H", [1, 4])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_cache_bits_depend_on_the_sequence_alone(nsa, seed, H):
    """Built whole, extended step by step, each sequence by itself, with gradients and by the module's own compression: the same bits (the
    block selection depends on them)."""
    from nsa_b200.decode import compress_cache, extend_compress_cache
    gen = torch.Generator(device=DEV).manual_seed(seed)
    mod = _module(nsa, gen)
    lens = [2100, 4096, 33, 700, 31, 9000]
    k, v = (torch.randn(sum(lens), H, 128, generator=gen, device=DEV).bfloat16() for _ in range(2))
    cu = _cum(lens)
    whole = compress_cache(mod, k, v, cu)
    grown = None
    for cut in (1500, 40, 17, 16, 1, 0):
        part = [max(n - cut, 20) if n > 40 else n for n in lens]
        keep = torch.cat([torch.arange(n, device=DEV) < p for n, p in zip(lens, part)])
        args = (k[keep], v[keep], _cum(part))
        grown = compress_cache(mod, *args) if grown is None else extend_compress_cache(mod, grown, *args)
    assert torch.equal(grown.ck, whole.ck) and torch.equal(grown.cv, whole.cv) and grown.cu_c == whole.cu_c
    mod.requires_grad_(True)
    with_grad = compress_cache(mod, k, v, cu)
    mod.requires_grad_(False)
    assert with_grad.ck.requires_grad and torch.equal(with_grad.ck, whole.ck) and torch.equal(with_grad.cv, whole.cv)
    for i, n in enumerate(lens):
        if n < 32:
            continue
        ks, vs, rows = k[cu[i]:cu[i + 1]], v[cu[i]:cu[i + 1]], slice(whole.cu_c[i], whole.cu_c[i + 1])
        alone = compress_cache(mod, ks, vs, [0, n])
        ck, cv, _ = mod.compressor(ks, vs, torch.tensor([0, n], dtype=torch.int32), None)
        for got_k, got_v in ((alone.ck, alone.cv), (ck[0], cv[0])):
            assert torch.equal(got_k, whole.ck[rows]) and torch.equal(got_v, whole.cv[rows])


def test_cache_before_the_first_block(nsa):
    """No sequence has reached 32 tokens yet: an empty cache, that grows like any other."""
    from nsa_b200.decode import compress_cache, extend_compress_cache
    gen = torch.Generator(device=DEV).manual_seed(1)
    mod = _module(nsa, gen)
    k, v = (torch.randn(200, 2, 128, generator=gen, device=DEV).bfloat16() for _ in range(2))
    cache = compress_cache(mod, k[:0], v[:0], [0, 0, 0, 0])
    assert cache.ck.shape == (0, 2, 128) and cache.cu_c == [0, 0, 0, 0]
    for lens in ((20, 5, 31), (20, 20, 31), (20, 20, 32), (33, 48, 100)):
        n = sum(lens)
        ks, vs = torch.zeros(2, n, 2, 128, device=DEV, dtype=torch.bfloat16)
        for i in range(3):   # sequence i is the first tokens of k, v from 10 i on
            ks[_cum(lens)[i]:_cum(lens)[i + 1]], vs[_cum(lens)[i]:_cum(lens)[i + 1]] = (x[10 * i:10 * i + lens[i]] for x in (k, v))
        cache = extend_compress_cache(mod, cache, ks, vs, _cum(lens))
        want = compress_cache(mod, ks, vs, _cum(lens))
        assert cache.cu == want.cu == _cum(lens) and cache.cu_c == want.cu_c
        assert torch.equal(cache.ck, want.ck) and torch.equal(cache.cv, want.cv)
        assert torch.equal(cache.order_dev, want.order_dev)
    assert cache.cu_c == [0, 1, 3, 8]
    none = compress_cache(mod, k, v, [0])
    assert none.ck.shape == (0, 2, 128) and none.cu_c == [0]


def test_a_cache_that_does_not_fit_is_refused(nsa):
    """Other head counts, head_dims or geometries than the old cache's, weights of another head_dim: an error on the host."""
    from nsa_b200.decode import compress_cache, extend_compress_cache
    gen = torch.Generator(device=DEV).manual_seed(1)
    mod = _module(nsa, gen)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    k2, k4, k64 = rnd(100, 2, 128), rnd(101, 4, 128), rnd(101, 2, 64)
    cache = compress_cache(mod, k2, k2, [0, 100])
    with pytest.raises(RuntimeError, match="does not fit"):
        extend_compress_cache(mod, cache, k4, k4, [0, 101])
    with pytest.raises(RuntimeError, match="does not fit"):
        extend_compress_cache(mod, cache, k64, k64, [0, 101])
    with pytest.raises(RuntimeError, match="does not fit"):
        compress_cache(mod, k64, k64, [0, 101])
    small = nsa.NSAAttention(128, True, compression_block=16, device=DEV, dtype=torch.bfloat16).requires_grad_(False)
    cache16 = compress_cache(small, k2, k2, [0, 100])
    with pytest.raises(RuntimeError, match="another block or stride"):
        extend_compress_cache(mod, cache16, k2, k2, [0, 100])


def test_keys_and_values_of_different_shapes(nsa):
    """More rows of one than of the other, or other head counts: each is compressed as it would be by itself."""
    from nsa_b200.decode import compress_cache, extend_compress_cache
    gen = torch.Generator(device=DEV).manual_seed(2)
    mod = _module(nsa, gen)
    k, v = (torch.randn(500, h, 128, generator=gen, device=DEV).bfloat16() for h in (2, 4))
    cu, cu1 = [0, 300, 450], [0, 299, 380]
    keep = torch.cat([torch.arange(299), 300 + torch.arange(81)]).to(DEV)
    cache = compress_cache(mod, k, v, cu)
    grown = extend_compress_cache(mod, compress_cache(mod, k[keep], v[keep], cu1), k, v, cu)
    kk, vv = compress_cache(mod, k[:450], k[:460], cu), compress_cache(mod, v, v[:450], cu)
    for c in (cache, grown):
        assert torch.equal(c.ck, kk.ck) and torch.equal(c.cv, vv.cv)


def test_decode_with_a_cache_made_from_its_parts(nsa):
    from nsa_b200.decode import CompressedCache, compress_cache, extend_compress_cache, nsa_decode
    gen = torch.Generator(device=DEV).manual_seed(3)
    mod = _module(nsa, gen)
    cu = [0, 40, 2040, 2100]
    k, v = (torch.randn(cu[-1], 4, 128, generator=gen, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(3, 64, 128, generator=gen, device=DEV).bfloat16()
    cache = compress_cache(mod, k, v, cu)
    same = CompressedCache(*cache)
    assert torch.equal(same.order_dev, cache.order_dev) and torch.equal(same.cu_c_dev, cache.cu_c_dev)
    assert torch.equal(nsa_decode(mod, q, k, v, cu, same), nsa_decode(mod, q, k, v, cu, cache))
    assert torch.equal(extend_compress_cache(mod, same, k, v, cu).ck, cache.ck)


def test_a_cache_keeps_its_tables_alone(nsa):
    from nsa_b200.decode import compress_cache, extend_compress_cache
    mod = _module(nsa, torch.Generator(device=DEV).manual_seed(4))
    k = torch.zeros(100, 1, 128, device=DEV, dtype=torch.bfloat16)
    cache = extend_compress_cache(mod, compress_cache(mod, k, k, [0, 64]), k, k, [0, 100])
    assert cache.table_dev.untyped_storage().nbytes() == 4 * (6 * 1 + 4)   # (not the 2 MB of weights in the kernels' layout)

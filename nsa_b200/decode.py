"""Decode step of NSAAttention: one new query token per sequence against that sequence's whole K/V cache.

The reference has no decode entry point (its module assumes len(q) == len(k), nsa/nsa.py:97); this evaluates
the same forward (nsa/nsa.py:94-135) for the single row t = L-1 of every sequence of a packed batch, all sequences
in one kernel launch (nsa_decode_fwd).  The compressed K/V are a cache: ``compress_cache`` builds it once,
``extend_compress_cache`` appends only the compressed positions that new tokens complete.
"""
import ctypes

import torch

from . import _lib
from .compression_kv import _compress, _ConvLayout


class CompressedCache:
    """Compressed K/V of a packed cache plus the (host and device) length tables the decode kernel needs.

    ck, cv [sum Tc,Hkv,D]; cu, cu_c: host lists [nseq+1] (cumulative lengths of k/v and of ck/cv); the device copies and
    the longest-first launch order are one table that is built with the cache, so that a decode step issues no
    host-to-device copy.  Saving and loading keeps ck, cv, cu and cu_c and makes the table anew."""

    def __init__(self, ck, cv, cu, cu_c):
        cu, cu_c = [int(c) for c in cu], [int(c) for c in cu_c]
        n = len(cu) - 1
        lens = [cu[i + 1] - cu[i] for i in range(n)]
        order = sorted(range(n), key=lambda i: -lens[i])
        values = [*cu, *cu_c] + [0] * (3 * n + 2) + order   # (the parts in between are read while a cache is built)
        self._set(ck, cv, (ctypes.c_int32 * len(values))(*values), torch.tensor(values, dtype=torch.int32, device=ck.device), n,
                  max([cu_c[i + 1] - cu_c[i] for i in range(n)] + [0]))

    def _set(self, ck, cv, table, table_dev, nseq, max_tc):
        self.ck, self.cv, self.nseq, self.max_tc = ck, cv, nseq, max_tc
        self._table, self.table_dev = table, table_dev   # layout: nsa_cache_plan in include/nsa_b200.h
        return self

    def __getstate__(self):
        return dict(ck=self.ck, cv=self.cv, cu=self.cu, cu_c=self.cu_c)

    def __setstate__(self, state):
        self.__init__(state["ck"], state["cv"], state["cu"], state["cu_c"])

    @property
    def cu(self):
        return list(self._table[:self.nseq + 1])

    @property
    def cu_c(self):
        return list(self._table[self.nseq + 1:2 * self.nseq + 2])

    @property
    def cu_dev(self):
        return self.table_dev[:self.nseq + 1]

    @property
    def cu_c_dev(self):
        return self.table_dev[self.nseq + 1:2 * self.nseq + 2]

    @property
    def order_dev(self):
        return self.table_dev[5 * self.nseq + 4:]

    def workspace(self, nbytes):
        """Scratch of the decode kernels (per-warp partial results), kept with the cache so a step allocates nothing."""
        ws = getattr(self, "_ws", None)
        if ws is None or ws.numel() < nbytes:
            ws = self._ws = torch.empty(nbytes, dtype=torch.uint8, device=self.ck.device)
        return ws

    def __iter__(self):   # (ck, cv, cu, cu_c), the tuple earlier callers unpack
        return iter((self.ck, self.cv, self.cu, self.cu_c))


def _lengths(cu_seqlens_k):
    return _lib.int32_array(cu_seqlens_k.tolist() if torch.is_tensor(cu_seqlens_k) else cu_seqlens_k)


@torch.no_grad()
def _build(module, k, v, cu_seqlens_k, old):
    """The compressed cache of packed k, v; the positions that ``old`` (a CompressedCache or None) holds are copied."""
    k, v = _lib.require(k, "k"), _lib.require(v, "v")
    cu = _lengths(cu_seqlens_k)
    n, L = len(cu) - 1, _lib.lib()
    conv_k, conv_v = module.compressor.compressor_k, module.compressor.compressor_v
    block, stride = module.compression_block, module.compression_stride
    wk, wv = _lib.require(conv_k.weight, "compressor_k.weight"), _lib.require(conv_v.weight, "compressor_v.weight")
    bk, bv = _lib.require(conv_k.bias, "compressor_k.bias"), _lib.require(conv_v.bias, "compressor_v.bias")
    old_table, ck_old, cv_old = None, None, None
    if old is not None:
        if n != old.nseq:
            raise ValueError("the number of sequences changed")
        old_table, ck_old, cv_old = old._table, _lib.require(old.ck, "cache.ck"), _lib.require(old.cv, "cache.cv")
    for x, w, b, c in ((k, wk, bk, ck_old), (v, wv, bv, cv_old)):
        D = x.shape[2]
        if w.shape != (D, D, block) or (b is not None and b.shape != (D,)):
            raise RuntimeError("head_dim %d does not fit compression weights %s" % (D, tuple(w.shape)))
        if c is not None and (c.shape[1:] != x.shape[1:] or c.shape[0] < old_table[2 * n + 1]):
            raise RuntimeError("a cache of %s does not fit %d positions of %s" % (tuple(c.shape), old_table[2 * n + 1], tuple(x.shape[1:])))
    table, info = (ctypes.c_int32 * (6 * n + 4))(), (ctypes.c_int32 * 3)()
    rc = L.nsa_cache_plan(cu, old_table, ctypes.byref(old_table, 4 * (n + 1)) if old is not None else None, n, block, stride,
                          table, info)
    if rc == -17:
        raise ValueError(L.nsa_last_error().decode())
    _lib.check(rc, "nsa_cache_plan")
    dev = k.device
    ck, cv = (torch.empty(info[0], *x.shape[1:], dtype=torch.bfloat16, device=dev) for x in (k, v))
    D = k.shape[2]
    weights = torch.empty(2 * block * D * D, dtype=torch.bfloat16, device=dev)   # scratch: the kernels' layout
    table_dev = torch.empty(6 * n + 4, dtype=torch.int32, device=dev)            # kept with the cache
    P = _lib.ptr

    def run(x, y, wx, wy, bx, by, x_old, y_old, cx, cy):
        _lib.check(L.nsa_cache_build(P(x), P(y), P(wx), P(wy), P(bx), P(by), P(weights), P(x_old), P(y_old), P(cx), P(cy), table,
                                     P(table_dev), n, min(x.shape[0], y.shape[0]), x.shape[1], D, block, stride, _lib.stream()),
                   "nsa_cache_build")

    if k.shape[1] == v.shape[1]:
        run(k, v, wk, wv, bk, bv, ck_old, cv_old, ck, cv)
    else:   # the two have different head counts: each by itself
        run(k, k, wk, wk, bk, bk, ck_old, ck_old, ck, torch.empty_like(ck))
        run(v, v, wv, wv, bv, bv, cv_old, cv_old, cv, torch.empty_like(cv))
    return CompressedCache.__new__(CompressedCache)._set(ck, cv, table, table_dev, n, info[1])


def compress_cache(module, k, v, cu_seqlens_k):
    """Compressed K/V of a packed cache: k, v [sum L,Hkv,D] -> CompressedCache (ck, cv [sum Tc,Hkv,D]).
    Tc = (L-block)//stride + 1 per sequence, the module's Conv1d rule (nsa/compression_kv.py:298-307)."""
    cache = _build(module, k, v, cu_seqlens_k, None)
    if torch.is_grad_enabled() and any(t.requires_grad for t in (k, v, *module.compressor.parameters())):
        comp = module.compressor   # differentiable on request: the same values through the autograd functions
        w_k, w_v = _ConvLayout.apply(comp.compressor_k.weight, comp.compressor_v.weight)
        cache.ck, cache.cv = _compress(k, v, w_k, w_v, comp.compressor_k.bias, comp.compressor_v.bias, cache.cu, cache.cu_c,
                                       module.compression_block, module.compression_stride)
    return cache


def extend_compress_cache(module, cache, k, v, cu_seqlens_k):
    """The cache after tokens were appended to the sequences: k, v [sum L',Hkv,D] are the grown packed K/V with lengths
    L' >= L.  Only the compressed positions that the new tokens complete are computed (each is one [block x D] window
    times the Conv1d weight, the same contraction as nsa/compression_kv.py:298-307); the existing entries are copied."""
    return _build(module, k, v, cu_seqlens_k, cache)


def nsa_decode(module, q, k, v, cu_seqlens_k, cache=None, return_parts=False):
    """q [nseq,Hq,D] (the newest token of every sequence), k, v [sum L,Hkv,D] packed with cu_seqlens_k.
    Returns o [nseq,Hq,D].  ``cache`` = a CompressedCache from ``compress_cache`` / ``extend_compress_cache`` skips the
    re-compression.  With ``return_parts`` also returns (o_cmp, o_slc, o_swa, lse [3,nseq,Hq], idx [nseq,Hkv,n])."""
    # (nothing below is recorded by autograd: the step takes pointers.  For one short sequence the kernels take 17 us, so the
    # host path counts: no grad-mode switch, no detached views, one allocation)
    q = _lib.require(q, "q")
    k = _lib.require(k, "k")
    v = _lib.require(v, "v")
    nseq, Hq, D = q.shape
    Hkv = k.shape[1]
    if cache is None:
        with torch.no_grad():
            cache = compress_cache(module, k, v, cu_seqlens_k)
    scale = module.softmax_scale
    if scale is None or scale is True:
        scale = 1.0 if scale is True else D ** -0.5
    gating = module.gating
    w_gate, b_gate = _lib.require(gating.weight, "gating.weight"), _lib.require(gating.bias, "gating.bias")
    P, L = _lib.ptr, _lib.lib()
    n_sel = module.selected_block_count
    o = torch.empty_like(q)
    ws_bytes = L.nsa_decode_workspace_bytes(nseq, Hkv)
    ck, total_k = cache.ck, k.shape[0]
    o_cmp = o_slc = o_swa = lse = None
    if return_parts:
        idx = torch.empty(nseq, Hkv, n_sel, dtype=torch.int32, device=q.device)
        o_cmp, o_slc, o_swa = (torch.empty_like(q) for _ in range(3))
        lse = torch.empty(3, nseq, Hq, dtype=torch.float32, device=q.device)
        ws = P(cache.workspace(ws_bytes))
        idx_p = P(idx)
    else:   # the selected blocks are scratch too
        ws = P(cache.workspace(ws_bytes + 4 * nseq * Hkv * n_sel))
        idx_p = ws + ws_bytes
    tab = P(cache.table_dev)
    _lib.check(L.nsa_decode_fwd(P(q), P(k), P(v), P(ck), P(cache.cv), tab, tab + 4 * (nseq + 1),
                                tab + 4 * (5 * nseq + 4), P(w_gate), P(b_gate), None, None, None, P(o), P(o_cmp), P(o_slc),
                                P(o_swa), P(lse), idx_p, ws, ws_bytes, nseq, total_k, ck.shape[0],
                                cache.max_tc, Hq, Hkv, D, module.compression_block, module.compression_stride,
                                module.selection_block_size, n_sel, module.sliding_window, float(scale),
                                _lib.stream()), "nsa_decode_fwd")
    if return_parts:
        return o, (o_cmp, o_slc, o_swa, lse, idx)
    return o

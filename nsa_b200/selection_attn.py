"""Selected-block + sliding-window attention with the reference's API (nsa/selection_attn.py)."""
from typing import Optional, Union

import torch

from . import _lib


def _sequences(offsets, T):
    """[(start, end)] of the packed sequences: one host read of cu_seqlens, or the whole tensor when there are none."""
    if offsets is None:
        return None
    cu = [int(c) for c in (offsets.tolist() if torch.is_tensor(offsets) else offsets)]
    if cu[0] != 0 or cu[-1] != T or any(b <= a for a, b in zip(cu[:-1], cu[1:])):
        raise ValueError("cu_seqlens must start at 0, end at the token count %d and increase: %s" % (T, cu))
    return list(zip(cu[:-1], cu[1:]))


def _forward(q, k, v, block_indices, block_counts, block_size, window_size, scale, offsets, need, g_slc=None, g_swa=None):
    """(o, o_slc, lse_slc, o_swa, lse_swa, idx, counts, seqs, reverse indices).  With gates o is the gated sum (o_slc is None
    where nothing needs it), else None."""
    B, T, Hq, D = q.shape
    Hkv = k.shape[2]
    if block_indices.dtype not in (torch.int32, torch.int64):
        raise TypeError("block_indices must be int32 or int64")
    idx = block_indices.contiguous()
    S = idx.shape[-1]
    counts = None
    if torch.is_tensor(block_counts):
        counts = block_counts.to(torch.int32).contiguous()
    seqs = _sequences(offsets, T)
    if seqs is not None and B != 1:
        raise ValueError("batch size must be 1 when cu_seqlens are provided")
    P, i64 = _lib.ptr, 1 if idx.dtype == torch.int64 else 0
    L, S_ = _lib.lib(), _lib.stream()
    covers, indices = _lib.sel_fwd_kv_covers(Hq, Hkv, D, S, block_size), []
    o = torch.empty_like(q) if g_slc is not None else None
    o_slc = torch.empty_like(q) if need or o is None or not covers else None
    lse_slc = torch.empty(B, T, Hq, dtype=torch.float32, device=q.device)
    o_swa = torch.empty_like(q) if window_size > 0 else None
    lse_swa = torch.empty_like(lse_slc) if window_size > 0 else None
    opt = lambda t, sl: P(t[:, sl]) if t is not None else None
    for a, b in (seqs or [(0, T)]):
        sl, n = slice(a, b), b - a
        ix = fws = None
        fws_bytes = 0
        if covers:
            # one reverse index for the forward and the backward (a forward that has no use for it leaves it to the backward)
            ix = torch.empty(L.nsa_sel_index_bytes(B, n, n, Hkv, S, block_size), dtype=torch.uint8, device=q.device)
            _lib.check(L.nsa_sel_index(P(idx[:, sl]), i64, opt(counts, sl), P(ix), ix.numel(), B, n, n, 0, Hkv, S, block_size,
                                       S_), "nsa_sel_index")
        if covers:
            fws_bytes = L.nsa_sel_swa_fwd_ix_workspace_bytes(B, n, n, Hq, Hkv, D, S, block_size)
            fws = torch.empty(fws_bytes, dtype=torch.uint8, device=q.device)
        indices.append(ix if need and _lib.SEL_DQ_FROM_KV else None)
        _lib.check(L.nsa_sel_swa_fwd_ix(
            P(q[:, sl]), P(k[:, sl]), P(v[:, sl]), P(idx[:, sl]), i64, opt(counts, sl), P(ix), opt(o_slc, sl),
            P(lse_slc[:, sl]), opt(o_swa, sl), opt(lse_swa, sl), opt(g_slc, sl), opt(g_swa, sl), None, None, opt(o, sl), P(fws),
            fws_bytes, B, n, Hq, Hkv, D, S, block_size, window_size, scale, n, 0, S_), "nsa_sel_swa_fwd")
    return o, o_slc, lse_slc, o_swa, lse_swa, idx, counts, seqs, indices


def _backward(q, k, v, lse_slc, lse_swa, idx, counts, indices, meta, do_slc, delta_slc, do_swa, delta_swa, g_slc=None, g_swa=None):
    """dq, dk, dv; do_x is the upstream gradient of branch x before its gate, delta_x includes the gate."""
    block_size, window_size, scale, seqs = meta
    B, T, Hq, D = q.shape
    Hkv, S, L = k.shape[2], idx.shape[-1], _lib.lib()
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    P, i64 = _lib.ptr, 1 if idx.dtype == torch.int64 else 0
    opt = lambda t, sl: P(t[:, sl]) if t is not None else None
    for (a, b), ix in zip(seqs or [(0, T)], indices):
        sl, n = slice(a, b), b - a
        shape = (B, n, n, Hq, Hkv, D, S, block_size)
        if ix is None and _lib.SEL_DQ_FROM_KV:
            ix = torch.empty(L.nsa_sel_index_bytes(B, n, n, Hkv, S, block_size), dtype=torch.uint8, device=q.device)
            _lib.check(L.nsa_sel_index(P(idx[:, sl]), i64, opt(counts, sl), P(ix), ix.numel(), B, n, n, 0, Hkv, S, block_size,
                                       _lib.stream()), "nsa_sel_index")
        ws_bytes = (L.nsa_sel_swa_bwd_ix_workspace_bytes(*shape, window_size) if ix is not None
                    else _lib.sel_swa_bwd_workspace_bytes(*shape))
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q.device)
        _lib.check(L.nsa_sel_swa_bwd_ix(
            P(q[:, sl]), P(k[:, sl]), P(v[:, sl]), P(idx[:, sl]), i64, opt(counts, sl), P(ix),
            P(do_slc[:, sl]), P(lse_slc[:, sl]), P(delta_slc[:, sl]), opt(g_slc, sl),
            opt(do_swa, sl), opt(lse_swa, sl), opt(delta_swa, sl), opt(g_swa, sl),
            P(dq[:, sl]), 0, P(dk[:, sl]), P(dv[:, sl]), P(ws), ws_bytes,
            B, b - a, Hq, Hkv, D, S, block_size, window_size, scale, b - a, 0, _lib.stream()), "nsa_sel_swa_bwd")
    return dq, dk, dv


class ParallelNSAFunction(torch.autograd.Function):
    """Drop-in for ``ParallelNSAFunction`` (nsa/selection_attn.py:679-737):
    apply(q, k, v, block_indices, block_counts, block_size, window_size, scale, offsets) -> (o_slc, o_swa).

    With ``offsets`` (= cu_seqlens, batch size 1) the tokens are packed sequences of different lengths; block indices
    and the causal / window masks are relative to each sequence's own start, as in the reference's varlen indexing
    (nsa/selection_attn.py:419-425).  Each sequence is one launch chain on its slice of the packed tensors."""

    @staticmethod
    def forward(ctx, q, k, v, block_indices, block_counts, block_size, window_size, scale, offsets):
        q, k, v = (_lib.require(t, n) for t, n in ((q, "q"), (k, "k"), (v, "v")))
        _, o_slc, lse_slc, o_swa, lse_swa, idx, counts, seqs, indices = _forward(
            q, k, v, block_indices, block_counts, block_size, window_size, float(scale), offsets, any(ctx.needs_input_grad))
        ctx.save_for_backward(q, k, v, o_slc, lse_slc, o_swa, lse_swa, idx, counts, *indices)
        ctx.meta = (block_size, window_size, float(scale), seqs)
        return o_slc, o_swa

    @staticmethod
    def backward(ctx, do_slc, do_swa):
        q, k, v, o_slc, lse_slc, o_swa, lse_swa, idx, counts, *indices = ctx.saved_tensors
        L = _lib.lib()

        def delta_of(o, do):
            d = torch.empty(q.shape[:3], dtype=torch.float32, device=q.device)
            _lib.check(L.nsa_rowdot(_lib.ptr(o), _lib.ptr(do), None, _lib.ptr(d), None, d.numel(), q.shape[3], _lib.stream()),
                       "nsa_rowdot")
            return d

        do_slc = _lib.require(do_slc, "do_slc") if do_slc is not None else torch.zeros_like(q)
        delta_slc, delta_swa = delta_of(o_slc, do_slc), None
        if ctx.meta[1] > 0:
            do_swa = _lib.require(do_swa, "do_swa") if do_swa is not None else torch.zeros_like(q)
            delta_swa = delta_of(o_swa, do_swa)
        else:
            do_swa = None
        dq, dk, dv = _backward(q, k, v, lse_slc, lse_swa, idx, counts, indices, ctx.meta, do_slc, delta_slc, do_swa, delta_swa)
        return dq, dk, dv, None, None, None, None, None, None


class _GatedNSA(torch.autograd.Function):
    """parallel_nsa for gates of the queries' type: the gated sum is formed by the selected branch's last kernel, the gates'
    gradients with the deltas in one pass (as torch operations they cost a further 13 % of the forward).  ``need``: whether
    there will be a backward (ctx.needs_input_grad is true under no_grad as well)."""

    @staticmethod
    def forward(ctx, q, k, v, g_slc, g_swa, block_indices, block_counts, block_size, window_size, scale, offsets, need):
        q, k, v, g_slc, g_swa = (_lib.require(t, n) for t, n in (
            (q, "q"), (k, "k"), (v, "v"), (g_slc, "g_slc"), (g_swa if window_size > 0 else None, "g_swa")))
        g_slc, g_swa = _lib.aligned(g_slc), _lib.aligned(g_swa)   # (the backward at head_dim 64 copies them 32 bytes at a time)
        o, o_slc, lse_slc, o_swa, lse_swa, idx, counts, seqs, indices = _forward(
            q, k, v, block_indices, block_counts, block_size, window_size, float(scale), offsets, need, g_slc, g_swa)
        if need:
            ctx.save_for_backward(q, k, v, g_slc, g_swa, o_slc, lse_slc, o_swa, lse_swa, idx, counts, *indices)
            ctx.meta = (block_size, window_size, float(scale), seqs)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, g_slc, g_swa, o_slc, lse_slc, o_swa, lse_swa, idx, counts, *indices = ctx.saved_tensors
        do = _lib.require(do, "do")
        L, P, win = _lib.lib(), _lib.ptr, o_swa is not None
        delta_slc, dg_slc = torch.empty_like(lse_slc), torch.empty_like(g_slc)
        delta_swa, dg_swa = (torch.empty_like(lse_slc), torch.empty_like(g_slc)) if win else (None, None)
        _lib.check(L.nsa_rowdot3(P(o_slc), P(o_swa), None, P(do), P(g_slc), P(g_swa), None, P(delta_slc), P(delta_swa), None,
                                 P(dg_slc), P(dg_swa), None, lse_slc.numel(), q.shape[3], _lib.stream()), "nsa_rowdot3")
        dq, dk, dv = _backward(q, k, v, lse_slc, lse_swa, idx, counts, indices, ctx.meta, do, delta_slc, do if win else None,
                               delta_swa, g_slc, g_swa)
        return dq, dk, dv, dg_slc, dg_swa, None, None, None, None, None, None, None


def parallel_nsa(q: torch.Tensor,
                 k: torch.Tensor,
                 v: torch.Tensor,
                 g_slc: torch.Tensor,
                 g_swa: torch.Tensor,
                 block_indices: torch.LongTensor,
                 block_counts: Optional[Union[torch.LongTensor, int]] = None,
                 block_size: int = 64,
                 window_size: int = 0,
                 scale: Optional[float] = None,
                 cu_seqlens: Optional[torch.LongTensor] = None,
                 head_first: bool = False) -> torch.Tensor:
    """Drop-in for ``parallel_nsa`` (nsa/selection_attn.py:740-814), exported as ``selection_attention``.

    q [B,T,HQ,K]; k,v [B,T,H,K]; g_slc,g_swa [B,T,HQ]; block_indices [B,T,H,S]; block_counts an int, a
    [B,T,H] tensor or None.  Returns o_slc*g_slc (+ o_swa*g_swa when window_size > 0), shape [B,T,HQ,K].
    ``head_first=True`` takes/returns the [B,H,T,...] layouts.
    """
    if scale is None:
        scale = k.shape[-1] ** -0.5
    if cu_seqlens is not None:
        assert q.shape[0] == 1, "batch size must be 1 when cu_seqlens are provided"
    if head_first:
        q, k, v, block_indices = (x.transpose(1, 2) for x in (q, k, v, block_indices))
        g_slc, g_swa = g_slc.transpose(1, 2), g_swa.transpose(1, 2)
        if isinstance(block_counts, torch.Tensor):
            block_counts = block_counts.transpose(1, 2)
    assert q.shape[2] % (k.shape[2] * 16) == 0, "Group size must be a multiple of 16 in NSA"
    if isinstance(block_counts, int):
        block_indices = block_indices[:, :, :, :block_counts]
        block_counts = None
    gates = (g_slc, g_swa) if window_size > 0 else (g_slc,)
    if all(torch.is_tensor(g) and g.is_cuda and g.dtype == q.dtype and g.shape == q.shape[:3] for g in gates):
        need = torch.is_grad_enabled() and any(t.requires_grad for t in (q, k, v, *gates))
        o = _GatedNSA.apply(q, k, v, g_slc, g_swa if window_size > 0 else None, block_indices, block_counts, block_size,
                            window_size, scale, cu_seqlens, need)
        return o.transpose(1, 2) if head_first else o
    o_slc, o_swa = ParallelNSAFunction.apply(q, k, v, block_indices, block_counts, block_size, window_size, scale,
                                             cu_seqlens)
    if window_size > 0:
        o = torch.addcmul(o_slc * g_slc.unsqueeze(-1), o_swa, g_swa.unsqueeze(-1))
    else:
        o = o_slc * g_slc.unsqueeze(-1)
    if head_first:
        o = o.transpose(1, 2)
    return o

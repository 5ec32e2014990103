"""The NSAAttention module with the reference's constructor, parameters and forward signature
(nsa/nsa.py:15-135)."""
import ctypes

import torch
from torch import nn

from . import _lib
from .compression_kv import KVCompressor


class _NSACore(torch.autograd.Function):
    """Everything of NSAAttention.forward between the compression and the output, for a query shard (context parallelism) or for a
    module whose compressor has to be called, as one autograd node: compressed attention + block selection, selected + sliding-window attention and the gated three-way
    sum (nsa/nsa.py:102-133).  Keeping the three branches in one node lets the backward feed dO and the gates straight
    to the kernels (no g*dO tensors are materialised, dQ is accumulated inside the kernels instead of by autograd)."""

    @staticmethod
    def forward(ctx, q, k, v, ck, cv, w_gate, b_gate, cfg):
        """q: [B,Tq,Hq,D] = the queries at sequence positions q0 .. q0+Tq-1; k, v: [B,T,Hkv,D] and ck, cv:
        [B,Tc,Hkv,D] cover the whole sequence; w_gate [3,D], b_gate [3]: the gate projection (rows: selected,
        window, compressed; nsa/nsa.py:59,117).  cfg[10] = q0; an optional cfg[11] = 1: causal selection scores."""
        (stride, block, causal, scale, pool_k, pool_s, pool_p, n_sel, sel_block, window, q0) = cfg[:11]
        score_mode = cfg[11] if len(cfg) > 11 else 0
        q, k, v, ck, cv = (_lib.require(t, n) for t, n in ((q, "q"), (k, "k"), (v, "v"), (ck, "ck"), (cv, "cv")))
        w_gate = _lib.aligned(_lib.require(w_gate, "gating.weight"))
        b_gate = _lib.require(b_gate, "gating.bias") if b_gate is not None else None
        B, Tq, Hq, D = q.shape
        T, Hkv, Tc = k.shape[1], k.shape[2], ck.shape[1]
        L, P, S = _lib.lib(), _lib.ptr, _lib.stream
        dev = q.device
        g_slc, g_swa, g_cmp = (torch.empty(B, Tq, Hq, dtype=q.dtype, device=dev) for _ in range(3))
        n_pool = L.nsa_pool_out_len(Tc, pool_k, pool_s, pool_p)
        if n_sel > n_pool:
            raise RuntimeError("selected index k out of range: %d blocks requested, %d exist" % (n_sel, n_pool))
        o_cmp, o_slc, o = torch.empty_like(q), torch.empty_like(q), torch.empty_like(q)
        o_swa = torch.empty_like(q) if window > 0 else None
        lse_cmp, lse_slc = (torch.empty(B, Tq, Hq, dtype=torch.float32, device=dev) for _ in range(2))
        lse_swa = torch.empty_like(lse_slc) if window > 0 else None
        idx = torch.empty(B, Tq, Hkv, n_sel, dtype=torch.int32, device=dev)
        _lib.check(L.nsa_gate_fwd(P(q), P(w_gate), P(b_gate), P(g_slc), P(g_swa), P(g_cmp), B * Tq * Hq, D, S()), "nsa_gate_fwd")
        _lib.check(L.nsa_cmp_attn_fwd_gated(P(q), P(ck), P(cv), P(o_cmp), P(lse_cmp), P(idx), None, None, None, None, None, None,
                                            B, T, Tc, Hq, Hkv, D, block, stride, 1 if causal else 0, scale, n_sel, pool_k,
                                            pool_s, pool_p, score_mode, Tq, q0, S()), "nsa_cmp_attn_fwd")
        fws_bytes = _lib.sel_swa_fwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, n_sel, sel_block)
        fws = torch.empty(fws_bytes, dtype=torch.uint8, device=dev) if fws_bytes else None
        _lib.check(L.nsa_sel_swa_fwd_ws(P(q), P(k), P(v), P(idx), 0, None, P(o_slc), P(lse_slc), P(o_swa),
                                        P(lse_swa), P(g_slc), P(g_swa), P(o_cmp), P(g_cmp), P(o), P(fws), fws_bytes, B, T,
                                        Hq, Hkv, D, n_sel, sel_block, window, scale, Tq, q0, S()), "nsa_sel_swa_fwd")
        ctx.save_for_backward(q, k, v, ck, cv, g_slc, g_swa, g_cmp, o_slc, o_swa, o_cmp, lse_slc, lse_swa, lse_cmp, idx,
                              w_gate)
        ctx.cfg = cfg
        ctx.has_bias = b_gate is not None
        return o

    @staticmethod
    def backward(ctx, do):
        (q, k, v, ck, cv, g_slc, g_swa, g_cmp, o_slc, o_swa, o_cmp, lse_slc, lse_swa, lse_cmp, idx,
         w_gate) = ctx.saved_tensors
        (stride, block, causal, scale, pool_k, pool_s, pool_p, n_sel, sel_block, window, q0) = ctx.cfg[:11]
        do = _lib.require(do, "do")
        B, Tq, Hq, D = q.shape
        T, Hkv, Tc = k.shape[1], k.shape[2], ck.shape[1]
        L, P, S = _lib.lib(), _lib.ptr, _lib.stream
        dev = q.device
        rows = B * Tq * Hq

        delta_slc, delta_cmp = (torch.empty(B, Tq, Hq, dtype=torch.float32, device=dev) for _ in range(2))
        delta_swa = torch.empty_like(delta_slc) if window > 0 else None
        dg_slc, dg_swa, dg_cmp = (torch.empty_like(g_slc) for _ in range(3))
        if window <= 0:
            dg_swa.zero_()
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        dck, dcv = torch.empty_like(ck), torch.empty_like(cv)
        ws_bytes = _lib.sel_swa_bwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, n_sel, sel_block)
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
        ws2_bytes = L.nsa_cmp_attn_bwd_workspace_bytes(B, T, Tc, Hkv, D)
        ws2 = torch.empty(ws2_bytes, dtype=torch.uint8, device=dev)
        # one streaming pass over dO: delta = g * rowsum(o * dO) and the gate gradients of all three branches
        _lib.check(L.nsa_rowdot3(P(o_slc), P(o_swa), P(o_cmp), P(do), P(g_slc), P(g_swa), P(g_cmp), P(delta_slc),
                                 P(delta_swa), P(delta_cmp), P(dg_slc), P(dg_swa), P(dg_cmp), rows, D, S()), "nsa_rowdot3")
        _lib.check(L.nsa_sel_swa_bwd_sharded(P(q), P(k), P(v), P(idx), 0, None, P(do), P(lse_slc), P(delta_slc),
                                             P(g_slc), P(do) if window > 0 else None, P(lse_swa), P(delta_swa), P(g_swa),
                                             P(dq), 0, P(dk), P(dv), P(ws), ws_bytes, B, T, Hq, Hkv, D, n_sel, sel_block,
                                             window, scale, Tq, q0, S()), "nsa_sel_swa_bwd")
        _lib.check(L.nsa_cmp_attn_bwd_sharded(P(q), P(ck), P(cv), P(lse_cmp), P(do), P(delta_cmp), P(g_cmp), P(dq), 1,
                                              P(dck), P(dcv), P(ws2), ws2_bytes, B, T, Tc, Hq, Hkv, D, block, stride,
                                              1 if causal else 0, scale, Tq, q0, S()), "nsa_cmp_attn_bwd")
        # gate projection backward: dq += dg . W in place (dq is complete here), dW and db by fixed-order reduction
        dw = torch.empty_like(w_gate)
        db = torch.empty(3, dtype=w_gate.dtype, device=dev) if ctx.has_bias else None
        ws_bytes = L.nsa_gate_bwd_workspace_bytes(rows, D)
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=dev)
        _lib.check(L.nsa_gate_bwd(P(q), P(dg_slc), P(dg_swa), P(dg_cmp), P(w_gate), P(dq), P(dw), P(db), P(ws), ws_bytes,
                                  rows, D, S()), "nsa_gate_bwd")
        return dq, dk, dv, dck, dcv, dw, db, None


def _carve(sizes):
    """Offsets of 256-byte aligned pieces of one buffer, and its size."""
    off, total = [], 0
    for n in sizes:
        off.append(total)
        total += (n + 255) & ~255
    return off, total


class _NSAModule(torch.autograd.Function):
    """NSAAttention.forward (nsa/nsa.py:94-135) as one autograd node: compression, gates, compressed attention + block
    selection, selected + sliding-window attention, gated sum.

    q [tok,Hq,D], k, v [tok,Hkv,D] packed; ``lens`` the sequence lengths.  Sequences are independent: runs of equal length
    are one batch in the attention kernels, the row-wise kernels and the compression take all of them at once, and every
    piece reads and writes its slice of the packed tensors in place.  Everything the backward needs beside q, k, v lies in
    one buffer, every other intermediate in one scratch buffer per piece, so a call makes a handful of allocations."""

    @staticmethod
    def forward(ctx, q, k, v, conv_k, conv_v, bias_k, bias_v, w_gate, b_gate, lens, cfg, need):
        # need: whether there will be a backward (ctx.needs_input_grad is true under no_grad as well)
        (stride, block, causal, scale, pool_k, pool_s, pool_p, n_sel, sel_block, window, fused, score_mode) = cfg
        names = ("q", "k", "v", "compressor_k.weight", "compressor_v.weight", "compressor_k.bias", "compressor_v.bias",
                 "gating.weight", "gating.bias")
        q, k, v, conv_k, conv_v, bias_k, bias_v, w_gate, b_gate = (
            _lib.require(t, n) for t, n in zip((q, k, v, conv_k, conv_v, bias_k, bias_v, w_gate, b_gate), names))
        tok, Hq, D = q.shape
        Hkv = k.shape[1]
        # (the kernels take the addresses: a module or keys of another head_dim would be read out of range)
        for t, name, shape in ((k, "k", (tok, Hkv, D)), (conv_k, names[3], (D, D, block)), (conv_v, names[4], (D, D, block)),
                               (bias_k, names[5], (D,)), (bias_v, names[6], (D,)), (w_gate, names[7], (3, D)), (b_gate, names[8], (3,))):
            if t is not None and t.shape != shape:
                raise RuntimeError("%s %s does not fit q %s" % (name, tuple(t.shape), tuple(q.shape)))
        w_gate = _lib.aligned(w_gate)   # (read 16 bytes at a time)
        L, P, S, chk = _lib.lib(), _lib.ptr, _lib.stream(), _lib.check
        # runs of equal-length sequences: (first token, sequences, tokens each, first compressed row, positions each)
        runs, t0, c0 = [], 0, 0
        for n in lens:
            tc = (n - block) // stride + 1 if n >= block else 0
            n_pool = L.nsa_pool_out_len(tc, pool_k, pool_s, pool_p)
            if n_sel > n_pool:
                raise RuntimeError("selected index k out of range: %d blocks requested, %d exist" % (n_sel, n_pool))
            if runs and runs[-1][2] == n:
                runs[-1][1] += 1
            else:
                runs.append([t0, 1, n, c0, tc])
            t0, c0 = t0 + n, c0 + tc
        rows, crow = tok * Hq, c0
        row_b, w_b = rows * D * 2, block * D * D * 2
        ix_bytes = [L.nsa_sel_index_bytes(B, T, T, Hkv, n_sel, sel_block) for _, B, T, _, _ in runs]
        use_ix = not fused and _lib.SEL_DQ_FROM_KV
        covers = _lib.sel_fwd_kv_covers(Hq, Hkv, D, n_sel, sel_block)
        keep_ix = use_ix and covers   # (the query-major forward has no use for the reverse index: the backward builds it)
        # saved: ck, cv, weights in the kernels' layout (k, v), gates (3), o_slc, o_cmp, o_swa, lse (3), idx, length tables,
        # one reverse index per run
        keep_slc = need or not keep_ix   # the key-major forward can add the gated sum without storing o_slc
        off, total = _carve([crow * Hkv * D * 2] * 2 + [w_b] * 2 + [rows * 2] * 3 +
                            [row_b if keep_slc else 0, row_b, row_b if window > 0 else 0] +
                            [rows * 4] * 3 + [tok * Hkv * n_sel * 4, 8 * (len(lens) + 1)] + (ix_bytes if keep_ix else []))
        saved = torch.empty(total, dtype=torch.uint8, device=q.device)
        o = torch.empty_like(q)
        base = saved.data_ptr()
        ck, cv, wk, wv, g_slc, g_swa, g_cmp, o_slc, o_cmp, o_swa, l_slc, l_cmp, l_swa, idx, cu = (base + x for x in off[:15])
        ix = [base + x for x in off[15:]] if keep_ix else [None] * len(runs)
        if window <= 0:
            o_swa = l_swa = None
        uniform = len(runs) == 1
        chk(L.nsa_conv_weight_layout(P(conv_k), P(conv_v), wk, wv, D, block, S), "nsa_conv_weight_layout")
        if not uniform:
            host, pos = [0], 0
            for n in lens:
                pos += n
                host.append(pos)
            host.append(0)
            for _, B, _, _, tc in runs:
                host += [host[-1] + tc * (i + 1) for i in range(B)]
            chk(L.nsa_upload_table((ctypes.c_int32 * len(host))(*host), len(host), cu, S), "nsa_upload_table")
        cus = (None, None) if uniform else (cu, cu + 4 * (len(lens) + 1))
        # one order of summation in the compression whatever the batch: the selection depends on the last bits of ck
        chk(L.nsa_compress_fwd_kv(P(k), P(v), wk, wv, P(bias_k), P(bias_v), ck, cv, *cus, len(lens), runs[0][2], runs[0][4], tok,
                                  crow, Hkv, D, block, stride, 0, S), "nsa_compress_fwd_kv")
        if not fused:
            chk(L.nsa_gate_fwd(P(q), P(w_gate), P(b_gate), g_slc, g_swa, g_cmp, rows, D, S), "nsa_gate_fwd")
        for i, (t0, B, T, c0, Tc) in enumerate(runs):
            r, kv, cb = t0 * Hq, t0 * Hkv * D * 2, c0 * Hkv * D * 2      # first row, byte offsets of k/v and ck/cv
            rb, ib = r * D * 2, idx + t0 * Hkv * n_sel * 4
            at = lambda p, x: None if p is None else p + x
            gate = (P(w_gate), P(b_gate), g_slc + 2 * r, g_swa + 2 * r, g_cmp + 2 * r) if fused else (None,) * 5
            chk(L.nsa_cmp_attn_fwd_gated(P(q) + rb, ck + cb, cv + cb, o_cmp + rb, l_cmp + 4 * r, ib, None, *gate, B, T, Tc, Hq,
                                         Hkv, D, block, stride, 1 if causal else 0, scale, n_sel, pool_k, pool_s, pool_p,
                                         score_mode, T, 0, S), "nsa_cmp_attn_fwd")
            ws_bytes = 0
            if covers:
                size = L.nsa_sel_swa_fwd_ix_workspace_bytes if keep_ix else L.nsa_sel_swa_fwd_workspace_bytes
                ws_bytes = size(B, T, T, Hq, Hkv, D, n_sel, sel_block)
            if keep_ix:
                chk(L.nsa_sel_index(ib, 0, None, ix[i], ix_bytes[i], B, T, T, 0, Hkv, n_sel, sel_block, S), "nsa_sel_index")
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=q.device) if ws_bytes else None
            chk(L.nsa_sel_swa_fwd_ix(P(q) + rb, P(k) + kv, P(v) + kv, ib, 0, None, ix[i], o_slc + rb if keep_slc else None, l_slc + 4 * r,
                                     at(o_swa, rb), at(l_swa, 4 * r), g_slc + 2 * r, g_swa + 2 * r, o_cmp + rb, g_cmp + 2 * r,
                                     P(o) + rb, P(ws), ws_bytes, B, T, Hq, Hkv, D, n_sel, sel_block, window, scale, T, 0, S),
                "nsa_sel_swa_fwd")
        if need:
            ctx.save_for_backward(q, k, v, w_gate, saved)
            ctx.meta = (cfg, runs, off, ix_bytes if use_ix else None, keep_ix, len(lens), b_gate is not None,
                        (bias_k is not None, bias_v is not None))
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, w_gate, saved = ctx.saved_tensors
        cfg, runs, off, ix_bytes, keep_ix, nseq, has_bg, has_bc = ctx.meta
        (stride, block, causal, scale, pool_k, pool_s, pool_p, n_sel, sel_block, window, fused, score_mode) = cfg
        do = _lib.require(do, "do")
        tok, Hq, D = q.shape
        Hkv, rows, dev = k.shape[1], tok * Hq, q.device
        L, P, S, chk = _lib.lib(), _lib.ptr, _lib.stream(), _lib.check
        base = saved.data_ptr()
        ck, cv, wk, wv, g_slc, g_swa, g_cmp, o_slc, o_cmp, o_swa, l_slc, l_cmp, l_swa, idx, cu = (base + x for x in off[:15])
        ix = [base + x for x in off[15:]] if keep_ix else [None] * len(runs)
        if window <= 0:
            o_swa = l_swa = None
        crow = sum(B * Tc for _, B, _, _, Tc in runs)
        need_w = ctx.needs_input_grad[3:7]
        empty = lambda *shape: torch.empty(*shape, dtype=torch.bfloat16, device=dev)
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        dwk, dwv = (empty(D, D, block) if n else None for n in need_w[:2])
        dbk, dbv = (empty(D) if n and has else None for n, has in zip(need_w[2:], has_bc))
        dw, db = torch.empty_like(w_gate), empty(3) if has_bg else None
        c_bytes = L.nsa_compress_bwd_kv_workspace_bytes(nseq, runs[0][4], crow, len(runs) > 1, Hkv, D, block, stride)
        gw_bytes = L.nsa_gate_bwd_workspace_bytes(rows, D)
        # scratch: delta (3), gate gradients (3), dck, dcv, workspaces of the gate and compression backward
        o2, total = _carve([rows * 4] * 3 + [rows * 2] * 3 + [crow * Hkv * D * 2] * 2 + [gw_bytes, c_bytes])
        scratch = torch.empty(total, dtype=torch.uint8, device=dev)
        d_slc, d_swa, d_cmp, dg_slc, dg_swa, dg_cmp, dck, dcv, gws, cws = (scratch.data_ptr() + x for x in o2)
        if window <= 0:
            scratch[o2[4]:o2[5]].zero_()   # the gate gradient of the branch that is not there
        at = lambda p, x: None if p is None else p + x
        win = window > 0
        add_gate = keep_ix
        if not fused:
            # one streaming pass over dO: delta = g * rowsum(o * dO) and the gate gradients of all three branches
            chk(L.nsa_rowdot3(o_slc, o_swa, o_cmp, P(do), g_slc, g_swa, g_cmp, d_slc, d_swa if win else None, d_cmp, dg_slc, dg_swa,
                              dg_cmp, rows, D, S), "nsa_rowdot3")
        for i, (t0, B, T, c0, Tc) in enumerate(runs):
            r, kv, cb = t0 * Hq, t0 * Hkv * D * 2, c0 * Hkv * D * 2
            rb, ib, r4, r2 = r * D * 2, idx + t0 * Hkv * n_sel * 4, 4 * r, 2 * r
            if ix_bytes and not keep_ix:
                index = torch.empty(ix_bytes[i], dtype=torch.uint8, device=dev)
                ix[i] = index.data_ptr()
                chk(L.nsa_sel_index(ib, 0, None, ix[i], ix_bytes[i], B, T, T, 0, Hkv, n_sel, sel_block, S), "nsa_sel_index")
            if ix_bytes:
                n1, n2 = L.nsa_attn_bwd_ix_workspace_bytes(B, T, Tc, Hq, Hkv, D, n_sel, sel_block, window), 0
            else:
                n1 = _lib.sel_swa_bwd_workspace_bytes(B, T, T, Hq, Hkv, D, n_sel, sel_block)
                n2 = L.nsa_cmp_attn_bwd_workspace_bytes(B, T, Tc, Hkv, D)
            ws = torch.empty(max(n1, n2), dtype=torch.uint8, device=dev)
            qp, kp, vp, dop = P(q) + rb, P(k) + kv, P(v) + kv, P(do) + rb
            if fused:
                # delta = g * rowsum(o * dO) and the gate gradients rowsum(o * dO) are formed inside the dQ kernels while
                # the dO tile is resident (no separate pass over o_slc, o_swa, o_cmp and dO)
                chk(L.nsa_sel_swa_bwd_fused(qp, kp, vp, ib, 0, None, o_slc + rb, at(o_swa, rb), dop, l_slc + r4, d_slc + r4,
                                            g_slc + r2, dg_slc + r2, at(l_swa, r4), d_swa + r4 if win else None, g_swa + r2,
                                            dg_swa + r2 if win else None, P(dq) + rb, 0, P(dk) + kv, P(dv) + kv, P(ws), n1, B,
                                            T, Hq, Hkv, D, n_sel, sel_block, window, scale, T, 0, S), "nsa_sel_swa_bwd_fused")
                chk(L.nsa_cmp_attn_bwd_fused(qp, ck + cb, cv + cb, o_cmp + rb, l_cmp + r4, dop, d_cmp + r4, g_cmp + r2,
                                             dg_cmp + r2, P(dq) + rb, 1, dck + cb, dcv + cb, P(ws), n2, B, T, Tc, Hq, Hkv, D,
                                             block, stride, 1 if causal else 0, scale, T, 0, S), "nsa_cmp_attn_bwd_fused")
            elif ix_bytes:
                chk(L.nsa_attn_bwd_ix(qp, kp, vp, ck + cb, cv + cb, ib, 0, None, ix[i], dop, l_slc + r4, at(l_swa, r4), l_cmp + r4,
                                      d_slc + r4, d_swa + r4, d_cmp + r4, g_slc + r2, g_swa + r2, g_cmp + r2, dg_slc + r2, dg_swa + r2,
                                      dg_cmp + r2, P(w_gate) if add_gate else None, P(dq) + rb,
                                      P(dk) + kv, P(dv) + kv, dck + cb, dcv + cb, P(ws), n1, B, T, Tc, Hq, Hkv, D, n_sel,
                                      sel_block, window, block, stride, 1 if causal else 0, scale, S), "nsa_attn_bwd")
            else:
                chk(L.nsa_sel_swa_bwd_ix(qp, kp, vp, ib, 0, None, ix[i], dop, l_slc + r4, d_slc + r4, g_slc + r2,
                                         dop if win else None, at(l_swa, r4), d_swa + r4 if win else None, g_swa + r2,
                                         P(dq) + rb, 0, P(dk) + kv, P(dv) + kv, P(ws), n1, B, T, Hq, Hkv, D, n_sel, sel_block,
                                         window, scale, T, 0, S), "nsa_sel_swa_bwd")
                chk(L.nsa_cmp_attn_bwd_sharded(qp, ck + cb, cv + cb, l_cmp + r4, dop, d_cmp + r4, g_cmp + r2, P(dq) + rb, 1,
                                               dck + cb, dcv + cb, P(ws), n2, B, T, Tc, Hq, Hkv, D, block, stride,
                                               1 if causal else 0, scale, T, 0, S), "nsa_cmp_attn_bwd")
        # gate projection backward: dq += dg . W in place (dq is complete here) unless the selected branch's reduction added it,
        # dW and db by fixed-order reduction
        chk(L.nsa_gate_bwd(P(q), dg_slc, dg_swa, dg_cmp, P(w_gate), None if add_gate else P(dq), P(dw), P(db), gws, gw_bytes, rows, D, S), "nsa_gate_bwd")
        # compression backward: its dX is added to dk, dv
        if c_bytes:
            cus = (None, None) if len(runs) == 1 else (cu, cu + 4 * (nseq + 1))
            chk(L.nsa_compress_bwd_kv(P(k), P(v), wk, wv, dck, dcv, P(dk), P(dv), 1, P(dwk), P(dwv), P(dbk), P(dbv), 2, cws,
                                      c_bytes, *cus, nseq, runs[0][2], runs[0][4], tok, crow, Hkv, D, block, stride, S),
                "nsa_compress_bwd_kv")
        else:   # a geometry the tensor-core kernels do not cover
            cin, cout = [0], [0]
            for _, B, T, _, Tc in runs:
                for _ in range(B):
                    cin.append(cin[-1] + T)
                    cout.append(cout[-1] + Tc)
            table = _lib.device_table(cin + cout, dev)
            cu_in, cu_out = P(table), P(table) + 4 * (nseq + 1)
            n = L.nsa_compress_bwd_workspace_bytes(nseq, Hkv, D, block)
            ws = torch.empty(n, dtype=torch.uint8, device=dev)
            for x, w, dy, dx, gw, gb in ((k, wk, dck, dk, dwk, dbk), (v, wv, dcv, dv, dwv, dbv)):
                part = torch.empty_like(dx)
                gw32 = torch.empty(block * D, D, dtype=torch.float32, device=dev) if gw is not None else None
                gb32 = torch.empty(D, dtype=torch.float32, device=dev) if gb is not None else None
                chk(L.nsa_compress_bwd(P(x), w, dy, P(part), P(gw32), P(gb32), P(ws), n, cu_in, cu_out, nseq, Hkv, D, block,
                                       stride, max(T for _, _, T, _, _ in runs), crow, S), "nsa_compress_bwd")
                dx.add_(part)
                if gw is not None:
                    gw.copy_(gw32.view(block, D, D).permute(2, 1, 0))
                if gb is not None:
                    gb.copy_(gb32)
        return dq, dk, dv, dwk, dwv, dbk, dbv, dw, db, None, None, None


_compressor_forward = KVCompressor.forward


class NSAAttention(nn.Module):
    """Drop-in for ``nsa.nsa.NSAAttention``.

    Same constructor arguments and defaults, same sub-modules and parameter names (``compressor`` holding
    ``compressor_k`` / ``compressor_v`` Conv1d parameter sets, ``gating`` = Linear(head_dim, 3)), so a
    reference ``state_dict`` loads unchanged.  ``forward`` takes packed q [B*T,Hq,D], k,v [B*T,Hkv,D] and
    ``cu_seqlens`` of equal-length sequences (as the reference's reshape at nsa/nsa.py:97 assumes) and returns
    [B*T,Hq,D].  Gates are the raw linear outputs (no activation), as in the reference.
    """

    def __init__(
        self,
        head_dim: int,
        causal=False,
        softmax_scale=None,
        attention_dropout=0.0,
        deterministic=False,
        compression_stride=16,
        compression_block=32,
        selection_block=64,
        selected_block_count=16,
        sliding_window=512,
        device=None,
        dtype=None,
    ):
        super().__init__()
        if attention_dropout not in (0, 0.0, None):
            raise NotImplementedError("attention dropout is not part of the NSA path (the reference never applies it)")
        self.causal = causal
        self.softmax_scale = softmax_scale
        self.drop_p = attention_dropout
        self.deterministic = deterministic
        self.sliding_window = sliding_window
        self.selected_block_count = selected_block_count
        self.selection_block_size = selection_block
        self.compression_stride = compression_stride
        self.compression_block = compression_block
        self.compressor = KVCompressor(compression_stride, compression_block, head_dim, device, dtype)
        self.pool_kernel_size = selection_block // compression_stride + 1
        self.pool_padding = compression_block // compression_stride - 2
        self.pool_stride = selection_block // compression_stride
        self.gating = nn.Linear(head_dim, 3, device=device, dtype=dtype)
        # Not a constructor argument (the signature stays the reference's).  True folds the gate projection into the
        # compressed-attention kernel and the backward's row pre-pass into the dQ kernels: three launches fewer per step,
        # which pays for small, launch-bound shapes; at the benchmark's shape the separate streaming kernels are faster
        # (they read rows fully coalesced; a thread-per-row epilogue does not), so the default is False.
        self.fuse_row_passes = False
        # Selection scores (also not a constructor argument).  "reference": what the reference's scoring does -- the
        # soft-max of the unscaled, unmasked q.ck over all compressed keys (nsa/torch_attention.py:121-125), so blocks in
        # a query's future can be selected and are then skipped.  "causal": the compressed branch's own attention
        # probabilities (scaled, causally masked), as in the NSA paper: every selected block is visible.
        self.score_mode = "reference"

    def forward(
        self,
        q: torch.Tensor,
        k: torch.Tensor,
        v: torch.Tensor,
        cu_seqlens: torch.Tensor,
        max_seqlen=None,
        cu_seqlens_k: torch.Tensor = None,
        max_seqlen_k=None,
        causal: bool = None,
    ) -> torch.Tensor:
        causal = self.causal if causal is None else causal
        cu_seqlens_k = cu_seqlens if cu_seqlens_k is None else cu_seqlens_k
        bs = cu_seqlens_k.numel() - 1
        head_qk_dim = q.shape[2]
        num_token = k.shape[0]
        lens = [num_token // bs] * bs
        if bs > 1 and (max_seqlen is None or bs * int(max_seqlen) != num_token):
            # Sequences of different lengths are accepted too (the reference's reshape at nsa/nsa.py:97 cannot take them).
            # Costs one host read of cu_seqlens.
            cu = [int(c) for c in cu_seqlens_k.tolist()]
            if any(b - a != cu[1] - cu[0] for a, b in zip(cu[:-1], cu[1:])):
                lens = [b - a for a, b in zip(cu[:-1], cu[1:])]
        # (equal lengths: q may be the first tokens of every sequence alone)
        prefix = q.shape[0] != num_token and q.shape[0] % bs == 0 and lens == [num_token // bs] * bs
        if sum(lens) != num_token or (q.shape[0] != num_token and not prefix) or v.shape != k.shape:
            raise ValueError("%d sequences over %d tokens do not fit q %s, k %s, v %s"
                             % (bs, sum(lens), tuple(q.shape), tuple(k.shape), tuple(v.shape)))
        scale = self.softmax_scale
        if scale is None or scale is True:
            # the reference's own callers pass `True` here positionally (tests/test_nsa_module.py:25), which its
            # kernels read as 1.0; None selects D^-0.5 in both attention entry points
            scale = 1.0 if scale is True else head_qk_dim ** -0.5
        cfg = (self.compression_stride, self.compression_block, bool(causal), float(scale), self.pool_kernel_size,
               self.pool_stride, self.pool_padding, self.selected_block_count, self.selection_block_size,
               self.sliding_window, bool(self.fuse_row_passes), {"reference": 0, "causal": 1}[self.score_mode])
        comp = self.compressor
        if prefix or not self._inlines_compressor():
            return self._through_compressor(q, k, v, cu_seqlens_k, lens, cfg)
        tensors = (q, k, v, comp.compressor_k.weight, comp.compressor_v.weight, comp.compressor_k.bias, comp.compressor_v.bias,
                   self.gating.weight, self.gating.bias)
        need = torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)
        return _NSAModule.apply(*tensors, lens, cfg, need)

    def _inlines_compressor(self):
        """Whether the compression can be part of the module's own node: not where someone would see that ``compressor`` is not
        called (hooks, a substitute or a wrapper for it) or where its geometry was set apart from the module's."""
        c = self.compressor
        return (type(c) is KVCompressor and KVCompressor.forward is _compressor_forward and "forward" not in c.__dict__
                and not (c._forward_hooks or c._forward_pre_hooks or c._backward_hooks or c._backward_pre_hooks)
                and not torch.nn.modules.module._has_any_global_hook()
                and c.block_size == self.compression_block and c.block_stride == self.compression_stride)

    def _through_compressor(self, q, k, v, cu, lens, cfg):
        """The forward with a call of ``self.compressor``, one sequence length at a time.  (``fuse_row_passes`` does not apply.)"""
        if any(n != lens[0] for n in lens):
            outs, t = [], 0
            for n in lens:
                one = torch.tensor([0, n], dtype=torch.int32, device=q.device)
                outs.append(self._through_compressor(q[t:t + n], k[t:t + n], v[t:t + n], one, [n], cfg))
                t += n
            return torch.cat(outs, 0)
        ck, cv, _ = self.compressor(k, v, cu, None)
        q4, k4, v4 = (x.reshape(len(lens), -1, *x.shape[1:]) for x in (q, k, v))
        o = _NSACore.apply(q4, k4, v4, ck, cv, self.gating.weight, self.gating.bias, cfg[:10] + (0, cfg[11]))
        return o.reshape(-1, *o.shape[2:])

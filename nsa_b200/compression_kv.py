"""K/V block compression with the reference's API (nsa/compression_kv.py).

``compress_kv``, ``calc_compressed_len``, ``KVCompressorVarlen`` and ``KVCompressor`` keep the reference's
names, arguments, parameter names/shapes and return values; the work is done by ``nsa_compress_fwd_kv`` and
``nsa_compress_bwd_kv`` of libnsa_b200.so (``nsa_compress_bwd`` where a block is not one or two strides).
"""
import math

import torch
import torch.nn as nn
from torch.nn import init

from . import _lib


def calc_compressed_len(x, stride, size):
    """nsa/compression_kv.py:9-10 (the functional path's length rule, one less than Conv1d's)."""
    return (x - size) // stride


class _CompressPair(torch.autograd.Function):
    """(ck, cv) = compress(k; w_k, b_k), compress(v; w_v, b_v).  k, v [tok,H,D]; weights [l*D, D]; biases [D] or None.  An output
    that nothing uses gives no gradients (None, not zeros).
    ``split``: see nsa_compress_fwd_kv; the package leaves it off, a block selection may follow."""

    @staticmethod
    def forward(ctx, k, v, w_k, w_v, b_k, b_v, cu_in, cu_out, block, stride, split, table=None):
        k, v, w_k, w_v = (_lib.require(t, n) for t, n in ((k, "k"), (v, "v"), (w_k, "w_k"), (w_v, "w_v")))
        b_k, b_v = _lib.require(b_k, "bias"), _lib.require(b_v, "bias")
        ctx.set_materialize_grads(False)
        tok, H, D = k.shape
        if v.shape != k.shape:
            raise ValueError("k %s and v %s differ in shape" % (tuple(k.shape), tuple(v.shape)))
        for w in (w_k, w_v):
            if w.shape != (block * D, D):
                raise ValueError("weight must have shape [block*D, D] = %s, got %s" % ((block * D, D), tuple(w.shape)))
        nseq, total_out = len(cu_in) - 1, cu_out[-1]
        ck = torch.empty(total_out, H, D, dtype=torch.bfloat16, device=k.device)
        cv = torch.empty(total_out, H, D, dtype=torch.bfloat16, device=k.device)
        if table is None:
            table = _lib.device_table([*cu_in, *cu_out], k.device)   # cu_in, then cu_out
        P, cin = _lib.ptr, table.data_ptr()
        if total_out > 0:
            _lib.check(_lib.lib().nsa_compress_fwd_kv(P(k), P(v), P(w_k), P(w_v), P(b_k), P(b_v), P(ck), P(cv), cin,
                                                      cin + 4 * (nseq + 1), nseq, 0, 0, tok, total_out, H, D, block, stride, split,
                                                      _lib.stream()),
                       "nsa_compress_fwd_kv")
        ctx.save_for_backward(k, v, w_k, w_v, table)
        ctx.meta = (nseq, H, D, block, stride, max([b - a for a, b in zip(cu_in[:-1], cu_in[1:])] + [0]), total_out)
        return ck, cv

    @staticmethod
    def backward(ctx, dck, dcv):
        k, v, w_k, w_v, table = ctx.saved_tensors
        nseq, H, D, block, stride, max_in, total_out = ctx.meta
        cin, cout = table.data_ptr(), table.data_ptr() + 4 * (nseq + 1)
        L, P = _lib.lib(), _lib.ptr
        used = (dck is not None, dcv is not None)
        if not any(used):
            return (None,) * 12
        need = [n and used[i % 2] for i, n in enumerate(ctx.needs_input_grad[:6])]
        ws_bytes = L.nsa_compress_bwd_kv_workspace_bytes(nseq, 0, total_out, 1, H, D, block, stride)
        if ws_bytes and total_out > 0:   # both tensors on the tensor cores (block = stride or 2 * stride)
            dck, dcv = _lib.require(dck if used[0] else dcv, "dck"), _lib.require(dcv if used[1] else dck, "dcv")   # (both are read)
            dk, dv = (torch.empty_like(x) if n else None for x, n in ((k, need[0]), (v, need[1])))
            dwk, dwv = (torch.empty_like(w) if n else None for w, n in ((w_k, need[2]), (w_v, need[3])))
            dbk, dbv = (torch.empty(D, dtype=torch.bfloat16, device=k.device) if n else None for n in need[4:6])
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device=k.device) if any(need[2:6]) else None
            _lib.check(L.nsa_compress_bwd_kv(P(k), P(v), P(w_k), P(w_v), P(dck), P(dcv), P(dk), P(dv), 0, P(dwk), P(dwv), P(dbk),
                                             P(dbv), 1, P(ws), ws_bytes, cin, cout, nseq, 0, 0, k.shape[0], total_out, H, D,
                                             block, stride, _lib.stream()), "nsa_compress_bwd_kv")
            return dk, dv, dwk, dwv, dbk, dbv, None, None, None, None, None, None
        ws_bytes = L.nsa_compress_bwd_workspace_bytes(nseq, H, D, block) if need[2] or need[3] else 0
        ws = torch.empty(ws_bytes, dtype=torch.uint8, device=k.device) if ws_bytes else None
        grads = []
        for i, (x, w, dy) in enumerate(((k, w_k, dck), (v, w_v, dcv))):
            if not used[i]:
                grads.append((None, None, None))
                continue
            dy = _lib.require(dy, "dy")
            dx = torch.empty_like(x) if need[i] else None
            dw = torch.empty(block * D, D, dtype=torch.float32, device=x.device) if need[2 + i] else None
            db = torch.empty(D, dtype=torch.float32, device=x.device) if need[4 + i] else None
            if total_out > 0:
                _lib.check(L.nsa_compress_bwd(P(x), P(w), P(dy), P(dx), P(dw), P(db), P(ws), ws_bytes, cin, cout, nseq, H,
                                              D, block, stride, max_in, total_out, _lib.stream()), "nsa_compress_bwd")
            else:
                for t in (dx, dw, db):
                    if t is not None:
                        t.zero_()
            grads.append((dx, dw, db))
        (dk, dwk, dbk), (dv, dwv, dbv) = grads
        return dk, dv, dwk, dwv, dbk, dbv, None, None, None, None, None, None


def _compress(k, v, w_k, w_v, b_k, b_v, cu_in, cu_out, block, stride, table=None):
    """_CompressPair, or each tensor by itself where their shapes differ (heads, head_dim, tokens behind the last sequence)."""
    args = (cu_in, cu_out, block, stride, False, table)
    if k.shape == v.shape:
        return _CompressPair.apply(k, v, w_k, w_v, b_k, b_v, *args)
    return _CompressPair.apply(k, k, w_k, w_k, b_k, b_k, *args)[0], _CompressPair.apply(v, v, w_v, w_v, b_v, b_v, *args)[0]


def _host_cu(cu_seq_len):
    if torch.is_tensor(cu_seq_len):
        return [int(c) for c in cu_seq_len.tolist()]   # one host sync, as nsa/compression_kv.py:184
    return [int(c) for c in cu_seq_len]


def compress_kv(k, v, w_k, w_v, cu_seq_len, block_stride, block_size):
    """Drop-in for ``compress_kv`` (nsa/compression_kv.py:269): returns (ck, cv, cu_out_len int32)."""
    cu_in = _host_cu(cu_seq_len)
    cu_out = [0]
    for i in range(len(cu_in) - 1):
        cu_out.append(cu_out[-1] + max(calc_compressed_len(cu_in[i + 1] - cu_in[i], block_stride, block_size), 0))
    table = _lib.device_table(cu_in + cu_out, k.device)
    ck, cv = _compress(k, v, w_k, w_v, None, None, cu_in, cu_out, block_size, block_stride, table)
    return ck, cv, table[len(cu_in):]


class _ConvLayout(torch.autograd.Function):
    """The two Conv1d weights [D,D,block] in the kernels' [block*D, D] layout (rows j*D+c, columns o), one launch."""

    @staticmethod
    def forward(ctx, w_k, w_v):
        w_k, w_v = _lib.require(w_k, "compressor_k.weight"), _lib.require(w_v, "compressor_v.weight")
        D, _, block = w_k.shape
        ctx.set_materialize_grads(False)
        ctx.dims = (D, block)
        out_k, out_v = (torch.empty(block * D, D, dtype=torch.bfloat16, device=w_k.device) for _ in range(2))
        P = _lib.ptr
        _lib.check(_lib.lib().nsa_conv_weight_layout(P(w_k), P(w_v), P(out_k), P(out_v), D, block, _lib.stream()),
                   "nsa_conv_weight_layout")
        return out_k, out_v

    @staticmethod
    def backward(ctx, *grads):
        D, block = ctx.dims
        return tuple(g.view(block, D, D).permute(2, 1, 0) if g is not None else None for g in grads)


def compress_conv(k, v, compressor, B):
    """Module-path compression of k, v [B*T,H,D] with the Conv1d parameters of a KVCompressor: the contraction of
    nsa/compression_kv.py:301-307, outputs [B,Tc,H,D] with Tc = (T-block)//stride + 1."""
    block, stride = compressor.block_size, compressor.block_stride
    w = _ConvLayout.apply(compressor.compressor_k.weight, compressor.compressor_v.weight)
    b = compressor.compressor_k.bias, compressor.compressor_v.bias

    def run(i, j):   # tensors i and j of (k, v)
        x, y = (k, v)[i], (k, v)[j]
        T = x.shape[0] // B
        Tc = (T - block) // stride + 1 if T >= block else 0
        out = _CompressPair.apply(x, y, w[i], w[j], b[i], b[j], [T * n for n in range(B + 1)], [Tc * n for n in range(B + 1)],
                                  block, stride, False)
        return [c.view(B, Tc, *c.shape[1:]) for c in out]

    return tuple(run(0, 1)) if k.shape == v.shape else (run(0, 0)[0], run(1, 1)[0])


class KVCompressorVarlen(nn.Module):
    """nsa/compression_kv.py:272-289: parameters k_weight, v_weight [block*D, D], kaiming-uniform."""

    def __init__(self, block_stride, block_size, head_dim, device, dtype):
        factory_kwargs = {"device": device, "dtype": dtype}
        super().__init__()
        self.block_stride = block_stride
        self.block_size = block_size
        self.k_weight = nn.Parameter(torch.empty(block_size * head_dim, head_dim, **factory_kwargs))
        self.v_weight = nn.Parameter(torch.empty(block_size * head_dim, head_dim, **factory_kwargs))
        self.reset_parameters()

    def forward(self, k, v, cu_seq_len, group=None):
        return compress_kv(k, v, self.k_weight, self.v_weight, cu_seq_len, self.block_stride, self.block_size)

    def reset_parameters(self) -> None:
        init.kaiming_uniform_(self.k_weight, a=math.sqrt(5))
        init.kaiming_uniform_(self.v_weight, a=math.sqrt(5))


class KVCompressor(nn.Module):
    """nsa/compression_kv.py:292-312: two nn.Conv1d(D, D, block, stride) parameter sets (state_dict
    keys compressor_k.weight/bias, compressor_v.weight/bias), applied by the CUDA compression kernel."""

    def __init__(self, block_stride, block_size, head_dim, device, dtype):
        super().__init__()
        factory_kwargs = {"device": device, "dtype": dtype}
        self.block_stride = block_stride
        self.block_size = block_size
        self.compressor_k = nn.Conv1d(head_dim, head_dim, block_size, block_stride, **factory_kwargs)
        self.compressor_v = nn.Conv1d(head_dim, head_dim, block_size, block_stride, **factory_kwargs)

    def forward(self, k, v, cu_seq_len, group=None):
        """k,v [B*T,H,D] (equal-length sequences) -> ck,cv [B,Tc,H*group,D], and cu_seq_len unchanged.
        ``group`` repeats every KV head ``group`` times as the reference does; pass None to keep the
        compact [B,Tc,H,D] form, which the compressed-attention kernel reads directly."""
        B = cu_seq_len.shape[0] - 1
        ck, cv = compress_conv(k, v, self, B)
        if group is not None:
            ck = ck.repeat_interleave(group, dim=2)
            cv = cv.repeat_interleave(group, dim=2)
        return ck, cv, cu_seq_len

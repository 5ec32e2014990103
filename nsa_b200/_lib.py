"""ctypes binding of libnsa_b200.so (the C ABI of include/nsa_b200.h).

There is no fallback: if the shared library is missing or a call fails, an exception is raised.
"""
import ctypes
import os

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "lib", "libnsa_b200.so")

_c_void_p, _c_int, _c_float, _c_size_t, _c_ll = (ctypes.c_void_p, ctypes.c_int, ctypes.c_float, ctypes.c_size_t,
                                                  ctypes.c_longlong)
P, I, F, Z, L = _c_void_p, _c_int, _c_float, _c_size_t, _c_ll

# name -> (restype, argtypes); mirrors include/nsa_b200.h declaration by declaration
SIGNATURES = {
    "nsa_abi_version": (I, []),
    "nsa_last_error": (ctypes.c_char_p, []),
    "nsa_device_status": (I, []),
    "nsa_kernel_launch_count": (L, []),
    "nsa_compress_fwd": (I, [P, P, P, P, P, P, I, I, I, I, I, I, P]),
    "nsa_compress_fwd_uniform": (I, [P, P, P, P, I, I, I, I, I, I, P]),
    "nsa_compress_fwd_kv": (I, [P] * 10 + [I, I, I, L, L, I, I, I, I, I, P]),
    "nsa_upload_table": (I, [P, I, P, P]),
    "nsa_conv_weight_layout": (I, [P, P, P, P, I, I, P]),
    "nsa_cache_plan": (I, [P, P, P, I, I, I, P, P]),
    "nsa_cache_build": (I, [P] * 13 + [I, L, I, I, I, I, P]),
    "nsa_compress_bwd_kv": (I, [P] * 8 + [I, P, P, P, P, I, P, Z, P, P, I, I, I, L, L, I, I, I, I, P]),
    "nsa_compress_bwd_kv_workspace_bytes": (Z, [I, I, L, I, I, I, I, I]),
    "nsa_compress_bwd": (I, [P, P, P, P, P, P, P, Z, P, P, I, I, I, I, I, I, I, P]),
    "nsa_compress_bwd_workspace_bytes": (Z, [I, I, I, I]),
    "nsa_compress_bwd_noalloc": (I, [P, P, P, P, P, P, P, P, I, I, I, I, I, I, I, P]),
    "nsa_cmp_attn_fwd": (I, [P, P, P, P, P, P, P, I, I, I, I, I, I, I, I, I, F, I, I, I, I, P]),
    "nsa_pool_out_len": (I, [I, I, I, I]),
    "nsa_cmp_attn_fwd_gated": (I, [P] * 12 + [I, I, I, I, I, I, I, I, I, F, I, I, I, I, I, I, I, P]),
    "nsa_cmp_attn_bwd": (I, [P, P, P, P, P, P, P, P, I, P, P, P, Z, I, I, I, I, I, I, I, I, I, F, P]),
    "nsa_cmp_attn_bwd_workspace_bytes": (Z, [I, I, I, I, I]),
    "nsa_sel_swa_fwd": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, I, I, I, F, P]),
    "nsa_sel_swa_bwd": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, I, P, P, P, Z, I, I, I, I, I, I, I, I, F, P]),
    "nsa_sel_swa_bwd_workspace_bytes": (Z, [I, I, I, I, I]),
    "nsa_sel_swa_bwd_workspace_bytes_dq": (Z, [I, I, I, I, I, I, I, I]),
    "nsa_cmp_attn_fwd_sharded": (I, [P, P, P, P, P, P, P, I, I, I, I, I, I, I, I, I, F, I, I, I, I, I, I, P]),
    "nsa_cmp_attn_bwd_sharded": (I, [P, P, P, P, P, P, P, P, I, P, P, P, Z, I, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_sel_swa_fwd_sharded": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_sel_swa_fwd_ws": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, P, Z, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_sel_index_bytes": (Z, [I, I, I, I, I, I]),
    "nsa_sel_index": (I, [P, I, P, P, Z, I, I, I, I, I, I, I, P]),
    "nsa_sel_swa_fwd_ix_workspace_bytes": (Z, [I, I, I, I, I, I, I, I]),
    "nsa_sel_swa_bwd_ix_workspace_bytes": (Z, [I, I, I, I, I, I, I, I, I]),
    "nsa_attn_bwd_ix_workspace_bytes": (Z, [I, I, I, I, I, I, I, I, I]),
    "nsa_attn_bwd_ix": (I, [P] * 6 + [I] + [P] * 22 + [Z] + [I] * 12 + [F, P]),
    "nsa_sel_swa_fwd_ix": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, P, P, Z, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_sel_swa_bwd_ix": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, P, I, P, P, P, Z, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_sel_swa_fwd_workspace_bytes": (Z, [I, I, I, I, I, I, I, I]),
    "nsa_sel_swa_bwd_sharded": (I, [P, P, P, P, I, P, P, P, P, P, P, P, P, P, P, I, P, P, P, Z, I, I, I, I, I, I, I, I,
                                    F, I, I, P]),
    "nsa_sel_swa_bwd_fused": (I, [P, P, P, P, I, P] + [P] * 11 + [P, I, P, P, P, Z, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_cmp_attn_bwd_fused": (I, [P] * 10 + [I, P, P, P, Z, I, I, I, I, I, I, I, I, I, F, I, I, P]),
    "nsa_gather_probe": (I, [P, P, P, I, I, I, I, I, I, I, I, P]),
    "nsa_decode_fwd": (I, [P] * 20 + [Z, I, L, L, I, I, I, I, I, I, I, I, I, F, P]),
    "nsa_decode_workspace_bytes": (Z, [I, I]),
    "nsa_rowdot": (I, [P, P, P, P, P, L, I, P]),
    "nsa_combine": (I, [P, P, P, P, P, P, P, L, I, P]),
    "nsa_gate_fwd": (I, [P, P, P, P, P, P, L, I, P]),
    "nsa_rowdot3": (I, [P] * 13 + [L, I, P]),
    "nsa_gate_bwd_workspace_bytes": (L, [L, I]),
    "nsa_gate_bwd": (I, [P] * 9 + [L, L, I, P]),
}

_lib = None


def lib():
    """The loaded library.  Raises if it has not been built (python -m nsa_b200.build)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(
                "libnsa_b200.so is missing at %s: build it with `python -m nsa_b200.build`. "
                "There is no CPU or PyTorch fallback for these operators." % LIB_PATH)
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            fn = getattr(handle, name)
            fn.restype = res
            fn.argtypes = args
        _lib = handle
    return _lib


def check(rc, what):
    if rc != 0:
        msg = lib().nsa_last_error().decode() if rc < 0 else "CUDA error %d at launch" % rc
        raise RuntimeError("%s failed (%d): %s" % (what, rc, msg))


def device_status():
    """Synchronise and raise if a kernel reported that it gave up waiting (never expected)."""
    rc = lib().nsa_device_status()
    if rc != 0:
        raise RuntimeError("nsa_b200 device status %d: %s" % (rc, lib().nsa_last_error().decode()))


# Selected-branch dQ from the key-major backward kernel (needs B*Tq*Hq*S*D*2 more bytes of workspace) or from the
# query-major dQ kernel.  The library picks the path from the workspace size it is handed.
SEL_DQ_FROM_KV = True


def sel_swa_bwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS):
    if SEL_DQ_FROM_KV and D == 128 and BS == 64:
        return lib().nsa_sel_swa_bwd_workspace_bytes_dq(B, T, Tq, Hq, Hkv, D, S, BS)
    return lib().nsa_sel_swa_bwd_workspace_bytes(B, T, Hkv, S, BS)


# Selected-branch forward key-major on the tensor cores (needs a workspace of about B*Tq*Hq*S*D*2 bytes) or query-major.
SEL_FWD_KV = True


def sel_fwd_kv_covers(Hq, Hkv, D, S, BS):
    return SEL_FWD_KV and D == 128 and BS == 64 and S <= 32 and Hq % (16 * Hkv) == 0


def sel_swa_fwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS):
    if sel_fwd_kv_covers(Hq, Hkv, D, S, BS):
        return lib().nsa_sel_swa_fwd_workspace_bytes(B, T, Tq, Hq, Hkv, D, S, BS)
    return 0


def int32_array(values):
    """Cumulative lengths (whole numbers of any kind, in ascending order) as a host array of int32."""
    n = len(values)
    try:
        a = (ctypes.c_int32 * n)(*values)
    except TypeError:   # (ctypes takes Python's own ints only)
        values = [int(x) for x in values]
        a = (ctypes.c_int32 * n)(*values)
    if n and not -0x80000000 <= values[-1] <= 0x7fffffff:
        raise RuntimeError("length %d does not fit 32 bits" % values[-1])
    return a


def device_table(values, device):
    """A host list of int32 as a device tensor, without a stream synchronisation."""
    a = int32_array(values)
    t = torch.empty(len(a), dtype=torch.int32, device=device)
    check(lib().nsa_upload_table(a, len(a), t.data_ptr(), stream()), "nsa_upload_table")
    return t


def ptr(t):
    return None if t is None else t.data_ptr()


def stream():
    """The current stream's handle (the raw getter: a torch.cuda.Stream object costs more than a kernel launch)."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())


def aligned(t):
    """The contiguous tensor t, copied where it does not start on a 16-byte boundary (a piece of a larger buffer)."""
    return t if t is None or t.data_ptr() % 16 == 0 else t.clone()


def require(t, name, dtype=torch.bfloat16):
    if t is None:
        return None
    if not t.is_cuda:
        raise RuntimeError("%s must be a CUDA tensor: nsa_b200 has no CPU path" % name)
    if dtype is not None and t.dtype != dtype:
        raise TypeError("%s must be %s (got %s)" % (name, dtype, t.dtype))
    return t.contiguous()

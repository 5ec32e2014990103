"""The gate projection at the edges of its row groups: 8 rows per half warp (head_dim 128) or quarter warp (64), 128 or 256 rows per
block, with and without a bias."""
import pytest
import torch

from parity_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows", [1, 15, 17, 31, 127, 128, 129, 255, 257, 5003])
@pytest.mark.parametrize("bias", [True, False])
def test_gate_projection(D, rows, bias):
    from nsa_b200 import _lib
    gen = torch.Generator(device=DEV).manual_seed(rows + D)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    q, w, b = rnd(rows, D), rnd(3, D), rnd(3)
    out = torch.full((3, rows + 1), 7.0, dtype=torch.bfloat16, device=DEV)
    _lib.check(_lib.lib().nsa_gate_fwd(_lib.ptr(q), _lib.ptr(w), _lib.ptr(b) if bias else None, *(out[g].data_ptr() for g in range(3)), rows, D,
                                       _lib.stream()), "nsa_gate_fwd")
    want = w.float() @ q.float().T + (b.float()[:, None] if bias else 0)
    # one rounding to bf16 (2^-9 of the value), and D products summed in fp32 (each partial sum at most sum |w q|)
    bound = want.abs() * 2.0 ** -8 + (w.float().abs() @ q.float().abs().T) * D * 2.0 ** -24
    assert ((out[:, :rows].float() - want).abs() <= bound).all()
    assert (out[:, rows] == 7.0).all()

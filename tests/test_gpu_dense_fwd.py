"""The tcgen05 forward of the sliding window where a row's maximum grows from one tile of 128 keys to the next."""
import pytest
import torch

from parity_util import DEV, close

pytestmark = pytest.mark.gpu


def test_largest_probability_is_not_rounded_at_head_dim_64():
    """Key 3 scores 0, key 130 scores 5 and all others vanish: o = (v_3 + e^5 v_130) / (1 + e^5).  With key 130's probability as the
    exact 1 the only error of note is the rounding of o itself, 2^-8; taken relative to key 3, e^5 = 148.41 would be rounded to
    148, another 2.8e-3."""
    from nsa_b200.selection_attn import ParallelNSAFunction
    T, Hq, D = 256, 16, 64
    gen = torch.Generator(device=DEV).manual_seed(1)
    q, k = torch.zeros(1, T, Hq, D, device=DEV), torch.zeros(1, T, 1, D, device=DEV)
    q[..., 0], k[..., 0], k[0, 3, 0, 0], k[0, 130, 0, 0] = 4.0, -32.0, 0.0, 1.25
    v = torch.rand(1, T, 1, D, generator=gen, device=DEV) + 1.0
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    idx = torch.zeros(1, T, 1, 1, dtype=torch.int32, device=DEV)
    _, o = ParallelNSAFunction.apply(q, k, v, idx, None, 64, 512, 1.0, None)
    e5 = torch.tensor(5.0, dtype=torch.float64, device=DEV).exp()
    ref = (v[0, 3, 0].double() + e5 * v[0, 130, 0].double()) / (1 + e5)
    err = ((o[0, 130:].double() - ref) / ref).abs().max()
    assert err <= 2.0 ** -8 * 1.02, "relative error %.2e" % float(err)


@pytest.mark.parametrize("scale", [0.0, -0.2])
def test_head_dim_64_takes_scales_of_any_sign(scale):
    """Zero (every visible key counts the same) and negative ones, forward and backward of the window and the compressed branch."""
    from nsa_b200.selection_attn import ParallelNSAFunction
    from nsa_b200.triton_attention import flash_attn_func
    T, H, D, window = 700, 16, 64, 200
    gen = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=gen, device=DEV).bfloat16()
    q, do, k, v = rnd(1, T, H, D), rnd(1, T, H, D), rnd(1, T, 1, D), rnd(1, T, 1, D)
    Tc = (T - 32) // 16 + 1
    idx = torch.zeros(1, T, 1, 1, dtype=torch.int32, device=DEV)
    t, j = torch.arange(T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
    for n, mask, call in ((T, (j <= t) & (j > t - window), lambda a: ParallelNSAFunction.apply(*a, idx, None, 64, window, scale, None)[1]),
                          (Tc, t >= 16 * torch.arange(Tc, device=DEV)[None] + 32, lambda a: flash_attn_func(*a, 16, 32, True, scale)[0])):
        leaf = [x.clone().requires_grad_(True) for x in (q, k[:, :n], v[:, :n])]
        o = call(leaf)
        got = [o, *torch.autograd.grad(o, leaf, do)]
        ref = [x.float().requires_grad_(True) for x in (q, k[:, :n], v[:, :n])]
        s = (torch.einsum("bthd,bsd->bhts", ref[0], ref[1][:, :, 0]) * scale).masked_fill(~mask, float("-inf"))
        p = torch.softmax(s.masked_fill(~mask.any(-1, keepdim=True), 0.0), -1).masked_fill(~mask, 0.0)
        ro = torch.einsum("bhts,bsd->bthd", p, ref[2][:, :, 0])
        want = [ro, *torch.autograd.grad(ro, ref, do.float())]
        for name, a, b in zip(("o", "dq", "dk", "dv"), got, want):
            close("%s, scale %g" % (name, scale), a, b, scaled=name in ("dk", "dv"))

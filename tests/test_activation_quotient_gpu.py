"""silu and sigmoid as the kernels of the short convolution and of the gated norms have them, against float64: their quotient
comes from an approximate reciprocal and one correction."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_silu_of_every_size_of_number():
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    n = 1 << 16
    size = torch.exp2(torch.rand(n, generator=g, device="cuda") * 160 - 150)
    x = torch.cat([size, -size, torch.linspace(-90, 90, n, device="cuda"), torch.randn(n, generator=g, device="cuda") * 3])
    x = torch.cat([x, torch.tensor([0.0, -0.0, 3e38, -3e38, math.inf, -math.inf, math.nan, 87.0, -87.0, -88.5, -103.0, -104.0] + [1.0] * 52,
                                   device="cuda")])
    C = 64
    x = x[: x.numel() // C * C].view(-1, C).contiguous()
    T = x.shape[0]
    w = torch.tensor([0.0, 0.0, 0.0, 1.0], device="cuda").repeat(C, 1).contiguous()       # a convolution that passes its input on
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    y = torch.where(torch.isfinite(x), x, torch.zeros_like(x))                            # (0 times infinity: one token at a time)
    got = ops.causal_conv(y, w, None, torch.zeros(1, 3, C, device="cuda"), i32([0, T]), torch.zeros(T, dtype=torch.int32, device="cuda"),
                          i32([0]), 1, True, i32([0])).double()
    d = y.double()
    want = d / (1 + torch.exp(-d))
    # the exponential (2 ulp), the sum (1/2) and the quotient (1), each relative to 2^-23; below 2^-126, and where the
    # exponential itself is beyond float32 (x below -88.7), zero will do
    far = torch.where(d < -88.7, want.abs(), torch.zeros_like(d))
    assert bool(((got - want).abs() <= 4 * 2.0 ** -23 * want.abs() + 2.0 ** -126 + far).all())
    odd = torch.tensor([math.inf, -math.inf, math.nan, 0.0] + [1.0] * (C - 4), device="cuda").view(1, C)
    one = ops.causal_conv(odd, w[:, 3:].contiguous(), None, torch.zeros(1, 0, C, device="cuda"), i32([0, 1]), i32([0]), i32([0]), 1, False, i32([0]))
    assert one[0, 0] == math.inf and bool(torch.isnan(one[0, 1:3]).all()) and one[0, 3] == 0


def every_bfloat16():
    """All 2^16 bit patterns, a warp's neighbours far apart in size."""
    bits = (torch.arange(1 << 16, device="cuda", dtype=torch.int64) * 40503) % (1 << 16)
    return torch.where(bits < 1 << 15, bits, bits - (1 << 16)).to(torch.int16).view(torch.bfloat16)


def same(a, b):
    return bool(((a == b) | (a.isnan() & b.isnan())).all())


def test_silu_of_bfloat16_rows_has_the_bits_of_the_form_with_one_channel_a_thread():
    """Four channels a thread (four taps, 2^22 inputs or more) and one (weights off their alignment), at every bfloat16 number;
    what is not finite spoils the three tokens behind it (0 times infinity), with one channel a thread all up to the next
    multiple of eight: such rows stand four ahead of one."""
    from rllm_b200.kernels import ops
    T, E = 2048, 2304
    x = every_bfloat16().repeat(T * E // 65536 + 1)[: T * E].view(T, E).clone()
    rest = torch.arange(T, device="cuda") % 8 != 4
    x[rest] = x[rest].nan_to_num(1.0, 2.0, -2.0)
    room = torch.zeros(E * 4 + 1, device="cuda", dtype=torch.bfloat16)
    w = torch.tensor([0.0, 0.0, 0.0, 1.0], device="cuda", dtype=torch.bfloat16).repeat(E, 1).contiguous()
    room[1:] = w.view(-1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    got = [ops.causal_conv(x, v, None, torch.zeros(1, 3, E, device="cuda"), i32([0, T]), torch.zeros(T, dtype=torch.int32, device="cuda"),
                           i32([0]), 1, True, i32([0])) for v in (w, room[1:].view(E, 4))]
    assert same(*got)
    d = x.double()
    want = d / (1 + torch.exp(-d))
    ok = got[0].isfinite()
    # one rounding to bfloat16; the rest as above
    far = torch.where(d < -88.7, want.abs(), torch.zeros_like(d))
    assert bool(((got[0].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -126 + far)[ok].all())
    assert bool(ok.view(T // 8, 8, E)[:, :4].all()) and not bool(ok.all())


def test_gates_of_every_number_have_the_bits_of_the_form_with_single_values():
    from rllm_b200.kernels import ops
    T, H = 32, 2048
    x, w = torch.randn(T, H, device="cuda"), torch.ones(H, device="cuda")
    wide = every_bfloat16().view(T, H)
    room = torch.zeros(T, H + 3, device="cuda", dtype=torch.bfloat16)
    room[:, 3:] = wide
    got = [ops.gated_rmsnorm(x, g, w, 1e-6, torch.bfloat16) for g in (wide, room[:, 3:])]
    assert same(*got)
    want = x.double() * torch.rsqrt(x.double().square().mean(1, keepdim=True) + 1e-6) * torch.sigmoid(wide.double())
    assert bool((got[0].isnan() == wide.isnan()).all())
    assert bool(((got[0].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-30)[~wide.isnan()].all())
    y, z = x * 1e-25, wide.nan_to_num(0.0, 1.0, -1.0)
    room[:, 3:] = z
    assert same(*[ops.silu_gated_group_rmsnorm(y, g, w, 1e-6, 2, torch.bfloat16) for g in (z, room[:, 3:])])

"""silu as the kernels of the short convolution have it, against float64: its quotient comes from an approximate reciprocal
and one correction."""
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

"""The float32 product over its tiles: a row's bits do not depend on the rows beside it (so neither on the tile that the
product's size picks), rows that start anywhere, remainders in every dimension, and float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,offset", [(1024, 2048, 0), (8192, 260, 0), (301, 40, 0), (77, 129, 1), (2080, 63, 3), (8192, 16, 0),
                                        (8200, 40, 0), (8192, 101, 1), (4100, 520, 2)])
def test_rows_of_the_float32_product_are_independent(N, K, offset):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(N + K)
    M = 200
    a = torch.randn(M, K + 4, generator=g, device="cuda")[:, offset: offset + K]
    w = torch.randn(N, K + 4, generator=g, device="cuda")[:, offset: offset + K]
    out = torch.empty(M, N, device="cuda")
    ops.gemm_f32(a, w, out)
    want = a.double() @ w.double().t()
    # K additions and products in order: |error| <= K 2^-24 times the sum of the terms' sizes
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
    assert bool(((out.double() - want).abs() <= bound).all())
    for m in (1, 7, 8, 9, 16, 17, 33, 65, 130):
        part = torch.full((m, N + 5), float("nan"), device="cuda")
        ops.gemm_f32(a[M - m:], w, part[:, 2: N + 2])
        assert torch.equal(part[:, 2: N + 2], out[M - m:])
        assert bool(torch.isnan(part[:, :2]).all()) and bool(torch.isnan(part[:, N + 2:]).all())

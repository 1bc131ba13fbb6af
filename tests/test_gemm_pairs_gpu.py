"""The tcgen05 product on CTAs of their own and on pairs: remainders of its tiles in rows (a pair's second CTA with no row),
columns and k (a stage whose second half is empty), every tile width and epilogue, more tiles than CTAs, strided rows."""
from ctypes import c_int

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,epilogue,form", [
    (2047, 3072, 2056, "store", -192), (1100, 2040, 4160, "store", 128), (6327, 2048, 2056, "store", -256), (6300, 2050, 2048, "store", -192),
    (4100, 2048, 4096, "f32", -256), (129, 389, 5000, "f32", -128), (2047, 3070, 2048, "f32", -192), (2048, 1344, 2048, "f32", 192),
    (1100, 120, 4200, "store", -128), (300, 8200, 2048, "silu_mul", 192), (513, 4090, 2184, "silu_mul", -192),
    (1, 100, 4104, "silu_mul", -128), (257, 1000, 4096, "silu_mul", -128), (4097, 3000, 2048, "silu_mul", -256),
    (700, 3072, 2040, "store", 128), (1024, 4100, 4096, "silu_mul", -256)])
def test_products_on_every_form_of_tile(M, N, K, epilogue, form):
    """``form``: the tile's width, negative for pairs of CTAs."""
    from rllm_b200.kernels import build, ops
    code = {"store": 0, "f32": 1, "silu_mul": 2}[epilogue]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f = build.load_library("gemm_tcgen05").rllm_gemm_tcgen05_form
    assert f(c_int(M), c_int(N), c_int(K), c_int(code), c_int(sms)) == form
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    rows = N * (2 if code == 2 else 1)
    x = torch.randn(M, K + 16, generator=g, device="cuda").bfloat16()[:, 8:8 + K]
    w = (torch.randn(rows, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    full = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.float32 if code == 1 else torch.bfloat16)
    ops.gemm_tcgen05(x, w, full[:, :N], "silu_mul" if code == 2 else "store")
    ops.check_gemm_errors(x.device)
    assert bool((full[:, N:] == 7.0).all())
    got, want, size = full[:, :N].double(), x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    off = K * 2.0 ** -23 * size                            # float32 sums over K terms
    if code == 2:
        gate, up = want[:, :N], want[:, N:]
        s = torch.sigmoid(gate)
        want = gate * s * up
        # what the sums' errors become (the gate's slope is at most 1.1), the short exponential and division (2^-20 of the
        # result), and one rounding to bfloat16
        off = 1.1 * up.abs() * off[:, :N] + gate.abs() * off[:, N:] + 1e-6 * want.abs()
    if code != 1:
        off = off + 2.0 ** -8 * want.abs()
    assert bool(((got - want).abs() <= off + 1e-6).all()), float(((got - want).abs() / (off + 1e-6)).max())

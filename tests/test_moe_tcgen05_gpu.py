"""The experts' products on the tcgen05 kernels against float64, at the edges of their tiles: pairs around a tile of
128 and an instruction width of 16, experts without a pair, one expert with nearly all, sizes that are no multiple of
the 64 of k or the 128 and 256 output rows of a tile, and the gate's constants."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def by_expert(h, ids, w_gate_up, w_down, limit, alpha, shift):
    T, H = h.shape
    top, F = ids.shape[1], w_down.shape[2]
    out = torch.zeros(T * top, H, dtype=torch.float64, device=h.device)
    for e in range(w_down.shape[0]):
        t, k = torch.nonzero(ids == e, as_tuple=True)
        z = h[t].double() @ w_gate_up[e].double().t()
        g, u = z[:, :F].clamp(max=limit), z[:, F:].clamp(-limit, limit)
        y = (g * torch.sigmoid(alpha * g) * (u + shift)).bfloat16().double()      # the activations are kept in bfloat16
        out[t * top + k] = y @ w_down[e].double().t()
    return out


@pytest.mark.parametrize("T,H,F,E,top,one", [
    (2048, 2048, 1024, 32, 4, None), (65, 8, 8, 1, 1, None), (128, 64, 128, 1, 1, None), (129, 136, 264, 1, 1, None),
    (100, 64, 24, 5, 2, None), (257, 200, 136, 40, 3, None), (1000, 128, 520, 4, 1, 870)])
@pytest.mark.parametrize("limit,alpha,shift", [(float("inf"), 1.0, 0.0), (1.5, 1.702, 1.0)])
def test_experts_on_tcgen05(T, H, F, E, top, one, limit, alpha, shift):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(T + F)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    h, wgu, wd = randn(T, H).bfloat16(), (randn(E, 2 * F, H) * H ** -0.5).bfloat16(), (randn(E, H, F) * F ** -0.5).bfloat16()
    ids = torch.rand(T, E, generator=g, device="cuda").topk(top, 1).indices.int().contiguous()
    if one is not None:
        ids[:] = 0
        ids[one:] = E - 1
    assert ops.moe_tcgen05_takes(T * top, h, wgu, wd)
    got = ops.moe_experts(h, ids, wgu, wd, limit, alpha, shift)
    want = by_expert(h, ids, wgu, wd, limit, alpha, shift)
    ops.check_gemm_errors(h.device)
    # a result is rounded once, by at most 2^-8 of itself (about 2^-9 in the mean); an activation that falls to the other
    # of two neighbours moves one of F terms by 2^-7 of it
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -8
    assert float((got.double() - want).abs().max()) <= 2.0 ** -8 * (float(want.abs().max()) + float(wd.abs().max()) * 8)


def test_which_calls_take_the_tcgen05_experts():
    from rllm_b200.kernels import ops
    h = torch.zeros(64, 64, dtype=torch.bfloat16, device="cuda")
    wgu = torch.zeros(4, 48, 64, dtype=torch.bfloat16, device="cuda")
    wd = torch.zeros(4, 64, 24, dtype=torch.bfloat16, device="cuda")
    assert ops.moe_tcgen05_takes(65, h, wgu, wd) and not ops.moe_tcgen05_takes(64, h, wgu, wd)
    assert not ops.moe_tcgen05_takes(128, h.float(), wgu.float(), wd.float())
    assert not ops.moe_tcgen05_takes(128, h[:, :60].contiguous(), wgu[:, :, :60].contiguous(), wd[:, :60].contiguous())
    assert not ops.moe_tcgen05_takes(128, h, wgu[:, :44].contiguous(), wd[:, :, :22].contiguous())
    shifted = torch.zeros(64 * 64 + 4, dtype=torch.bfloat16, device="cuda")[4:].view(64, 64)
    assert not ops.moe_tcgen05_takes(128, shifted, wgu, wd)


@pytest.mark.parametrize("T,H,F,E,top,one", [
    (65, 8, 8, 1, 1, None), (128, 64, 128, 1, 1, None), (129, 136, 264, 1, 1, None), (100, 64, 24, 5, 2, None),
    (257, 200, 136, 40, 3, None), (1000, 128, 520, 4, 1, 870), (65, 1024, 512, 8, 1, None)])
def test_small_experts_on_tcgen05(T, H, F, E, top, one, monkeypatch):
    """The sizes that ordinarily take the row tiles, on the tcgen05 kernels all the same."""
    from rllm_b200.kernels import ops
    assert (H * F >= 1 << 19) == ops.moe_tcgen05_pays(E, H, F)
    monkeypatch.setenv("RLLM_GEMM", "tcgen05")
    assert ops.moe_tcgen05_pays(E, H, F)
    test_experts_on_tcgen05(T, H, F, E, top, one, 1.5, 1.702, 1.0)

"""Which kernel a call takes, as far as sizes and strides decide it: no GPU."""
import pytest
import torch

from rllm_b200.kernels import build, ops

BF16 = torch.bfloat16


def test_products_per_head_whose_rows_tma_cannot_address_keep_the_general_kernel():
    a, b = torch.empty(2048, 16, 128, dtype=BF16, device="meta"), torch.empty(16, 512, 128, dtype=BF16, device="meta")
    c = torch.empty(2048, 16, 512, dtype=BF16, device="meta")
    takes = lambda x: ops.head_gemm_tcgen05_takes(x, b, c)  # noqa: E731
    assert takes(a) and takes(a.new_empty(16, 2048, 128).transpose(0, 1))
    assert not takes(a[:1].expand(2048, 16, 128)) and not takes(a[:, :1].expand(2048, 16, 128))
    flat = torch.empty(2048 * 64 + 16 * 8 + 128, dtype=BF16, device="meta")
    assert not takes(flat.as_strided((2048, 16, 128), (64, 128, 1))) and not takes(flat.as_strided((2048, 16, 128), (128, 8, 1)))
    assert not takes(torch.empty(1, dtype=BF16, device="meta").as_strided((2048, 16, 128), (2 ** 39, 128, 1)))


@pytest.mark.parametrize("E,H,F,pairs,takes", [
    (32, 2048, 1024, 65, True), (32, 2048, 1024, 64, False), (1 << 20, 8, 512, 4096, True),
    (1 << 20, 8, 520, 4096, False), (1 << 20, 1024, 8, 4096, True), (1 << 20, 1032, 8, 4096, False),
    (1, 8, 1 << 15, 1 << 28, True), (1, 8, 1 << 15, 1 << 30, False)])
def test_experts_beyond_the_tensor_maps_keep_the_kernels_that_took_them(E, H, F, pairs, takes):
    h = torch.empty(4, H, dtype=BF16, device="meta")
    wgu, wd = torch.empty(E, 2 * F, H, dtype=BF16, device="meta"), torch.empty(E, H, F, dtype=BF16, device="meta")
    assert ops.moe_tcgen05_takes(pairs, h, wgu, wd) is takes


@pytest.mark.parametrize("q_lens,keys,heads,dv,window,tcgen05", [
    ([2048], 2048, 16, 512, 0, True), ([80], 4096, 16, 512, 0, False), ([88], 4096, 16, 512, 0, True),
    ([8] * 8, 4096, 16, 512, 0, False), ([10] * 8, 4096, 16, 512, 0, False), ([11] * 8, 4096, 16, 512, 0, True), ([64], 512, 16, 512, 0, True),
    ([64], 4096, 16, 512, 500, True), ([128], 4096, 8, 256, 0, False), ([160], 4096, 8, 256, 0, False), ([256], 4096, 8, 256, 0, True),
    ([2] * 128, 2048, 16, 512, 0, False), ([2] * 64, 2048, 16, 512, 0, True), ([2] * 128, 512, 8, 256, 0, False),
    ([4] * 64, 128, 16, 512, 0, False), ([8] * 32, 128, 16, 512, 0, False), ([32] * 16, 128, 16, 512, 0, True),
    ([64] * 8, 128, 8, 256, 0, True), ([2] * 64, 128, 8, 256, 0, False), ([1792, 3], 1792, 16, 512, 0, True),
    ([40], 4136, 32, 128, 0, False), ([100], 4096, 32, 128, 0, True), ([512], 4608, 4, 128, 0, False), ([4] * 300, 4, 32, 128, 0, False),
    ([4] * 300, 204, 32, 128, 0, False), ([32] * 16, 64, 16, 512, 0, False), ([64] * 8, 64, 8, 256, 0, True), ([64] * 8, 164, 32, 128, 0, True)])
def test_which_prompt_portions_the_tcgen05_latent_attention_pays_for(q_lens, keys, heads, dv, window, tcgen05):
    assert ops.latent_attention_tcgen05_pays(q_lens, [keys] * len(q_lens), heads, dv, window) is tcgen05


@pytest.mark.parametrize("q_lens,starts,sizes,window,pays", [
    ([2048], 0, "A", 0, True), ([33], 4096, "A", 0, True), ([17], 4096, "A", 0, False), ([8], 0, "A", 0, True), ([2], 0, "A", 0, False),
    ([8], 1024, "A", 0, False), ([300], 4096, "A", 512, True), ([33], 4096, "B", 0, False), ([64], 4096, "B", 0, True),
    ([128], 4096, "D", 0, False), ([300], 4096, "D", 0, True), ([4] * 64, 0, "A", 0, False), ([16] * 64, 200, "D", 0, False),
    ([33] * 16, 1000, "A", 0, True), ([33] * 16, 1000, "C", 0, False), ([350] * 5, 0, "C", 0, True), ([512], 30000, "A", 0, True), ([512], 60000, "A", 0, False),
    ([4096], 30000, "A", 0, True)])
def test_which_prompt_portions_run_with_every_heads_own_keys_and_values(q_lens, starts, sizes, window, pays):
    sizes = {"A": (16, 128, 128, 512, 64), "B": (8, 64, 64, 256, 32), "C": (64, 128, 128, 512, 64), "D": (4, 64, 64, 128, 32)}[sizes]
    assert ops.latent_expanded_pays(q_lens, [q + starts for q in q_lens], *sizes, window) is pays


@pytest.mark.parametrize("dtype,nope,rot,v,kv,scale,ok", [
    (BF16, 128, 64, 128, 512, 0.1, True), (BF16, 64, 8, 128, 40, 0.1, True), (torch.float32, 128, 64, 128, 512, 0.1, False),
    (BF16, 96, 64, 128, 512, 0.1, False), (BF16, 128, 64, 96, 512, 0.1, False), (BF16, 128, 0, 128, 512, 0.1, False),
    (BF16, 128, 72, 128, 512, 0.1, False), (BF16, 128, 12, 128, 512, 0.1, False), (BF16, 128, 64, 128, 500, 0.1, False),
    (BF16, 128, 64, 128, 512, -0.1, False)])
def test_which_mixers_have_that_form(dtype, nope, rot, v, kv, scale, ok, monkeypatch):
    assert ops.latent_expanded_shapes(dtype, nope, rot, v, kv, scale) is ok
    monkeypatch.delenv("RLLM_LATENT_ATTENTION", raising=False)
    assert ops.latent_expanded_allowed()
    monkeypatch.setenv("RLLM_LATENT_ATTENTION", "mma")
    assert not ops.latent_expanded_allowed()


@pytest.mark.parametrize("E,H,F,pays", [(32, 2048, 1024, True), (16, 1024, 1024, True), (8, 1024, 512, True), (4, 1024, 512, False),
                                        (1, 2048, 256, True), (1, 1024, 1024, False), (128, 512, 512, False), (8, 64, 64, False)])
def test_which_experts_the_tcgen05_kernels_pay_for(E, H, F, pays, monkeypatch):
    monkeypatch.delenv("RLLM_GEMM", raising=False)
    assert ops.moe_tcgen05_pays(E, H, F) is pays
    monkeypatch.setenv("RLLM_GEMM", "tcgen05")
    assert ops.moe_tcgen05_pays(E, H, F)


def test_how_many_warps_share_a_row_of_the_cuda_core_attention():
    """The keys that a row can see decide, not the width of the table alone."""
    from ctypes import c_int, c_longlong
    f = build.load_library("attention_simt").rllm_attention_simt_warps
    f.argtypes = [c_longlong] + [c_int] * 5
    page = 16
    for width in (64, 512, 8192):                          # keys that the table has room for
        for window, kept, chunk in ((0, 0, 0), (64, 0, 0), (500, 11, 0), (500, 12, 0), (128, 0, 0), (128, 1, 0), (630, 9, 0), (630, 10, 0), (0, 0, 64),
                                    (4000, 4, 100), (2 ** 31 - 1, 2 ** 31 - 1, 2 ** 31 - 1)):
            keys = min(width, window + kept if window else width, chunk or width)
            for rows in (1, 512, 516, 1024, 2044, 2048, 4096, 4097):
                want = 8 if rows <= 4096 and keys > 128 and keys >= min(rows // 4, 640) else 1
                assert f(rows, width // page, page, window, kept, chunk) == want


@pytest.mark.parametrize("M,N,K,epilogue,sms,form", [
    (2047, 3072, 2048, 0, 148, -192), (2047, 2048, 4096, 0, 148, -256), (2047, 2048, 2048, 0, 148, 256), (2047, 4096, 2048, 2, 148, -256),
    (1024, 2048, 8192, 0, 148, -128), (6327, 2048, 2048, 1, 148, -256), (2048, 1024, 1024, 0, 148, 128), (100, 200, 64, 0, 148, 128),
    (700, 3072, 2048, 0, 148, 128), (2047, 2048, 4096, 0, 1, 256), (8192, 1344, 8192, 0, 148, -256), (16384, 1344, 4096, 0, 148, -256),
    (8192, 1344, 4096, 0, 148, -128), (8192, 200, 8192, 0, 148, -128), (16384, 672, 4096, 2, 148, -256)])
def test_which_tile_a_product_takes(M, N, K, epilogue, sms, form):
    """The tile's width, negative for pairs of CTAs; a device of one SM has no pairs."""
    from ctypes import c_int
    f = build.load_library("gemm_tcgen05").rllm_gemm_tcgen05_form
    assert f(c_int(M), c_int(N), c_int(K), c_int(epilogue), c_int(sms)) == form


@pytest.mark.parametrize("library,chunks,heads,num_seqs,d,dv,pays", [
    ("ssd", 16, 10, 1, 128, 64, True), ("ssd", 16, 4, 1, 64, 64, False), ("ssd", 7, 4, 5, 64, 64, True), ("ssd", 6, 6, 1, 64, 64, False),
    ("ssd", 3, 4, 2, 64, 64, False), ("ssd", 3, 10, 1, 64, 64, True), ("ssd", 2, 1, 1, 64, 64, True), ("ssd", 6, 4, 1, 128, 64, False),
    ("ssd", 5, 4, 1, 128, 64, True), ("ssd", 6, 6, 1, 128, 64, True), ("ssd", 4, 2, 1, 64, 128, False), ("ssd", 4, 4, 1, 64, 128, True),
    ("ssd", 6, 1, 1, 128, 128, False), ("ssd", 6, 2, 1, 128, 128, True), ("lightning", 6, 1, 1, 128, 128, True),
    ("lightning", 6, 4, 1, 64, 64, False), ("lightning", 4, 4, 1, 64, 64, True), ("lightning", 16, 4, 1, 128, 128, False),
    ("lightning", 16, 5, 1, 128, 128, True)])
def test_which_portions_the_tcgen05_recurrences_pay_for(library, chunks, heads, num_seqs, d, dv, pays):
    f = getattr(build.load_library(library), f"rllm_{library}_tcgen05_pays")
    assert bool(f(chunks, heads, num_seqs, d, dv)) is pays


def test_the_recurrences_are_told_how_many_tokens_decode(monkeypatch):
    """Their scans walk those apart from the portions that are cut into chunks."""
    from types import SimpleNamespace

    from rllm_b200.parts import lightning, state_space
    seen = []

    def scan(*a, num_decode, **k):
        seen.append(num_decode)
        return torch.zeros(7, 8)
    for module in (lightning, state_space):
        monkeypatch.setattr(module, "linear", lambda x, w, **k: torch.zeros(7, 64))
    for name in ("lightning_scan", "ssd_scan"):
        monkeypatch.setattr(ops, name, scan)
    for name in ("gated_rmsnorm", "silu_gated_group_rmsnorm", "causal_conv"):
        monkeypatch.setattr(ops, name, lambda *a, **k: None)
    ctx = SimpleNamespace(q_start=None, state_slots=None, token_seq=None, num_seqs=4, num_tokens=7, num_decode=3, err=None, max_q_len=4)
    a = lightning.LightningAttention.__new__(lightning.LightningAttention)
    a.heads, a.d, a.dv, a.eps, a.w_in, a.w_o, a.w_norm, a.decay_dev = 2, 4, 4, 0.0, None, None, None, None
    a.forward(torch.zeros(7, 8), ctx, SimpleNamespace(state=None))
    b = state_space.StateSpace.__new__(state_space.StateSpace)
    b.__dict__.update(w={k: None for k in ("dt", "conv", "conv_bias", "dt_bias", "a_log", "d", "norm", "o")}, inner=8, heads=2, groups=1, state=4,
                      dv=4, eps=0.0, norm_groups=1, w_in=None)
    b.forward(torch.zeros(7, 8), ctx, (SimpleNamespace(state=None),) * 2)
    assert seen == [3, 3]

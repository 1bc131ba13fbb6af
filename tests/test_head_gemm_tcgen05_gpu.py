"""The products per head on the tcgen05 kernel: strided slices, remainders of tiles in rows, columns and k, every tile
width; what lies beside a slice of the result stays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,heads,ka,K,N,wide", [(2048, 16, 192, 128, 512, 576), (1025, 16, 512, 512, 128, 128), (700, 30, 40, 24, 104, 117),
                                                 (129, 128, 72, 72, 130, 132), (4097, 3, 64, 64, 190, 200)])
def test_products_per_head(M, heads, ka, K, N, wide, monkeypatch):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    a = torch.randn(M, heads, ka, generator=g, device="cuda").bfloat16()[:, :, :K]
    b = (torch.randn(heads, N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    full = torch.full((M, heads, wide), 7.0, device="cuda").bfloat16()
    assert M * heads * N >= ops.HEAD_GEMM_TCGEN05_FROM and ops.head_gemm_tcgen05_takes(a, b, full[:, :, :N])
    ops.head_gemm(a, b, full[:, :, :N], b_kn=False)
    ops.check_gemm_errors(a.device)
    want = torch.einsum("mhk,hnk->mhn", a.double(), b.double())
    size = torch.einsum("mhk,hnk->mhn", a.double().abs(), b.double().abs())
    # one rounding to bfloat16 (2^-8 of the result) and float32 sums over K terms
    assert bool(((full[:, :, :N].double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * size).all())
    assert bool((full[:, :, N:] == 7.0).all())
    assert not ops.head_gemm_tcgen05_takes(a.float(), b.float(), full)
    monkeypatch.setenv("RLLM_GEMM", "no_tcgen05")
    assert not ops.head_gemm_tcgen05_takes(a, b, full)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,heads,dim,rot,turns,kv", [(5, 3, 10, 6, 2, 22), (33, 16, 128, 64, 64, 512), (2, 7, 8, 600, 598, 16), (9, 1, 4, 2, 0, 8)])
def test_rotation_of_the_queries_part(dtype, T, heads, dim, rot, turns, kv):
    """More pairs than a block has threads, fewer, one head, none that turns."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(rot)
    q = torch.randn(T, heads, dim + rot, generator=g, device="cuda").to(dtype)
    qt = torch.full((T, heads, kv + rot), 7.0, device="cuda", dtype=dtype)
    pos = torch.randint(0, 5000, (T,), generator=g, device="cuda", dtype=torch.int32)
    f = torch.rand(max(turns // 2, 1), generator=g, device="cuda", dtype=torch.float64)
    ops.latent_q_rot(q.view(T, -1), qt.view(T, -1), pos, f, heads, dim, rot, turns, kv, magnitude=1.25)
    part = q[:, :, dim:].double()
    a = pos.double()[:, None] * f[: turns // 2]
    c, s = (1.25 * torch.cos(a))[:, None], (1.25 * torch.sin(a))[:, None]
    u, v = part[..., :turns:2], part[..., 1:turns:2]
    want = part.clone()
    want[..., :turns:2], want[..., 1:turns:2] = u * c - v * s, v * c + u * s
    # rounded once to the type; the angle's cosine is good to about 1e-6 in float32
    tol = 2.0 ** -8 if dtype is torch.bfloat16 else 4e-6
    assert bool(((qt[:, :, kv:].double() - want).abs() <= tol * want.abs() + 1e-5).all())
    assert bool((qt[:, :, :kv] == 7.0).all())


@pytest.mark.parametrize("form", ["one row for all", "one head for all", "rows that overlap"])
def test_products_of_rows_that_share_memory(form):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    M, heads, K, N = 2048, 16, 128, 128
    if form == "rows that overlap":
        a = torch.randn(M * 64 + heads * 8192 * 2, generator=g, device="cuda").bfloat16().as_strided((M, heads, K), (64, 8192, 1))
    else:
        a = torch.randn(M, heads, K, generator=g, device="cuda").bfloat16()
        a = a[:1].expand(M, heads, K) if form == "one row for all" else a[:, :1].expand(M, heads, K)
    b, c = torch.randn(heads, N, K, generator=g, device="cuda").bfloat16(), torch.empty(M, heads, N, device="cuda").bfloat16()
    ops.head_gemm(a, b, c, b_kn=False)
    ops.check_gemm_errors(a.device)
    want = torch.einsum("mhk,hnk->mhn", a.double(), b.double())
    size = torch.einsum("mhk,hnk->mhn", a.double().abs(), b.double().abs())
    assert bool(((c.double() - want).abs() <= 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * size).all())


@pytest.mark.parametrize("T,heads,rot,turns", [(255, 16, 64, 64), (256, 16, 64, 48), (256, 31, 32, 32), (256, 33, 32, 32), (300, 3, 600, 598)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotation_has_the_same_bits_a_token_at_a_time(dtype, T, heads, rot, turns):
    """Around the size from which a block takes a token: a token alone is rotated a thread a pair."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(T + heads)
    q = torch.randn(T, heads * (8 + rot), generator=g, device="cuda").to(dtype)
    pos = torch.randint(0, 9000, (T,), generator=g, device="cuda", dtype=torch.int32)
    f = torch.rand(turns // 2, generator=g, device="cuda", dtype=torch.float64)
    many, one = (torch.full((T, heads * (16 + rot)), 7.0, device="cuda", dtype=dtype) for _ in range(2))
    ops.latent_q_rot(q, many, pos, f, heads, 8, rot, turns, 16, magnitude=0.75)
    for t in range(0, T, 5):
        ops.latent_q_rot(q[t: t + 1], one[t: t + 1], pos[t: t + 1], f, heads, 8, rot, turns, 16, magnitude=0.75)
        assert torch.equal(one[t], many[t])
    assert bool((many.view(T, heads, -1)[:, :, :16] == 7.0).all())

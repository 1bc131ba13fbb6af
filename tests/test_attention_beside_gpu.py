"""Prompts' attention on tcgen05 beside that of tokens which decode: the same bits as one behind the other, also for what
reads the result next, whichever of the two takes longer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("decode,prompts", [([5000, 17, 9000], [40]), ([33], [900, 300]), ([700] * 7, [200]), ([12000] * 3, [64, 3])])
def test_two_attentions_side_by_side(decode, prompts, d):
    from test_parts_gpu import DEV, context_for, load_part

    from rllm_b200.cache import CacheStorage
    from rllm_b200.kernels import ops
    from rllm_b200.models.decoder import CacheLayout
    from rllm_b200.parts import PartSpec, build_part
    hidden, nq, nkv, dt = 256, 8, 2, torch.bfloat16
    names = {k: k for k in "qkvo"}
    spec = PartSpec.of("attention", tensor_names=names, hidden_size=hidden, num_heads=nq, num_kv_heads=nkv, head_dim=d, window=None,
                       position=PartSpec.of("rotary", head_dim=d, rotary_dim=d, theta=5000.0, scaling=None, interleaved=False))
    part = build_part("mixer", spec)
    load_part(part, dt)
    entries = [(f"d{i}", [0], n) for i, n in enumerate(decode)] + [(f"p{i}", [0] * n, 0) for i, n in enumerate(prompts)]
    pages = sum(-(-(n + 1) // 16) for n in decode) + sum(-(-n // 16) for n in prompts) + 4
    storage = CacheStorage(CacheLayout([part.cache_need()], [[0]], [0], [0]), 16, [pages], len(entries), dt, DEV)
    ctx, cache = context_for([part.cache_need()], 16, pages, entries, dt)
    g = torch.Generator(device="cuda")
    g.manual_seed(d + len(decode))
    view = storage.view(0)
    view.k.copy_(torch.randn(view.k.shape, generator=g, device="cuda"))
    view.v.copy_(torch.randn(view.v.shape, generator=g, device="cuda"))
    x = torch.randn(ctx.num_tokens, hidden, generator=g, device="cuda").to(dt)
    assert ctx.num_decode == len(decode)
    real, sides = ops.attention_prefill_tcgen05, []

    def behind(*a, beside_decode=False, **k):
        sides.append(beside_decode)
        real(*a, **k)
    ops.attention_prefill_tcgen05 = behind
    try:
        want = part.forward(x, ctx, view).clone()
    finally:
        ops.attention_prefill_tcgen05 = real
    assert sides == [True]
    torch.cuda.synchronize()
    for _ in range(30):                                    # the layer again and again, nothing waited for in between
        got = part.forward(x, ctx, view)
        assert torch.equal(got, want)
    assert int(ctx.err.item()) == 0

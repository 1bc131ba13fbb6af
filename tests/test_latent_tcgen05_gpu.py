"""Attention of prompt portions over latent rows on the tcgen05 kernel against float64: rows of one to nine panels (with
one set of value panels and two, with values in one part and two), heads that do and do not divide a tile of 128 rows,
every page size, windows whose old pages are gone, sinks, several sequences of which the first are another kernel's, and
cache rows that no token has written (NaN)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,news,first,heads,dk,dv,page,window,sink", [
    ([83, 41, 190], [50, 7, 190], 0, 16, 576, 512, 16, 0, True), ([129, 64, 65], [1, 64, 65], 1, 16, 576, 512, 16, 0, False),
    ([700], [65], 0, 16, 576, 512, 16, 100, True), ([300], [120], 0, 8, 288, 256, 16, 0, True),
    ([83, 41], [50, 19], 0, 3, 56, 48, 16, 0, True), ([129, 64], [129, 64], 0, 5, 144, 128, 8, 33, False),
    ([90], [90], 0, 1, 40, 40, 16, 1, False), ([150, 260], [140, 33], 0, 2, 304, 264, 16, 0, False),
    ([150], [150], 0, 20, 96, 64, 32, 0, True), ([500], [70], 0, 7, 512, 512, 64, 0, False),
    ([257], [200], 0, 16, 448, 392, 4, 77, True), ([64], [64], 0, 128, 384, 320, 16, 0, True), ([33], [33], 0, 200, 64, 64, 128, 0, False)])
def test_latent_attention_on_tcgen05(lens, news, first, heads, dk, dv, page, window, sink):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk + heads)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    S, T = len(lens), sum(news)
    pages = sum(-(-n // page) for n in lens)
    order = torch.randperm(pages + 2, generator=g, device="cuda").tolist()
    cache = torch.full((pages + 2, 1, page, dk), float("nan"), dtype=torch.bfloat16, device="cuda")
    table = torch.full((S, max(-(-n // page) for n in lens)), -1, dtype=torch.int32)
    rows = []
    for s, n in enumerate(lens):
        r = randn(n, dk).bfloat16()
        rows.append(r.double())
        for b in range(-(-n // page)):
            if window and (b + 1) * page <= n - news[s] - window + 1:
                continue                                       # given back: no query of this step sees it
            table[s, b] = order.pop()
            m = min(page, n - b * page)
            cache[table[s, b], 0, :m] = r[b * page: b * page + m]
    q = randn(T, heads * dk).bfloat16()
    sk = randn(heads) + 1.0 if sink else None
    starts = [0]
    for m in news:
        starts.append(starts[-1] + m)
    out = torch.full((T, heads * dv), 7.0, dtype=torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.latent_attention_tcgen05(q, out, cache, table.cuda(), torch.tensor(starts, dtype=torch.int32, device="cuda"),
                                 torch.tensor(lens, dtype=torch.int32, device="cuda"), first, S, T - starts[first], heads, dk,
                                 dv, window, dk ** -0.5, sk, err)
    assert int(err.item()) == 0
    assert bool((out[: starts[first]] == 7.0).all())
    for s in range(first, S):
        n, m = lens[s], news[s]
        pos, key = torch.arange(n - m, n, device="cuda")[:, None], torch.arange(n, device="cuda")
        hidden = (key > pos) | ((key <= pos - window) if window else (key < 0))
        for h in range(heads):
            sc = q[starts[s]: starts[s + 1], h * dk: (h + 1) * dk].double() @ rows[s].t() * dk ** -0.5
            sc = sc.masked_fill(hidden, -math.inf)
            if sink:
                sc = torch.cat([sc, sk[h].double().expand(m, 1)], 1)
            p = torch.softmax(sc, 1)[:, :n]
            want = p @ rows[s][:, :dv]
            got = out[starts[s]: starts[s + 1], h * dv: (h + 1) * dv].double()
            # weights and the result are each rounded once to bfloat16, by at most 2^-8 of themselves (a significand of 8
            # bits): together 2^-7 of the sum of the terms' sizes, beside which the float32 sums and exponentials are small
            bound = 2.0 ** -7 * (p @ rows[s][:, :dv].abs()) + 1e-5
            assert bool(((got - want).abs() <= bound).all()), (s, h, float(((got - want).abs() / bound).max()))


def test_which_prompt_portions_take_the_tcgen05_latent_attention(monkeypatch):
    from rllm_b200.kernels import ops
    c = torch.zeros(2, 1, 16, 576, dtype=torch.bfloat16, device="cuda")
    assert ops.latent_attention_tcgen05_takes(torch.bfloat16, 576, 512, 1024, c)
    assert not ops.latent_attention_tcgen05_takes(torch.bfloat16, 576, 512, 1023, c)
    assert not ops.latent_attention_tcgen05_takes(torch.float32, 576, 512, 4096, c)
    assert not ops.latent_attention_tcgen05_takes(torch.bfloat16, 584, 512, 4096, c)
    assert not ops.latent_attention_tcgen05_takes(torch.bfloat16, 300, 260, 4096, c)
    assert not ops.latent_attention_tcgen05_takes(torch.bfloat16, 576, 512, 4096, c.view(-1)[4:])
    monkeypatch.setenv("RLLM_LATENT_ATTENTION", "mma")
    assert not ops.latent_attention_tcgen05_takes(torch.bfloat16, 576, 512, 4096, c)


@pytest.mark.parametrize("heads,dk,dv,window", [(16, 576, 512, 100), (8, 288, 256, 40), (128, 144, 128, 1)])
def test_rows_that_the_window_hides_do_not_reach_the_output(heads, dk, dv, window):
    """Rows behind every query's window that still have their page hold infinities and NaN."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(dk)
    n, m, page = 300, 24, 16
    first = n - m - window + 1                             # the oldest key that the oldest query sees
    rows = torch.randn(n, dk, generator=g, device="cuda").bfloat16()
    cache = torch.zeros(-(-n // page), 1, page, dk, dtype=torch.bfloat16, device="cuda")
    cache.view(-1, dk)[:n] = rows
    cache.view(-1, dk)[:first] = math.inf
    cache.view(-1, dk)[:first:3] = math.nan
    table = torch.arange(cache.shape[0], dtype=torch.int32, device="cuda")[None].contiguous()
    q = torch.randn(m, heads * dk, generator=g, device="cuda").bfloat16()
    out, err = torch.empty(m, heads * dv, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.latent_attention_tcgen05(q, out, cache, table, torch.tensor([0, m], dtype=torch.int32, device="cuda"),
                                 torch.tensor([n], dtype=torch.int32, device="cuda"), 0, 1, m, heads, dk, dv, window, dk ** -0.5,
                                 None, err)
    assert int(err) == 0
    pos, key = torch.arange(n - m, n, device="cuda")[:, None], torch.arange(n, device="cuda")
    hidden = (key > pos) | (key <= pos - window)
    sc = torch.einsum("mhd,kd->hmk", q.view(m, heads, dk).double(), rows.double()) * dk ** -0.5
    p = torch.softmax(sc.masked_fill(hidden, -math.inf), 2)
    want, size = p @ rows[:, :dv].double(), p @ rows[:, :dv].double().abs()
    got = out.view(m, heads, dv).transpose(0, 1).double()
    assert bool(((got - want).abs() <= 2.0 ** -7 * size + 1e-5).all())       # the bound of the test above


@pytest.mark.parametrize("window,sink", [(None, False), (37, True), (None, True)])
def test_a_step_of_decoded_tokens_and_prompts_through_the_mixer(window, sink, monkeypatch):
    """The part alone: prompts first, then a step in which three requests decode beside two portions, one of them behind
    rows of an earlier step.  The portions run on tcgen05, the decoded tokens on mma.sync."""
    from test_parts_gpu import DEV, context_for, load_part

    from rllm_b200.cache import CacheStorage
    from rllm_b200.kernels import ops
    from rllm_b200.models.decoder import CacheLayout
    from rllm_b200.parts import PartSpec, build_part
    hidden, H, nope, rot, vdim, kv, dt = 96, 32, 24, 16, 40, 64, torch.bfloat16
    names = {k: k for k in ("dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "sink", "o")}
    spec = PartSpec.of("latent_attention", tensor_names=names, hidden_size=hidden, num_heads=H, nope_dim=nope, rot_dim=rot,
                       v_dim=vdim, q_rank=56, kv_rank=kv, scale=(nope + rot) ** -0.5, eps=1e-6, window=window, sink=sink,
                       position=PartSpec.of("rotary", head_dim=rot, rotary_dim=rot, theta=5000.0, scaling=None, interleaved=True))
    part = build_part("mixer", spec)
    w = load_part(part, dt)
    storage = CacheStorage(CacheLayout([part.cache_need()], [[0]], [0], [0]), 16, [64], 8, dt, DEV)
    torch.manual_seed(3)
    before, new = {"a": 70, "b": 9, "c": 130, "d": 50, "e": 0}, {"a": 1, "b": 1, "c": 1, "d": 64, "e": 41}
    xs = {r: (torch.randn(before[r] + new[r], hidden) * 2).to(dt) for r in before}
    ctx, cache = context_for([part.cache_need()], 16, 64, [(r, [0] * n, 0) for r, n in before.items() if n], dt)
    part.forward(torch.cat([xs[r][: before[r]] for r in "abcd"]).to(DEV), ctx, storage.view(0))
    ran = []
    for name in ("latent_attention_tcgen05", "latent_attention_mma"):
        real = getattr(ops, name)
        monkeypatch.setattr(ops, name, lambda *a, _f=real, _n=name, **k: (ran.append(_n), _f(*a, **k))[1])
    ctx, cache = context_for([part.cache_need()], 16, 64, [(r, [0] * n, before[r]) for r, n in new.items()], dt, cache)
    assert ctx.num_decode == 3
    got = part.forward(torch.cat([xs[r][before[r]:] for r in new]).to(DEV), ctx, storage.view(0)).double().cpu()
    assert ran == ["latent_attention_tcgen05", "latent_attention_mma"] and int(ctx.err.item()) == 0

    def norm(x, g):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * g

    def turn(x, pos):                                      # pairs (2 i, 2 i + 1)
        a = pos[:, None] * 5000.0 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / rot)
        c, s = a.cos().view(len(pos), *([1] * (x.ndim - 2)), -1), a.sin().view(len(pos), *([1] * (x.ndim - 2)), -1)
        u, v = x[..., ::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    at = 0
    for r, m in new.items():
        x, n = xs[r].double(), before[r] + m
        pos = torch.arange(n, dtype=torch.float64)
        q = (norm(x @ w["dq"].t(), w["dq_norm"]) @ w["uq"].t()).view(n, H, nope + rot)
        a = x @ w["dkv"].t()
        rows = torch.cat([norm(a[:, :kv], w["dkv_norm"]), turn(a[:, kv:], pos)], 1)
        qt = torch.cat([torch.einsum("thn,hnk->thk", q[..., :nope], w["uk"].view(H, nope, kv)), turn(q[..., nope:], pos)], 2)
        sc = torch.einsum("thk,jk->htj", qt, rows) * (nope + rot) ** -0.5
        hidden_keys = pos[None] > pos[:, None]
        if window:
            hidden_keys |= pos[None] <= pos[:, None] - window
        sc = sc.masked_fill(hidden_keys, -math.inf)
        if sink:
            sc = torch.cat([sc, w["sink"].view(H, 1, 1).expand(H, n, 1)], 2)
        o = torch.einsum("htj,jk->thk", torch.softmax(sc, 2)[:, :, :n], rows[:, :kv])
        want = torch.einsum("thk,hvk->thv", o, w["uv"].view(H, vdim, kv)).reshape(n, H * vdim) @ w["o"].t()
        # a dozen roundings to bfloat16 one after the other, as the parts' other tests allow for: 2 % of the largest result
        assert float((got[at: at + m] - want[before[r]:]).abs().max()) <= 2e-2 * float(want.abs().max()), r
        at += m

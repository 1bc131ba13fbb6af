"""Latent attention of prompt portions with every head's own keys and values, against float64: both widths of the heads'
parts, shared parts that do not fill a panel, portions around the tiles' edges, rows of an earlier step, windows whose old
pages are gone, sinks, several sequences of which the first are another kernel's, cache rows that no token has written or
that only other queries see (NaN, infinities)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,news,first,heads,nope,rot,v,kv,page,window,sink", [
    ([83, 41, 190], [50, 7, 190], 0, 4, 128, 64, 128, 512, 16, 0, True), ([129, 64, 65], [1, 64, 65], 1, 3, 128, 64, 128, 96, 16, 0, False),
    ([700], [65], 0, 2, 128, 32, 64, 256, 16, 100, True), ([300], [128], 0, 2, 64, 32, 64, 256, 16, 0, True),
    ([383, 941], [129, 127], 0, 3, 64, 8, 64, 40, 8, 33, False), ([257, 130], [257, 2], 0, 2, 64, 24, 128, 64, 32, 0, True),
    ([640, 64, 900], [300, 64, 513], 0, 1, 64, 64, 64, 128, 64, 300, False), ([1], [1], 0, 2, 128, 64, 64, 72, 16, 0, False),
    ([512, 515], [256, 3], 0, 5, 128, 40, 128, 512, 128, 1, True)])
def test_prompt_portions_with_every_heads_own_keys_and_values(lens, news, first, heads, nope, rot, v, kv, page, window, sink):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(nope + heads + kv)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    S, T, dk = len(lens), sum(news), kv + rot
    pages = sum(-(-n // page) for n in lens)
    order = torch.randperm(pages + 2, generator=g, device="cuda").tolist()
    cache = torch.full((pages + 2, 1, page, dk), float("nan"), dtype=torch.bfloat16, device="cuda")
    table = torch.full((S, max(-(-n // page) for n in lens)), -1, dtype=torch.int32)
    rows = []
    for s, n in enumerate(lens):
        r = randn(n, dk).bfloat16()
        seen = max(0, n - news[s] - window + 1) if window else 0      # the oldest key that a query of this step sees
        r[: seen] = math.inf
        rows.append(r)
        for b in range(-(-n // page)):
            if b % 2 and (b + 1) * page <= seen:
                continue                                       # given back
            table[s, b] = order.pop()
            m = min(page, n - b * page)
            cache[table[s, b], 0, :m] = r[b * page: b * page + m]
    starts = [0]
    for m in news:
        starts.append(starts[-1] + m)
    q = randn(T, heads * (nope + rot)).bfloat16()
    turned, pos = q.clone(), torch.cat([torch.arange(n - m, n, dtype=torch.int32) for n, m in zip(lens, news)]).cuda()
    dims = rot - rot % 16
    freq = torch.rand(max(dims // 2, 1), generator=g, device="cuda", dtype=torch.float64)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    q_start, seq_lens, dtable, err = i32(starts), i32(lens), table.cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    n = ops.latent_expanded_rows(news[first:], lens[first:], window)
    got_rows = torch.full((n, dk), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.latent_expand_prep(turned, cache, got_rows, dtable, q_start, seq_lens, first, S, pos, freq if dims else None,
                           starts[first], heads, nope, rot, dims, window, err, magnitude=1.25)
    # the queries: the bits of the rotation that the other form has
    want_q = q.clone()
    ops.latent_q_rot(q, want_q, pos, freq if dims else None, heads, nope, rot, dims, nope, magnitude=1.25)
    want_q[: starts[first]] = q[: starts[first]]
    assert torch.equal(turned, want_q)
    at = 0
    bases = {}
    for s in range(first, S):
        seen = max(0, lens[s] - news[s] - window + 1) if window else 0
        lo = seen // 128 * 128
        want = rows[s][lo:].clone()
        want[: seen - lo] = 0
        assert torch.equal(got_rows[at: at + lens[s] - lo], want)
        bases[s] = at - lo
        at += lens[s] - lo
    assert at == n
    wkv = (randn(heads * (nope + v), kv) * kv ** -0.5).bfloat16()
    kvs = torch.empty(n, heads * (nope + v), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05(got_rows[:, :kv], wkv, kvs)
    sk = randn(heads) + 1.0 if sink else None
    out = torch.full((T, heads * v), 7.0, dtype=torch.bfloat16, device="cuda")
    scale = (nope + rot) ** -0.5
    ops.latent_expanded_tcgen05(turned, kvs, got_rows, out, q_start, seq_lens, first, S, T - starts[first], heads, nope, rot, v,
                                kv, window, scale, sk, err)
    assert int(err.item()) == 0
    ops.check_gemm_errors(out.device)
    assert bool((out[: starts[first]] == 7.0).all())
    for s in range(first, S):
        ln, m = lens[s], news[s]
        p0 = max(0, ln - m - window + 1) if window else 0
        p, key = torch.arange(ln - m, ln, device="cuda")[:, None], torch.arange(p0, ln, device="cuda")
        hidden = (key > p) | ((key <= p - window) if window else (key < 0))
        mine = slice(bases[s] + p0, bases[s] + ln)
        for h in range(heads):
            k = torch.cat([kvs[mine, h * nope: (h + 1) * nope], got_rows[mine, kv:]], 1).double()
            val = kvs[mine, heads * nope + h * v: heads * nope + (h + 1) * v].double()
            sc = turned[starts[s]: starts[s + 1], h * (nope + rot): (h + 1) * (nope + rot)].double() @ k.t() * scale
            sc = sc.masked_fill(hidden, -math.inf)
            if sink:
                sc = torch.cat([sc, sk[h].double().expand(m, 1)], 1)
            w = torch.softmax(sc, 1)[:, : ln - p0]
            want = w @ val
            got = out[starts[s]: starts[s + 1], h * v: (h + 1) * v].double()
            # weights and the result are each rounded once to bfloat16, by at most 2^-8 of themselves: together 2^-7 of the
            # sum of the terms' sizes, beside which the float32 sums and exponentials are small
            bound = 2.0 ** -7 * (w @ val.abs()) + 1e-5
            assert bool(((got - want).abs() <= bound).all()), (s, h, float(((got - want).abs() / bound).max()))


def test_another_sequences_rows_do_not_reach_the_output():
    """The next sequence's rows, in the last tile of keys of the one before."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    lens, heads, nope, rot, v, kv = [200, 70], 2, 128, 64, 128, 64
    n, dk = sum(lens), kv + rot
    rows = torch.randn(n, dk, generator=g, device="cuda").bfloat16()
    kvs = torch.randn(n, heads * (nope + v), generator=g, device="cuda").bfloat16()
    q = torch.randn(n, heads * (nope + rot), generator=g, device="cuda").bfloat16()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")  # noqa: E731
    call = lambda o, e: ops.latent_expanded_tcgen05(q, kvs, rows, o, i32([0, 200, 270]), i32(lens), 0, 2, n, heads, nope, rot, v, kv,  # noqa: E731
                                                    0, 0.07, None, e)
    clean, dirty = (torch.empty(n, heads * v, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    call(clean, err)
    kvs[200:] = math.nan
    rows[201:] = math.inf
    call(dirty, err)
    assert int(err) == 0 and torch.equal(clean[:200], dirty[:200])

"""The CUDA-core attention with one warp a row and with eight: a row has the same bits in a batch of many rows as alone, at
the edges of the 128-key parts, with windows, kept keys, chunks and sinks; and float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 128), (40, 72), (48, 256)])
@pytest.mark.parametrize("opts", [dict(), dict(window=200), dict(window=130, keep_first=5), dict(chunk=150), dict(window=300, keep_first=140, chunk=400)])
def test_a_row_alone_and_among_many(d, dv, opts):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(d + dv)
    n, page, nq, nkv = 700, 16, 8, 2
    pages = -(-n // page)
    k = torch.randn(pages, nkv, page, d, generator=g, device="cuda")
    v = torch.randn(pages, nkv, page, dv, generator=g, device="cuda")
    table = torch.randperm(pages, generator=g, device="cuda").int()[None].contiguous()
    q = torch.randn(n, nq * d, generator=g, device="cuda")
    sinks = torch.randn(nq, generator=g, device="cuda") if opts.get("keep_first") else None
    pos, seq = torch.arange(n, device="cuda", dtype=torch.int32), torch.zeros(n, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(a, b):
        out = torch.empty(b - a, nq * dv, device="cuda")
        o = dict(opts)
        ops.attention_simt_kv(q[a:b], nq * d, out, k, v, table, pos[a:b], seq[a:b], nq, nkv, o.pop("window", 0), d ** -0.5, err,
                              sinks=sinks, **o)
        return out

    many = run(0, n)                                        # 5,600 rows: a warp each
    for p in (0, 1, 31, 32, 126, 127, 128, 129, 255, 256, 300, 511, 512, 699):
        assert torch.equal(run(p, p + 1)[0], many[p])       # eight rows: eight warps each
    assert int(err) == 0
    keys, vals = (x[table[0].long()].transpose(1, 2).reshape(-1, nkv, x.shape[3])[:n].double() for x in (k, v))
    j, p = torch.arange(n, device="cuda")[None], torch.arange(n, device="cuda")[:, None]
    seen = j <= p
    if opts.get("window"):
        seen &= (j > p - opts["window"]) | (j < opts.get("keep_first", 0))
    if opts.get("chunk"):
        seen &= j // opts["chunk"] == p // opts["chunk"]
    for h in range(nq):
        s = q[:, h * d: (h + 1) * d].double() @ keys[:, h // 4].t() * d ** -0.5
        s = s.masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
        w = torch.softmax(s, 1)[:, :n]
        want, size = w @ vals[:, h // 4], w @ vals[:, h // 4].abs()
        # a score is a sum of d float32 products (some d 2^-24 of its size), which its weight takes over; then as many sums
        assert bool(((many[:, h * dv: (h + 1) * dv].double() - want).abs() <= 3e-5 * size + 1e-7).all())


@pytest.mark.parametrize("d", [64, 40])
@pytest.mark.parametrize("bad,seen", [((256, 257), 257), ((128, 256), 300), ((384, 400), 400), ((130, 131), 200)])
def test_a_key_that_is_not_a_number_shows_in_the_result(d, bad, seen):
    """NaN scores that fill a part of 128 keys, or all of a part that the row sees, behind a part of numbers."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(d + seen)
    page, nq = 16, 4
    pages = 64
    k, v = (torch.randn(pages, 1, page, d, generator=g, device="cuda") for _ in range(2))
    k.view(-1, d)[bad[0]: bad[1]] = math.nan
    table = torch.arange(pages, dtype=torch.int32, device="cuda")[None].contiguous()
    for rows in (1, 1100):                                  # eight warps a row (the table is wide), and one
        q = torch.randn(rows, nq * d, generator=g, device="cuda")
        out, err = torch.zeros(rows, nq * d, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        pos = torch.full((rows,), seen - 1, dtype=torch.int32, device="cuda")
        ops.attention_simt_kv(q, nq * d, out, k, v, table, pos, torch.zeros_like(pos), nq, 1, 0, d ** -0.5, err)
        assert int(err) == 0 and bool(torch.isnan(out).all())
        pos.fill_(bad[0] - 1)                               # and does not where the key lies ahead
        ops.attention_simt_kv(q, nq * d, out, k, v, table, pos, torch.zeros_like(pos), nq, 1, 0, d ** -0.5, err)
        assert bool(torch.isfinite(out).all())

"""The kernels that take eight (the convolution: four) values an access, at the sizes and alignments where they begin and
end, against float64 and against the forms with single values, which rows that start elsewhere still take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device="cuda")


def close(got, want, size):
    # one rounding to bfloat16 (at most 2^-8 of the result) and a few of float32
    return bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5 * size + 1e-7).all())


@pytest.mark.parametrize("T,H,pad,wd", [(5, 8, 0, "float32"), (3, 2048, 8, "float32"), (2, 8192, 16, "bfloat16"), (2, 8200, 8, "float32"),
                                        (4, 264, 3, "float32"), (1, 1000, 8, "bfloat16")])
def test_gated_rmsnorm_rows(T, H, pad, wd):
    from rllm_b200.kernels import ops
    r = gen(H + pad)
    x, w = r(T, H) * 3, (1 + 0.1 * r(H)).to(getattr(torch, wd))
    g = r(T, H + pad).bfloat16()[:, pad:]
    got = ops.gated_rmsnorm(x, g, w, 1e-5, torch.bfloat16)
    want = x.double() * torch.rsqrt(x.double().square().mean(1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(g.double())
    assert close(got, want, 4.0)


@pytest.mark.parametrize("T,E,groups,pad", [(3, 4096, 2, 8), (5, 64, 4, 0), (2, 8192, 1, 8), (2, 16400, 2, 8), (3, 96, 3, 5), (2, 20, 5, 4)])
def test_silu_gated_group_rmsnorm_rows(T, E, groups, pad):
    from rllm_b200.kernels import ops
    r = gen(E + pad)
    y, w = r(T, E) * 2, 1 + 0.1 * r(E)
    z = r(T, E + pad).bfloat16()[:, pad:]
    got = ops.silu_gated_group_rmsnorm(y, z, w, 1e-5, groups, torch.bfloat16)
    v = (y.double() * torch.nn.functional.silu(z.double())).view(T, groups, -1)
    want = (v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5)).view(T, E) * w.double()
    assert close(got, want, 8.0)


@pytest.mark.parametrize("T,K,H", [(1, 1, 8), (7, 4, 2048), (33, 5, 264), (9, 2, 100)])
@pytest.mark.parametrize("extra", ["none", "row", "gated"])
def test_weighted_sum_of_slots(T, K, H, extra):
    from rllm_b200.kernels import ops
    r = gen(T + H)
    y, c, e, g = r(T * K, H).bfloat16(), r(T, K), r(T, H).bfloat16(), r(T)
    out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    ops.weighted_slot_sum(y, c, out, extra=None if extra == "none" else e, extra_gate=g if extra == "gated" else None)
    want = torch.einsum("tk,tkh->th", c.double(), y.double().view(T, K, H))
    if extra != "none":
        want = want + e.double() * (torch.sigmoid(g.double())[:, None] if extra == "gated" else 1.0)
    assert close(out, want, 4.0 * K)


@pytest.mark.parametrize("P,E", [(1, 1), (31, 3), (33, 40), (2048, 5), (8192, 32), (5000, 2048)])
@pytest.mark.parametrize("bm", [16, 64, 128])
def test_pairs_sorted_by_expert(P, E, bm):
    """Every pair once, within its expert's range, and tiles that cover the ranges."""
    from rllm_b200.kernels import build
    from rllm_b200.kernels.ops import _check, _ptr, _stream, c_int
    r = torch.Generator(device="cuda")
    r.manual_seed(P)
    ids = torch.randint(0, E, (P,), generator=r, device="cuda", dtype=torch.int32)
    most = min(P, -(-P // bm) + E)
    off, pairs, te, tr, n = (torch.full((k,), -1, dtype=torch.int32, device="cuda") for k in (E + 1, P, most, most, 1))
    _check(build.load_library("moe").rllm_moe_sort(_ptr(ids), c_int(P), c_int(E), c_int(bm), _ptr(off), _ptr(pairs), _ptr(te),
                                                   _ptr(tr), _ptr(n), _stream()), "moe_sort")
    count = torch.bincount(ids.long(), minlength=E)
    assert off.tolist() == [0] + count.cumsum(0).tolist()
    assert sorted(pairs.tolist()) == list(range(P)) and bool((ids[pairs.long()].diff() >= 0).all())
    at, off, te, tr = 0, off.tolist(), te.tolist(), tr.tolist()
    for e in range(E):
        rows, covered = [], off[e]
        while at < int(n) and te[at] == e:
            rows.append(tr[at])
            at += 1
        for i, r0 in enumerate(rows):
            end = rows[i + 1] if i + 1 < len(rows) else off[e + 1]
            assert r0 == covered and 0 < end - r0 <= bm
            covered = end
        assert covered == off[e + 1]
    assert at == int(n)


@pytest.mark.parametrize("lens", [[1], [8], [2, 1, 1, 30, 3], [9, 17], [64], [1, 7, 8, 1]])
@pytest.mark.parametrize("E,pad,bias", [(4, 0, True), (512, 4, True), (516, 8, False), (1028, 2, True)])
def test_convolution_of_prompt_portions(lens, E, pad, bias):
    """Runs of eight tokens within a sequence, across sequences and behind the last; tails that go on from before."""
    from rllm_b200.kernels import ops
    r = gen(E + sum(lens))
    T, S = sum(lens), len(lens)
    x = r(T, E + pad).bfloat16()[:, pad:]
    w, b = r(E, 4) * 0.4, r(E) * 0.1 if bias else None
    tail = r(S + 1, 3, E)
    starts = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(S, dtype=torch.int32), torch.tensor(lens)).cuda()
    slots = torch.arange(S, 0, -1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    new, at = tail.clone(), 0
    got = ops.causal_conv(x, w, b, new, starts, seq, slots, S, True, err)
    for s, n in enumerate(lens):
        past = torch.cat([tail[slots[s].long()].double(), x[at: at + n].double()])
        acc = sum(w[:, k].double() * past[k: k + n] for k in range(4)) + (b.double() if bias else 0.0)
        assert close(got[at: at + n], torch.nn.functional.silu(acc), 4.0)
        assert torch.equal(new[slots[s].long()], past[n:].float())
        at += n
    assert int(err) == 0 and torch.equal(new[0], tail[0])


def conv_of(x, w, b, tail, lens, any_long):
    from rllm_b200.kernels import ops
    S = len(lens)
    starts = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
    seq = torch.repeat_interleave(torch.arange(S, dtype=torch.int32), torch.tensor(lens)).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = ops.causal_conv(x, w, b, tail, starts, seq, torch.arange(S, dtype=torch.int32, device="cuda"), S, any_long, err)
    assert int(err) == 0
    return out


@pytest.mark.parametrize("E", [512, 4608])
def test_a_decoded_token_of_the_convolution_does_not_depend_on_its_batch(E):
    """The same bits in a step of decoded tokens and beside a prompt portion, and the portion the same bits whether its
    rows are read four channels at a time or one; sums of -100 to 100, where an exponential is least good."""
    r = gen(E)
    n = (1 << 22) // E                                     # a portion large enough for four channels a thread
    x, w, b = (r(5 + n, E) * 20).bfloat16(), r(E, 4), r(E) * 0.1
    alone, mixed, single = (r(6, 3, E) for _ in range(3))
    mixed.copy_(alone)
    single.copy_(alone)
    decoded = conv_of(x[:5], w, b, alone, [1] * 5, False)
    both = conv_of(x, w, b, mixed, [1] * 5 + [n], True)
    assert torch.equal(decoded, both[:5]) and torch.equal(alone[:5], mixed[:5])
    assert torch.equal(conv_of(shifted(x), w, b, single, [1] * 5 + [n], True), both) and torch.equal(single, mixed)
    assert float(both.float().min()) < -0.2 and float(both.float().max()) > 50


@pytest.mark.parametrize("lens", [[128], [2, 1, 1, 30, 3, 100], [9, 17, 103], [1, 7, 8, 1, 120], [5] * 3 + [1] + [113]])
def test_convolution_with_four_channels_a_thread(lens):
    """Runs of eight tokens within a sequence, across sequences and behind the last: the bits of the form with one channel."""
    r, E = gen(sum(lens)), 1 << 15
    x, w, b = r(sum(lens), E).bfloat16(), r(E, 4) * 0.4, r(E) * 0.1
    tail = r(len(lens) + 1, 3, E)
    four, one = tail.clone(), tail.clone()
    got = conv_of(x, w, b, four, lens, True)
    assert torch.equal(got, conv_of(shifted(x), w, b, one, lens, True)) and torch.equal(four, one)
    at = 0
    for s, n in enumerate(lens):
        past = torch.cat([tail[s].double(), x[at: at + n].double()])
        acc = sum(w[:, k].double() * past[k: k + n] for k in range(4)) + b.double()
        assert close(got[at: at + n], torch.nn.functional.silu(acc), 4.0)
        assert torch.equal(four[s], past[n:].float())
        at += n


def shifted(t):
    """The same rows one element further, where they no longer start on 16 bytes."""
    wide = torch.zeros(t.shape[0], t.shape[1] + 1, dtype=t.dtype, device="cuda")
    wide[:, 1:] = t
    return wide[:, 1:]


# gates at which an exponential or a reciprocal of fewer bits shows: e^-x large, near the largest float32, and past it
EDGES = (-5.0, -20.0, -60.0, -86.0, -88.0, -100.0, 20.0, 100.0)


@pytest.mark.parametrize("T,E,groups", [(3, 4096, 2), (7, 64, 4), (2, 8192, 1), (3, 360, 3), (33, 2048, 1)])
def test_group_rmsnorm_has_the_bits_of_its_single_value_form(T, E, groups):
    from rllm_b200.kernels import ops
    r = gen(E)
    y, z, w = r(T, E) * 2, (r(T, E) * 8).bfloat16(), 1 + 0.1 * r(E)
    for i, v in enumerate(EDGES):
        z[:, i::11] = v
    y[-1] *= 1e33                                          # a row whose small gates carry it
    z[-1] = -88.0
    got = ops.silu_gated_group_rmsnorm(y, z, w, 1e-5, groups, torch.bfloat16)
    assert torch.equal(got, ops.silu_gated_group_rmsnorm(y, shifted(z), w, 1e-5, groups, torch.bfloat16))
    v = (y.double() * torch.nn.functional.silu(z.double())).view(T, groups, -1)
    want = (v * torch.rsqrt(v.square().mean(-1, keepdim=True) + 1e-5)).view(T, E) * w.double()
    assert close(got, want, 8.0)


@pytest.mark.parametrize("T,H,wd", [(513, 1024, "float32"), (512, 1024, "float32"), (3, 2056, "float32"), (2, 8192, "bfloat16"), (33, 1032, "bfloat16")])
def test_gated_rmsnorm_has_the_bits_of_its_single_value_form(T, H, wd):
    from rllm_b200.kernels import ops
    r = gen(H)
    x, g, w = r(T, H) * 3, (r(T, H) * 8).bfloat16(), (1 + 0.1 * r(H)).to(getattr(torch, wd))
    for i, v in enumerate(EDGES):
        g[:, i::11] = v
    got = ops.gated_rmsnorm(x, g, w, 1e-5, torch.bfloat16)
    assert torch.equal(got, ops.gated_rmsnorm(x, shifted(g), w, 1e-5, torch.bfloat16))
    want = x.double() * torch.rsqrt(x.double().square().mean(1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(g.double())
    assert close(got, want, 4.0)


@pytest.mark.parametrize("heads,d,dv", [(3, 32, 64), (2, 64, 128), (2, 128, 128)])
def test_chunk_passes_have_the_same_bits_wherever_rows_start(heads, d, dv):
    """Rows on 16-byte boundaries (eight values a load), on 8-byte boundaries and on 4-byte boundaries."""
    from rllm_b200.kernels import ops
    r = gen(d + dv)
    T, cols = 1000, heads * (2 * d + dv)
    a = (r(T, cols) * 12).bfloat16()
    for i, v in enumerate(EDGES):
        a[:, i::13] = v
    outs = []
    for pad in (0, 4, 2):
        wide = torch.zeros(T, cols + pad, dtype=torch.bfloat16, device="cuda")
        wide[:, pad:] = a
        q, k, v = wide[:, pad: pad + heads * d], wide[:, pad + heads * d: pad + 2 * heads * d], wide[:, pad + 2 * heads * d:]
        state, err = r(1, heads, d, dv) * 0 + 0.5, torch.zeros(1, dtype=torch.int32, device="cuda")
        decay = torch.linspace(0.9, 0.99, heads, device="cuda")
        o = ops.lightning_scan(q, k, v, decay, state, torch.tensor([0, T], dtype=torch.int32, device="cuda"),
                               torch.zeros(1, dtype=torch.int32, device="cuda"), 1, err, max_q_len=T)
        assert int(err) == 0
        outs.append((o, state))
    for o, state in outs[1:]:
        assert torch.equal(o, outs[0][0]) and torch.equal(state, outs[0][1])


@pytest.mark.parametrize("T,K,H", [(64, 4, 2048), (63, 4, 2048), (497, 3, 264), (2048, 1, 64)])
@pytest.mark.parametrize("extra", ["none", "row", "gated"])
def test_weighted_sum_of_slots_has_the_same_bits_a_row_at_a_time(T, K, H, extra):
    """Around 2^17 results, from which eight values a thread are taken: a row alone takes single values."""
    from rllm_b200.kernels import ops
    r = gen(T + H)
    y, c, e, g = r(T * K, H).bfloat16(), r(T, K), r(T, H).bfloat16(), r(T)
    many, one = (torch.empty(T, H, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    opts = lambda a, b: dict(extra=None if extra == "none" else e[a:b], extra_gate=g[a:b] if extra == "gated" else None)  # noqa: E731
    ops.weighted_slot_sum(y, c, many, **opts(0, T))
    for t in range(T):
        ops.weighted_slot_sum(y[t * K: (t + 1) * K], c[t: t + 1], one[t: t + 1], **opts(t, t + 1))
    assert torch.equal(one, many)
    want = torch.einsum("tk,tkh->th", c.double(), y.double().view(T, K, H))
    if extra != "none":
        want = want + e.double() * (torch.sigmoid(g.double())[:, None] if extra == "gated" else 1.0)
    assert close(many, want, 4.0 * K)

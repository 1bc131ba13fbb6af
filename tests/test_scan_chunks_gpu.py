"""The recurrences over chunks of 128 tokens (states first, outputs after) against the token-by-token recurrence in float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def recurrence(q, k, v, decay, step, skip, state):
    """q, k [T, heads, d], v [T, heads, dv], decay and step [T, heads], state [heads, d, dv], all float64."""
    out = torch.empty_like(v)
    for t in range(len(v)):
        state = decay[t][:, None, None] * state + step[t][:, None, None] * k[t][:, :, None] * v[t][:, None, :]
        out[t] = (q[t][:, :, None] * state).sum(1) + skip[:, None] * v[t]
    return out, state


def inputs(steps, heads, groups, d, dv, T, seed):
    g = torch.Generator().manual_seed(seed)
    if steps:
        x = torch.randn(T, heads * dv + 2 * groups * d, generator=g).bfloat16()
        dt, bias, a_log, skip = (torch.randn(*s, generator=g) for s in ((T, heads), (heads,), (heads,), (heads,)))
        step = torch.nn.functional.softplus(dt.to(F64) + bias.to(F64))
        v, k, q = torch.split(x.to(F64), [heads * dv, groups * d, groups * d], 1)
        share = torch.arange(heads) // (heads // groups)
        return (x, dt, bias, a_log, skip), (q.view(T, groups, d)[:, share], k.view(T, groups, d)[:, share], v.view(T, heads, dv),
                                            torch.exp(-torch.exp(a_log.to(F64)) * step), step, skip.to(F64))
    a = torch.randn(T, heads * (2 * d + dv), generator=g).bfloat16()
    lam = torch.tensor(([1.0, 0.0, 0.97, 0.5] * heads)[:heads])
    act = torch.nn.functional.silu(a.to(F64)).float().bfloat16().to(F64)
    q, k, v = torch.split(act, [heads * d, heads * d, heads * dv], 1)
    return (a, lam), (q.view(T, heads, d), k.view(T, heads, d), v.view(T, heads, dv), lam.to(F64).expand(T, heads),
                      torch.ones(T, heads, dtype=F64), torch.zeros(heads, dtype=F64))


def scan(steps, heads, groups, d, dv, args, state, lens, slots, **more):
    from rllm_b200.kernels import ops
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    starts = i32([sum(lens[:i]) for i in range(len(lens) + 1)])
    args = [x.cuda() for x in args]
    if steps:
        out = ops.ssd_scan(*args, state, starts, i32(slots), len(lens), heads, groups, d, dv, err, max_q_len=max(lens), **more)
    else:
        q, k, v = torch.split(args[0], [heads * d, heads * d, heads * dv], 1)
        out = ops.lightning_scan(q, k, v, args[1], state, starts, i32(slots), len(lens), err, max_q_len=max(lens), **more)
    assert int(err.item()) == 0
    return out.view(-1, heads, dv)


# both sides of the line where the chunks of 128 are taken (their number; heads times their size), portions around a chunk,
# groups of one head, of some and of all, more pairs of chunk and head than an SM each, few and many CTAs a head
@pytest.mark.parametrize("steps,heads,groups,d,dv,lens", [
    (True, 4, 2, 128, 64, [129, 128, 1]), (True, 3, 3, 64, 64, [127, 257, 130]), (True, 6, 3, 64, 64, [127, 257, 130]), (True, 2, 1, 64, 128, [300, 2]),
    (True, 2, 1, 128, 128, [511]), (True, 12, 2, 128, 64, [900, 640, 5]), (True, 40, 4, 128, 64, [700]), (True, 2, 1, 128, 64, [900]),
    (False, 3, 0, 128, 128, [129, 128, 1]), (False, 2, 0, 64, 64, [127, 257, 130]), (False, 2, 0, 64, 128, [300, 2]),
    (False, 2, 0, 128, 64, [511]), (False, 6, 0, 128, 128, [900, 3]), (False, 2, 0, 128, 128, [900])])
def test_chunks_of_128_tokens(steps, heads, groups, d, dv, lens):
    """A factor that is split in two bfloat16 numbers keeps 16 bits: 2^-17 of each term, at random over a row's terms; the
    states' error adds as much again.  An earlier call's state is carried on, other slots stay as they are."""
    T, slots = sum(lens), [4, 0, 2][:len(lens)]
    args, ref = inputs(steps, heads, groups, d, dv, T, heads + d + dv + T)
    g = torch.Generator().manual_seed(T)
    first = torch.randn(6, heads, d, dv, generator=g)
    state = first.cuda()
    got = scan(steps, heads, groups, d, dv, args, state, lens, slots)
    at = 0
    for s, n in enumerate(lens):
        out, end = recurrence(*(x[at:at + n] for x in ref[:5]), ref[5], first[slots[s]].to(F64))
        assert ((got[at:at + n].cpu() - out).norm() / out.norm()) <= 2.0 ** -16
        assert ((state[slots[s]].cpu() - end).norm() / end.norm()) <= 2.0 ** -16
        at += n
    kept = [i for i in range(6) if i not in slots]
    assert torch.equal(state[kept].cpu(), first[kept])


@pytest.mark.parametrize("steps", [True, False])
def test_a_value_that_is_not_finite_reaches_later_tokens_of_its_column_only(steps):
    heads, d, dv, lens, bad = 4, 128, 64, [300, 140], 170
    args, _ = inputs(steps, heads, heads, d, dv, sum(lens), 3)
    col = (0 if steps else 2 * heads * d) + 1 * dv + 7                      # head 1, column 7
    state = torch.zeros(2, heads, d, dv, device="cuda")
    clean = scan(steps, heads, heads, d, dv, args, state.clone(), lens, [0, 1])
    args[0][bad, col] = math.inf
    got = scan(steps, heads, heads, d, dv, args, state, lens, [0, 1])
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[bad:lens[0], 1, 7] = True
    assert not torch.isfinite(got[hit]).any()
    assert torch.equal(got[~hit], clean[~hit])


@pytest.mark.parametrize("steps,heads,groups,d,dv,prompts", [(True, 4, 2, 64, 64, [129]), (True, 12, 1, 128, 64, [200, 900]), (True, 2, 1, 24, 40, [300]),
                                                             (False, 3, 0, 128, 128, [130, 2]), (False, 2, 0, 32, 64, [500]), (False, 2, 0, 48, 20, [140])])
def test_decoded_tokens_beside_prompts_have_the_bits_of_either_alone(steps, heads, groups, d, dv, prompts):
    """With as many decoded tokens as are walked apart, and a few more."""
    from rllm_b200.kernels import ops
    decode = -(-ops.SCAN_APART_FROM // (heads * dv)) + 2
    lens = [1] * decode + prompts
    args, _ = inputs(steps, heads, groups, d, dv, sum(lens), d + dv)
    g = torch.Generator().manual_seed(d)
    first = torch.randn(len(lens) + 2, heads, d, dv, generator=g).cuda()
    slots = torch.randperm(len(lens) + 2, generator=g)[: len(lens)].tolist()
    both, alone, behind = first.clone(), first.clone(), first.clone()
    got = scan(steps, heads, groups, d, dv, args, both, lens, slots, num_decode=decode)
    part = lambda lo, hi: [x[lo:hi] if len(x) == sum(lens) else x for x in args]  # noqa: E731
    want = torch.cat([scan(steps, heads, groups, d, dv, part(0, decode), alone, [1] * decode, slots[:decode]),
                      scan(steps, heads, groups, d, dv, part(decode, None), behind, prompts, slots[decode:])])
    assert torch.equal(got, want)
    assert torch.equal(both[slots], torch.cat([alone[slots[:decode]], behind[slots[decode:]]]))

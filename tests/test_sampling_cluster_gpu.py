"""Sampling by a cluster of CTAs a row against the one-CTA kernel, token for token: the sizes at which the cluster, its
threads and where a range is kept change (one, two and eight CTAs a row; up to 14 rows and more; ranges too long for
shared memory, ranges too long for words of 14 bits), rows that start anywhere, ties across the edges between ranges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,R", [(2048, 3), (2049, 14), (16385, 15), (128256, 1), (128257, 14), (128256, 33),
                                 (500003, 3), (2097152, 1), (2097153, 2), (5000001, 1), (64, 300), (3001, 130), (3001, 260),
                                 (20000, 50), (20000, 70), (50001, 65), (210000, 40), (210001, 64), (420001, 20)])
def test_clusters_draw_the_tokens_of_one_cta(V, R):
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(V + R)
    full = torch.randn(R, V + 3, generator=g, device="cuda") * 3
    full[0] = torch.round(full[0])                         # ties at every threshold, in every range
    full[R - 1, V // 8 - 2: V // 8 + 3] = 11.0             # the largest values lie across an edge between ranges
    for offset in (0, 1):
        logits = full[:, offset: offset + V]
        pick = lambda *v: [v[i % len(v)] for i in range(R)]  # noqa: E731
        temperature = torch.tensor(pick(0.8, 1.2, 0.0, 0.5), device="cuda")
        for k, p, m in ((-1, 0.9, 0.0), (50, 1.0, 0.0), (V - 1, 0.5, 0.02), (-1, 1.0, 0.1)):
            top_k = torch.full((R,), k, dtype=torch.int32, device="cuda")
            top_p = torch.full((R,), p, device="cuda")
            min_p = torch.full((R,), m, device="cuda")
            seeds = torch.arange(R, device="cuda") * 1001 + k
            gen = torch.arange(R, device="cuda") + 5
            one, many = (torch.full((R,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
            ops.sample_one_cta(logits, temperature, top_k, top_p, min_p, seeds, gen, one)
            ops.sample(logits, temperature, top_k, top_p, min_p, seeds, gen, many)
            assert one.tolist() == many.tolist()


@pytest.mark.parametrize("V,R", [(1500, 2), (5000, 9), (20000, 16), (128256, 2)])
@pytest.mark.parametrize("like", [1, 63, 65, 130, 511, 513, 1400])
def test_rows_of_like_values_draw_the_tokens_of_one_cta(V, R, like):
    """``like`` logits that share 22 bits with the threshold, all in one range or spread over all, equal or not: on both sides
    of what the ranges' lists hold, of which one alone may run over."""
    from rllm_b200.kernels import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(V + like)
    for spread in (False, True):
        for differ in (0, 1):
            bits = torch.full((like,), 0x40400000, dtype=torch.int32, device="cuda") + differ * torch.randint(0, 1000, (like,), generator=g, device="cuda")
            logits = torch.randn(R, V, generator=g, device="cuda") - 6
            at = torch.randperm(V, generator=g, device="cuda")[:like] if spread else (torch.arange(like, device="cuda") + V // 9) % V
            logits[:, at] = bits.to(torch.int32).view(torch.float32)
            for k, p in ((max(1, like // 2 + 1), 1.0), (-1, 0.6), (like + 3, 0.9)):
                args = (torch.ones(R, device="cuda"), torch.full((R,), k, dtype=torch.int32, device="cuda"), torch.full((R,), p, device="cuda"),
                        torch.zeros(R, device="cuda"), torch.arange(R, device="cuda") * 77, torch.arange(R, device="cuda") + 3)
                one, many = (torch.full((R,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
                ops.sample_one_cta(logits, *args, one)
                ops.sample(logits, *args, many)
                assert one.tolist() == many.tolist()

"""Sampling with top-k and top-p where top-k leaves a short list, as many tokens as the list holds, and more because of equal
logits: the tokens that the full passes choose, and only kept ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [300, 5000, 151936])
@pytest.mark.parametrize("k", [1, 50, 1024, 1025, 4000])
@pytest.mark.parametrize("ties", [False, True])
def test_list_after_top_k(V, k, ties):
    from tinyserve_b200.kernels import ops
    B = 24
    g = torch.Generator().manual_seed(V + k)
    x = torch.randn(B, V, generator=g) * 3
    if ties:
        x = (x * 2).round() / 2                  # some thousand equal logits at the border
    x = x.cuda()
    temp = torch.full((B,), 0.8).cuda()
    streams, steps = torch.arange(B).cuda(), torch.arange(B, dtype=torch.int32).cuda()
    top_k, top_p = torch.full((B,), k, dtype=torch.int32).cuda(), torch.full((B,), 0.9).cuda()
    inverse = (1.0 / torch.tensor(0.8)).cuda()
    both = ops.sample(x, temp, streams, steps, 7, top_k=top_k, top_p=top_p).cpu()
    only_k = ops.sample(x, temp, streams, steps, 7, top_k=top_k).cpu()
    for b in range(B):
        y = (x[b] * inverse).double().cpu()
        kept = y >= (y.sort(descending=True).values[min(k, V) - 1] if k < V else -float("inf"))
        assert kept[only_k[b]] and kept[both[b]]
        p = torch.where(kept, (y - y.max()).exp(), torch.zeros(()).double())
        order = y.sort(descending=True, stable=True)
        mass = p[order.indices].cumsum(0) / p.sum()
        # top-p keeps what is at least as large as the token at which 0.9 of the mass is passed (weights carry 2^-32 each)
        edge = order.values[int((mass > 0.9 + 1e-4).float().argmax())]
        assert y[both[b]] >= edge
    # rows with everything but the kept tokens taken out, sampled without top-k, give the same tokens
    masked = x.clone()
    for b in range(B):
        y = x[b] * inverse
        if k < V:
            masked[b][y < y.sort(descending=True).values[k - 1]] = -float("inf")
    assert torch.equal(ops.sample(masked, temp, streams, steps, 7).cpu(), only_k)
    assert torch.equal(ops.sample(masked, temp, streams, steps, 7, top_p=top_p).cpu(), both)


@pytest.mark.parametrize("k", [8191, 8192, 8193, 20000])
def test_list_of_eight_blocks(k):
    """Up to eight times the length of a block's list top-k may leave lists, above there are none."""
    from tinyserve_b200.kernels import ops
    B, V = 2, 151936
    g = torch.Generator().manual_seed(k)
    x = (torch.randn(B, V, generator=g) * 3).cuda()
    temp, streams, steps = torch.full((B,), 0.8).cuda(), torch.arange(B).cuda(), torch.arange(B, dtype=torch.int32).cuda()
    top_k, top_p = torch.full((B,), k, dtype=torch.int32).cuda(), torch.full((B,), 0.9).cuda()
    inverse = (1.0 / torch.tensor(0.8)).cuda()
    masked = x.clone()
    for b in range(B):
        y = x[b] * inverse
        masked[b][y < y.sort(descending=True).values[k - 1]] = -float("inf")
    assert torch.equal(ops.sample(masked, temp, streams, steps, 7), ops.sample(x, temp, streams, steps, 7, top_k=top_k))
    assert torch.equal(ops.sample(masked, temp, streams, steps, 7, top_p=top_p),
                       ops.sample(x, temp, streams, steps, 7, top_k=top_k, top_p=top_p))

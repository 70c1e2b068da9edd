"""Decode attention over a few keys, where one block walks them all without its cluster, against the 64-bit softmax:
lengths around the border, alone and beside longer requests, plain and with a window, sinks and slopes."""
import pytest
import torch
from types import SimpleNamespace as NS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,page", [(128, 64), (128, 16), (64, 32), (32, 8)])
@pytest.mark.parametrize("lengths", [[1], [63, 64, 65], [128, 129, 127, 130], [2, 700, 128, 192, 193]])
@pytest.mark.parametrize("window,keep_first,sinks,slopes", [(0, 0, False, False), (100, 0, True, False), (70, 5, False, True)])
def test_decode_attention_of_short_walks(head_dim, page, lengths, window, keep_first, sinks, slopes):
    from tinyserve_b200.kernels import ops
    H, Hkv, D, B = 8, 2, head_dim, len(lengths)
    g = torch.Generator().manual_seed(sum(lengths) + D)
    pages = -(-max(lengths) // page)
    k, v = (torch.randn(B * pages + 1, Hkv, page, D, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(B, H, D, generator=g).bfloat16().cuda()
    table = (torch.randperm(B * pages, generator=g) + 1).int().view(B, pages).cuda()
    ctx = NS(cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_lens=torch.tensor(lengths, dtype=torch.int32).cuda(),
             num_requests=B, max_q_len=1, max_kv_len=1024)
    s = torch.randn(H, generator=g).cuda() if sinks else None
    m = torch.rand(H, generator=g).cuda() * 0.1 if slopes else None
    out = ops.paged_attention(q, k, v, NS(block_table=table, page_size=page), ctx, D ** -0.5, window, keep_first=keep_first, sinks=s, slopes=m)
    for b, n in enumerate(lengths):
        rows = [x[table[b].long()].transpose(0, 1).reshape(Hkv, -1, D)[:, :n].double().repeat_interleave(H // Hkv, 0) for x in (k, v)]
        score = torch.einsum("hd,hnd->hn", q[b].double(), rows[0]) * D ** -0.5
        j = torch.arange(n, device="cuda")
        if slopes:
            score -= m.double()[:, None] * (n - 1 - j)
        if window:
            score[:, ~((j > n - 1 - window) | (j < keep_first))] = -float("inf")
        if sinks:
            score = torch.cat([score, s.double()[:, None]], 1)
        p = score.softmax(1)[:, :n]
        want = torch.einsum("hn,hnd->hd", p, rows[1])
        # the probabilities and the result are rounded to bfloat16
        assert (out[b].double() - want).abs().max() <= 2.0 ** -8 * (want.abs().max() + rows[1].abs().max())
    assert ops.attention_mma_error(D) == 0


@pytest.mark.parametrize("D", [80, 96, 256])
@pytest.mark.parametrize("B", [12, 16])
def test_short_walks_of_wide_heads_in_small_clusters(D, B):
    """Clusters of three (12 requests) and of two (16): either side of the number of tiles that a block walks alone."""
    from tinyserve_b200.kernels import ops
    H, page = 8, 16
    lengths = ([1, 63, 64, 65, 127, 128, 129, 192] * 2)[:B]
    assert ops.decode_splits(B, 1024, H, H) == (3 if B == 12 else 2)
    g = torch.Generator().manual_seed(D + B)
    k, v = (torch.randn(B * 12 + 1, H, page, D, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(B, H, D, generator=g).bfloat16().cuda()
    table = (torch.randperm(B * 12, generator=g) + 1).int().view(B, 12).cuda()
    ctx = NS(cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_lens=torch.tensor(lengths, dtype=torch.int32).cuda(),
             num_requests=B, max_q_len=1, max_kv_len=1024)
    out, want = (ops.paged_attention(q, k, v, NS(block_table=table, page_size=page), ctx, D ** -0.5, num_splits=n).float() for n in (None, 1))
    # a probability is rounded to bfloat16 (2^-9) against its range's maximum on either side, and so is the result
    assert (out - want).abs().max() <= 2.0 ** -8 * (want.abs().max() + v.float().abs().max())
    assert ops.attention_mma_error(D) == 0


@pytest.mark.parametrize("lengths", [[1], [64, 128, 129, 40], [127, 500]])
def test_decode_attention_from_the_projection_of_short_walks(lengths):
    """The kernel that makes the newest key and value itself against the two kernels."""
    from tinyserve_b200.kernels import ops
    H, Hkv, D, B, page = 16, 8, 128, len(lengths), 64
    g = torch.Generator().manual_seed(sum(lengths))
    pages = -(-max(lengths) // page)
    caches = [torch.randn(B * pages + 1, Hkv, page, D, generator=g).bfloat16().cuda() for _ in range(2)]
    qkv = torch.randn(B, (H + 2 * Hkv) * D, generator=g).bfloat16().cuda()
    angles = torch.rand(1024, D // 2, generator=g).cuda() * 6
    rotary = NS(cos=angles.cos(), sin=angles.sin(), rotary_dim=D, interleaved=False)
    w = (1 + 0.1 * torch.randn(D, generator=g)).bfloat16().cuda()
    table = (torch.randperm(B * pages, generator=g) + 1).int().view(B, pages).cuda()
    kv = torch.tensor(lengths, dtype=torch.int32).cuda()
    slots = torch.tensor([int(table[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(lengths)], dtype=torch.int32).cuda()
    ctx = NS(cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_lens=kv, num_requests=B, max_q_len=1, max_kv_len=1024)
    view, results = NS(block_table=table, page_size=page, slot_mapping=slots), []
    for fused in (True, False):
        k, v = (c.clone() for c in caches)
        results.append((ops.attention_from_qkv(qkv, kv - 1, H, Hkv, D, rotary, w, w, 1e-6, k, v, view, ctx, D ** -0.5, fused=fused), k, v))
    assert torch.equal(results[0][1], results[1][1]) and torch.equal(results[0][2], results[1][2])
    torch.testing.assert_close(results[0][0].float(), results[1][0].float(), rtol=2.0 ** -7, atol=2.0 ** -9)

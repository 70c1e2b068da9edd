"""Decode attention over pages that come whole (16 to 64 keys) and by pieces (8), with NaN in every slot that no request
uses: head sizes and head groups on either side of the kernels' forms, few keys and many, in clusters and by scratch."""
import pytest
import torch
from types import SimpleNamespace as NS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page", [8, 16, 32, 64])
@pytest.mark.parametrize("H,Hkv,D", [(8, 2, 128), (2, 2, 64), (24, 2, 128), (9, 1, 64), (16, 2, 256), (12, 4, 96), (40, 2, 128)])
@pytest.mark.parametrize("lengths", [[1, 15, 16, 17], [64, 65, 130, 200, 333], [700, 3], [1500]])
def test_pages(page, H, Hkv, D, lengths):
    from tinyserve_b200.kernels import ops
    B = len(lengths)
    g = torch.Generator().manual_seed(sum(lengths) + D + H)
    pages = -(-max(lengths) // page)
    data = [torch.randn(B, pages * page, Hkv, D, generator=g).bfloat16().cuda() for _ in range(2)]
    table = (torch.randperm(B * pages, generator=g) + 1).int().view(B, pages).cuda()
    caches = []
    for x in data:
        cache = torch.full((B * pages + 1, page, Hkv, D), float("nan"), dtype=torch.bfloat16, device="cuda")
        cache[0] = 0
        for b, n in enumerate(lengths):
            rows = x[b].clone()
            rows[n:] = float("nan")
            cache[table[b].long()] = rows.view(pages, page, Hkv, D)
        caches.append(cache.transpose(1, 2).contiguous())
    kv = torch.tensor(lengths, dtype=torch.int32).cuda()
    ctx = NS(cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_lens=kv, num_requests=B, max_q_len=1, max_kv_len=max(1024, max(lengths)))
    slots = torch.tensor([int(table[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(lengths)], dtype=torch.int32).cuda()
    view = NS(block_table=table, page_size=page, slot_mapping=slots)
    q = torch.randn(B, H, D, generator=g).bfloat16().cuda()
    want, size = [], 0.0
    for b, n in enumerate(lengths):
        k, v = (x[b, :n].transpose(0, 1).double().repeat_interleave(H // Hkv, 0) for x in data)
        want.append(torch.einsum("hn,hnd->hd", (torch.einsum("hd,hnd->hn", q[b].double(), k) * D ** -0.5).softmax(1), v))
        size = max(size, float(want[-1].abs().max() + v.abs().max()))
    want = torch.stack(want)
    # the probabilities and the result are rounded to bfloat16
    for splits in (None, 1, 12):
        out = ops.paged_attention(q, *caches, view, ctx, D ** -0.5, num_splits=splits)
        assert (out.double() - want).abs().max() <= 2.0 ** -8 * size, splits
    # from a projection whose rows are the same: no norm, no turn
    qkv = torch.cat([q] + [torch.stack([x[b, n - 1] for b, n in enumerate(lengths)]) for x in data], 1).view(B, -1)
    rot = NS(cos=torch.ones(2048, D // 2, device="cuda"), sin=torch.zeros(2048, D // 2, device="cuda"), rotary_dim=D, interleaved=False)
    for c in caches:
        for s in slots.tolist():
            c[s // page, :, s % page] = float("nan")
    out = ops.attention_from_qkv(qkv, kv - 1, H, Hkv, D, rot, None, None, 0.0, *caches, view, ctx, D ** -0.5)
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * size
    for cache, x in zip(caches, data):
        for b, n in enumerate(lengths):
            s = int(slots[b])
            assert torch.equal(cache[s // page, :, s % page], x[b, n - 1])
    assert ops.attention_mma_error(D) == 0


@pytest.mark.parametrize("page", [8, 16, 32, 64])
@pytest.mark.parametrize("H,Hkv,D", [(8, 2, 128), (9, 1, 64), (4, 2, 256), (40, 2, 128), (12, 4, 96)])
@pytest.mark.parametrize("window,keep_first", [(1, 0), (40, 0), (100, 5), (200, 70)])
def test_what_lies_before_a_window(page, H, Hkv, D, window, keep_first):
    """NaN in every key and value before the window that is not kept, in pages of their own and in pages that the window
    begins in, with walks long enough that a stage takes a second tile."""
    from tinyserve_b200.kernels import ops
    lengths = [1, 63, 130, 333, 700]
    B = len(lengths)
    g = torch.Generator().manual_seed(window + D + H)
    pages = -(-max(lengths) // page)
    data = [torch.randn(B, pages * page, Hkv, D, generator=g).bfloat16().cuda() for _ in range(2)]
    table = (torch.randperm(B * pages, generator=g) + 1).int().view(B, pages).cuda()
    caches = []
    for x in data:
        cache = torch.full((B * pages + 1, page, Hkv, D), float("nan"), dtype=torch.bfloat16, device="cuda")
        for b, n in enumerate(lengths):
            rows = x[b].clone()
            rows[n:] = float("nan")
            rows[keep_first:max(keep_first, n - window)] = float("nan")
            cache[table[b].long()] = rows.view(pages, page, Hkv, D)
        caches.append(cache.transpose(1, 2).contiguous())
    kv = torch.tensor(lengths, dtype=torch.int32).cuda()
    ctx = NS(cu_q=torch.arange(B + 1, dtype=torch.int32).cuda(), kv_lens=kv, num_requests=B, max_q_len=1, max_kv_len=max(lengths))
    slots = torch.tensor([int(table[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(lengths)], dtype=torch.int32).cuda()
    view = NS(block_table=table, page_size=page, slot_mapping=slots)
    q = torch.randn(B, H, D, generator=g).bfloat16().cuda()

    def wanted(kept):
        rows, size = [], 0.0
        for b, n in enumerate(lengths):
            seen = [j for j in range(n) if j >= n - window or j < kept]
            k, v = (x[b, seen].transpose(0, 1).double().repeat_interleave(H // Hkv, 0) for x in data)
            rows.append(torch.einsum("hn,hnd->hd", (torch.einsum("hd,hnd->hn", q[b].double(), k) * D ** -0.5).softmax(1), v))
            size = max(size, float(rows[-1].abs().max() + v.abs().max()))
        return torch.stack(rows), size

    # (the bound of test_pages)
    want, size = wanted(keep_first)
    for splits in (None, 1, 2, 12):
        out = ops.paged_attention(q, *caches, view, ctx, D ** -0.5, window=window, keep_first=keep_first, num_splits=splits)
        assert (out.double() - want).abs().max() <= 2.0 ** -8 * size, splits
    if keep_first == 0:
        qkv = torch.cat([q] + [torch.stack([x[b, n - 1] for b, n in enumerate(lengths)]) for x in data], 1).view(B, -1)
        rot = NS(cos=torch.ones(2048, D // 2, device="cuda"), sin=torch.zeros(2048, D // 2, device="cuda"), rotary_dim=D, interleaved=False)
        for most in (max(lengths), 200):           # (key ranges that a few tiles are cut into, and few)
            ctx.max_kv_len = most
            out = ops.attention_from_qkv(qkv, kv - 1, H, Hkv, D, rot, None, None, 0.0, *caches, view, ctx, D ** -0.5, window=window)
            assert (out.double() - want).abs().max() <= 2.0 ** -8 * size, most
    assert ops.attention_mma_error(D) == 0

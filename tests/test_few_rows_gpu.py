"""The 32-bit products (chains of k dealt to threads) against the sums that define it, bit by bit, and
the sampler's rows over clusters of blocks against one row at a time and against a plain restatement."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def chain_sums(x, w, bias=None):
    """fmaf over 64 consecutive k in order, the chains' results added in order, in 32-bit.  (A product of
    two floats is exact in 64 bits, and the 64-bit sum of it with a float, rounded to 32 bits, is fmaf up to a
    double rounding, which the operands below cannot show: they have 8 significant bits.)"""
    x, w = x.double().cpu().numpy(), w.double().cpu().numpy()
    total = np.zeros((x.shape[0], w.shape[0]), np.float32)
    for k0 in range(0, x.shape[1], 64):
        part = np.zeros_like(total)
        for k in range(k0, min(k0 + 64, x.shape[1])):
            part = (part.astype(np.float64) + x[:, k:k + 1] * w[None, :, k]).astype(np.float32)
        total = total + part
    return total if bias is None else total + bias.cpu().numpy()


# K: less than a chain, whole chains, a ragged last chain, fewer and more chains than a block has in
# flight at a time (16); N: edges of a block's rows; M: every width of the kernel and its edges
@pytest.mark.parametrize("K", [4, 60, 64, 96, 160, 1024, 1100, 2052])
@pytest.mark.parametrize("M,N", [(1, 1), (1, 8192), (2, 33), (3, 4100), (4, 17), (5, 2048), (8, 2056), (9, 100), (17, 1030), (64, 96), (256, 40), (640, 1100)])
def test_product_of_few_rows_is_the_chain_sum(M, N, K):
    from tinyserve_b200.kernels import ops
    if M * N * K > 2 ** 24 and (M < 640 or K > 96):
        pytest.skip("the restatement would take long; the shape's edges are covered by smaller ones")
    g = torch.Generator().manual_seed(M * 7 + N * 3 + K)
    x, w = (torch.randn(r, K, generator=g).bfloat16().float().cuda() for r in (M, N))
    bias = torch.randn(N, generator=g).cuda()
    out = ops.linear(x, w, bias)
    np.testing.assert_array_equal(out.cpu().numpy(), chain_sums(x, w, bias))


@pytest.mark.parametrize("M,N,K", [(640, 1100, 1100), (641, 1087, 2052), (65, 12224, 260), (1030, 600, 300)])
def test_rows_of_large_products_are_those_of_few_rows(M, N, K):
    """Tiles of many rows (whole and ragged, whole rounds of four chains and not) against the kernel for few."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M)
    x, w, bias = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda(), torch.randn(N, generator=g).cuda()
    assert torch.equal(ops.linear(x, w, bias), torch.cat([ops.linear(rows.contiguous(), w, bias) for rows in x.split(8)]))


@pytest.mark.parametrize("M", [2, 5, 24, 300])
def test_product_of_few_rows_takes_leading_dimensions(M):
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, 144, generator=g).cuda(), torch.randn(96, 144, generator=g).cuda()
    for k, at in ((128, 0), (128, 4), (126, 0), (128, 1)):          # aligned, aligned inside a row, a ragged K, unaligned
        xs, ws = x[:, at:at + k], w[:, at:at + k]
        want = ops.linear(xs.contiguous()[:1], ws.contiguous())
        got = ops.linear(xs, ws)
        assert torch.equal(got[:1], want)
        torch.testing.assert_close(got.double(), xs.double() @ ws.double().T, rtol=0, atol=2e-5)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices")
def test_products_on_two_devices_of_one_process():
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(1)
    for M, N in ((1, 4096), (8, 4096), (600, 1024)):
        x, w, results = torch.randn(M, 1024, generator=g), torch.randn(N, 1024, generator=g), []
        for device in range(2):
            with torch.cuda.device(device):
                results.append(ops.linear(x.cuda(), w.cuda()).cpu())
        assert torch.equal(*results)


# a short K, where the rule goes over to the tiled kernel (first and last of each line: either side of it)
@pytest.mark.parametrize("M,N,K", [(8, 32000, 16), (40, 32000, 16), (64, 32000, 200), (65, 4096, 16), (512, 9000, 4), (4096, 64, 64), (4096, 64, 320),
                                   (20000, 33, 16), (20000, 256, 96), (20000, 256, 200), (100000, 8, 32), (100000, 8, 260)])
def test_rows_of_products_of_a_short_k(M, N, K):
    from tinyserve_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w, bias = (torch.randn(*s, generator=g, device="cuda") for s in ((M, K), (N, K), (N,)))
    out = ops.linear(x, w, bias)
    for rows in (torch.arange(8), torch.arange(M - 8, M), torch.randint(M, (8,)), torch.randint(M, (3,))):
        rows = rows.cuda()
        assert torch.equal(out[rows], ops.linear(x[rows].contiguous(), w, bias))
        torch.testing.assert_close(out[rows].double(), x[rows].double() @ w.double().T + bias.double(), rtol=0, atol=2e-4)


@pytest.mark.parametrize("M", [65535 * 8, 65535 * 8 + 1, 65535 * 64 + 1, 65535 * 128])
def test_products_of_very_many_rows(M):
    """A grid has 65,535 blocks of rows at most, which every kernel reaches at another number of rows."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(3)
    w = torch.randn(3, 8, generator=g).cuda()
    x = torch.randn(1024, 8, generator=g).cuda().repeat(-(-M // 1024), 1)[:M]
    out, want = ops.linear(x, w), ops.linear(x[:1024], w)
    assert torch.equal(out, want.repeat(-(-M // 1024), 1)[:M])


def test_more_rows_than_any_grid_covers_are_refused():
    from tinyserve_b200.kernels import ops
    with pytest.raises(RuntimeError, match="too large"):
        ops.linear(torch.zeros(65535 * 128 + 1, 4, device="cuda"), torch.zeros(3, 4, device="cuda"))


# both kernels that fetch W early (few rows; many rows, one wave of tiles and more), the weight made by the product just
# before or by the one before that
@pytest.mark.parametrize("between", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 2048, 1024), (8, 4096, 512), (200, 512, 1024), (1024, 1536, 1024)])
def test_a_weight_may_be_the_product_before(M, N, K, between):
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M)
    x, a, b = (torch.randn(r, c, generator=g).cuda() for r, c in ((M, K), (N, 2048), (K, 2048)))
    for _ in range(3):
        stale = torch.full((N, K), float("nan"), device="cuda")            # what an early read of the weight finds
        torch.cuda.synchronize()
        del stale
        w = ops.linear(a, b)
        for _ in range(between):
            ops.linear(x[:1], a[:, :K])
        out = [ops.linear(x, w), ops.gated_linear(x, w), ops.activated_linear(x, w, "relu_squared")]
        torch.cuda.synchronize()
        want = [ops.linear(x, w, constant_weight=True), ops.gated_linear(x, w, constant_weight=True),
                ops.activated_linear(x, w, "relu_squared", constant_weight=True)]
        for got, expected in zip(out, want):
            assert torch.equal(got, expected)
    torch.testing.assert_close(w.double(), a.double() @ b.double().T, rtol=0, atol=2e-3)


def plain_sample(x, temp, k, p):
    """The tokens that may be drawn: top-k with ties, then top-p over exact integer weights."""
    y = (x * np.float32(1.0 / np.float32(temp))).astype(np.float32)
    keep = np.ones(len(y), bool)
    if 0 < k < len(y):
        keep &= y >= np.sort(y)[-k]
    if p < 1:
        mx = y[keep].max()
        weight = np.exp((y - mx).astype(np.float64)) * keep
        order = np.argsort(-y, kind="stable")
        before = np.cumsum(weight[order]) - weight[order]
        keep_p = np.zeros_like(keep)
        keep_p[order[before <= p * weight.sum()]] = True
        keep &= keep_p
    return keep


@pytest.mark.parametrize("V", [1, 5, 257, 8191, 8192, 16384, 40000, 151936])
@pytest.mark.parametrize("B", [1, 3, 40, 80, 150])
def test_sampled_rows_do_not_depend_on_the_blocks_that_share_them(V, B):
    """The number of blocks per row follows from the number of rows: a row alone, and the same row among
    others, must give the same token, greedy or with any filter."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(V + B)
    x = (torch.randn(B, V, generator=g) * 3).cuda()
    x[:, V // 2] = x.max(dim=1).values                                # a tie for the largest
    temp = torch.tensor([(0.0, 0.7, 1.3, 0.9)[i % 4] for i in range(B)]).cuda()
    ks = torch.tensor([(0, 50, 0, 7)[i % 4] for i in range(B)], dtype=torch.int32).cuda()
    ps = torch.tensor([(1.0, 0.9, 0.5, 1.0)[i % 4] for i in range(B)]).cuda()
    streams, steps = torch.arange(B).cuda(), torch.arange(B, dtype=torch.int32).cuda()
    together = ops.sample(x, temp, streams, steps, 11, top_k=ks, top_p=ps).cpu()
    for i in sorted({0, 1 % B, 2 % B, 3 % B, B - 1}):
        one = slice(i, i + 1)
        alone = ops.sample(x[one], temp[one], streams[one], steps[one], 11, top_k=ks[one], top_p=ps[one]).cpu()
        assert alone[0] == together[i]
        row = x[i].cpu().numpy()
        if temp[i] == 0:
            assert together[i] == int(np.flatnonzero(row == row.max())[0])
        else:
            assert plain_sample(row, float(temp[i]), int(ks[i]), float(ps[i]))[int(together[i])]


# the longest row that one block reads for its maximum, and one more; the fewest tokens that get a cluster; odd rows;
# numbers of rows around those whose clusters of eight, four and two have a place at once
@pytest.mark.parametrize("V", [8188, 8192, 32768, 32769, 50257])
@pytest.mark.parametrize("B", [1, 14, 15, 16, 17, 18, 19, 33, 37, 38, 74, 75, 148, 149])
def test_maximum_of_rows_by_any_number_of_blocks(V, B):
    from tinyserve_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(V + B)
    x = torch.randn(B, V, generator=g, device="cuda")
    at = torch.randint(V, (B,), generator=g, device="cuda")
    x[torch.arange(B), at] = 9.0
    x[:, V - 1] = 9.0                                                    # a tie: the lower index wins
    zero, one = torch.zeros(B, device="cuda"), torch.full((B,), 1e-3, device="cuda")
    streams, steps = torch.arange(B, device="cuda"), torch.zeros(B, dtype=torch.int32, device="cuda")
    assert torch.equal(ops.sample(x, zero, streams, steps, 5), at.int())
    x[:, V - 1] = 0.0
    x[torch.arange(B), at] = 9.0
    # at so low a temperature the noise cannot lift another token over the largest
    assert torch.equal(ops.sample(x, one, streams, steps, 5), at.int())
    mixed = torch.where(streams % 2 == 0, zero, one)
    keep = torch.full((B,), 3, dtype=torch.int32, device="cuda")
    assert torch.equal(ops.sample(x, mixed, streams, steps, 5, top_k=keep, top_p=torch.full((B,), 0.5, device="cuda")), at.int())


def test_rows_of_infinities_and_nans():
    from tinyserve_b200.kernels import ops
    x = torch.full((4, 20000), -float("inf")).cuda()
    x[1, 12345] = float("inf")
    x[2, 7] = 1.0
    x[3] = 0.5
    x[3, ::2] = float("nan")
    zero, streams, steps = torch.zeros(4).cuda(), torch.arange(4).cuda(), torch.zeros(4, dtype=torch.int32).cuda()
    assert ops.sample(x, zero, streams, steps, 1).tolist() == [0, 12345, 7, 1]
    one = torch.ones(4).cuda()
    assert ops.sample(x, one, streams, steps, 1).tolist()[1:3] == [12345, 7]

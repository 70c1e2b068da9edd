"""The 32-bit sums of the bfloat16 product for few tokens: how close they are to 64 bits, and the order of their parts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1024, 4096])
@pytest.mark.parametrize("M", [1, 16, 33, 64])
def test_sums_of_one_sign(M, K):
    """Of operands of one sign nothing cancels, and every step of an accumulator may cut off one unit in the
    last place of a running sum that is on average half of the final one.  A K step of 64 is one step of each
    of the four accumulators: K / 64 steps of 2^-23, halved."""
    from tinyserve_b200.kernels import ops
    N = 148 * 128                 # as many row tiles as multiprocessors: not cut along K, which would shorten the sums
    assert ops.gemm_splits(M, N, K) == 1
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.rand(M, K, generator=g, device="cuda").bfloat16()
    w = torch.rand(N, K, generator=g, device="cuda").bfloat16()
    out, want = ops.linear(x, w, out_float32=True).double(), x.double() @ w.double().T
    assert ((out - want).norm() / want.norm()).item() <= K / 64 * 2.0 ** -24
    assert ops.gemm_tcgen05_error() == 0


@pytest.mark.parametrize("splits", [2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 100])
def test_parts_add_up_in_order(M, splits):
    """The block that arrives last adds the parts in the order of K, several at a time: the same bits as one by one."""
    from tinyserve_b200.kernels import ops
    N, K = 640, 16 * 64
    g = torch.Generator(device="cuda").manual_seed(M + splits)
    x, w = (torch.randn(r, K, generator=g, device="cuda").bfloat16() for r in (M, N))
    parts = ops._linear_tcgen05(x, w, False, splits=splits, partials_only=True)
    tile = ops._tile_t(M)
    buffer = parts.data.view(splits, N // 128, tile, 128)
    want = torch.zeros(M, N, device="cuda")
    for s in range(splits):
        want += buffer[s].permute(1, 0, 2).reshape(tile, N)[:M]
    assert torch.equal(ops._linear_tcgen05(x, w, True, splits=splits), want)
    assert ops.gemm_tcgen05_error() == 0

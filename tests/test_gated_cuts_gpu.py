"""The gated product of a few tokens whose K is cut inside clusters, against the product and the activation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# N (gate and up rows): one row tile, several, 48 (the gate/up product of a small model), 147 (the most that are cut), 160 (one cut);
# K: one slice and a ragged one (no cut), cuts of unequal length, eight cuts
@pytest.mark.parametrize("N,K", [(128, 64), (128, 2048), (256, 1096), (640, 520), (6144, 1024), (147 * 128, 512), (160 * 128, 256)])
@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64])
@pytest.mark.parametrize("activation,limit", [("silu", 0.0), ("gelu_tanh", 0.0), ("bounded_swish", 0.5)])
def test_gated_product_of_few_row_tiles(M, N, K, activation, limit):
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).bfloat16().cuda()
    w = (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    blocks = w.double().view(N // 128, 2, 64, K)
    gate, up = ((x.double() @ blocks[:, i].reshape(N // 2, K).T) for i in (0, 1))
    if activation == "silu":
        want = torch.nn.functional.silu(gate) * up
    elif activation == "gelu_tanh":
        want = torch.nn.functional.gelu(gate, approximate="tanh") * up
    else:
        gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
        want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    launches = ops.launch_count()
    got = ops.gated_linear(x, w, activation, ops.GATED_BLOCK, limit)
    assert ops.launch_count() - launches == 1, "one kernel"
    assert got.dtype == torch.bfloat16 and got.shape == want.shape
    # one rounding to bfloat16 (2^-9 of the value) and 32-bit sums of K terms of about 1 / sqrt(K)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 4e-6).all()
    assert torch.equal(got, ops.gated_linear(x, w, activation, ops.GATED_BLOCK, limit)), "the same bits every time"
    assert ops.gemm_tcgen05_error() == 0


@pytest.mark.parametrize("M,kernels", [(32, 1), (33, 2), (64, 2)])
def test_more_row_tiles_than_run_at_once(M, kernels):
    """51,200 rows are 400 row tiles, more than two a multiprocessor: above 32 tokens the activation is a kernel of its own."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, 128, generator=g, device="cuda").bfloat16(), (torch.randn(51200, 128, generator=g, device="cuda") / 11).bfloat16()
    blocks = w.double().view(400, 2, 64, 128)
    gate, up = ((x.double() @ blocks[:, i].reshape(25600, 128).T) for i in (0, 1))
    want = torch.nn.functional.silu(gate) * up
    launches = ops.launch_count()
    got = ops.gated_linear(x, w, "silu", ops.GATED_BLOCK).double()
    assert ops.launch_count() - launches == kernels
    # of two kernels gate and up are rounded to bfloat16 as well: 2^-9 each, silu's slope is at most 1.1 and its argument's
    # rounding 2^-9 of it
    bound = 2.0 ** -8 * want.abs() + 4e-6 + (kernels - 1) * 2.0 ** -8 * (want.abs() + 1.1 * gate.abs() * up.abs())
    assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M", [1, 16, 31, 64])
def test_any_number_of_cuts(M, splits):
    """Cuts of unequal length, and one without a slice (5 cuts of 16 slices)."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, 1024, generator=g).bfloat16().cuda(), (torch.randn(640, 1024, generator=g) / 32).bfloat16().cuda()
    blocks = w.double().view(5, 2, 64, 1024)
    gate, up = ((x.double() @ blocks[:, i].reshape(320, 1024).T) for i in (0, 1))
    want = torch.nn.functional.silu(gate) * up
    got = ops._linear_tcgen05(x, w, False, splits=splits, gated=ops.ACTIVATIONS["silu"] + 1)
    assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 4e-6).all()
    assert ops.gemm_tcgen05_error() == 0


@pytest.mark.parametrize("M", [1, 5, 16, 17, 40, 64])
def test_rows_without_their_norm_factor(M):
    """Up to 16 rows from the product for few tokens; more (which only the paired product makes) are normalised first."""
    from tinyserve_b200.kernels import ops
    g = torch.Generator().manual_seed(M)
    x, o = torch.randn(M, 1024, generator=g).bfloat16().cuda(), (torch.randn(1024, 1024, generator=g) * 0.03).bfloat16().cuda()
    w = (torch.randn(768, 1024, generator=g) * 0.03).bfloat16().cuda()
    norm = (1 + 0.1 * torch.randn(1024, generator=g)).bfloat16().cuda()
    residual = torch.randn(M, 1024, generator=g).cuda()
    rows = ops.add_rmsnorm(ops.PendingProduct(x, o, wide=M > 16), residual, norm, 1e-6, torch.bfloat16, scaled_ok=True)
    assert isinstance(rows, ops.ScaledRows)
    got = ops.gated_linear(rows, w, "silu", ops.GATED_BLOCK).double()
    h = rows.data.double() * torch.rsqrt(residual.double().square().mean(1, keepdim=True) + 1e-6)
    blocks = w.double().view(6, 2, 64, 1024)
    gate, up = ((h @ blocks[:, i].reshape(384, 1024).T) for i in (0, 1))
    want = torch.nn.functional.silu(gate) * up
    if M > 16:
        # five roundings to bfloat16 of 2^-9 at most each: the normalised rows' (in gate and in up), gate's, up's, the result's
        assert (got - want).norm() <= 5 * 2.0 ** -9 * want.norm()
    else:
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()

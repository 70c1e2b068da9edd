"""The product that keeps its weights in registers (up to 8 tokens, weights of up to 16 MB) against 64 bits: ragged rows and K,
one token to eight, every form, and the ends of its range."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -8          # unit of a result rounded to bfloat16 (half an ulp is 2^-9 of the value)


def operands(M, N, K, seed=0):
    g = torch.Generator().manual_seed(seed + M * 131 + N * 7 + K)
    x = torch.randn(M, K + 8, generator=g).bfloat16().cuda()[:, :K]           # (a leading dimension of its own)
    return x, (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16().cuda()


@pytest.mark.parametrize("M", [1, 2, 7, 8])
@pytest.mark.parametrize("N,K", [(1, 8), (16, 64), (130, 248), (384, 256), (1000, 1024), (4096, 1032), (1024, 3072), (2048, 4096), (8191, 1024)])
def test_plain_and_partial_forms(M, N, K):
    from tinyserve_b200.kernels import ops
    assert ops._gemv_fits(M, N, K)
    x, w = operands(M, N, K)
    want = x.double() @ w.double().T
    # the products are exact in 32 bits; up to K / 64 steps of an MMA in each of four accumulators, each cut off at 2^-22 of it
    bound = 2.0 ** -22 * (K / 16 + 8) * (x.double().abs() @ w.double().abs().T) + 1e-12
    out = ops.linear(x, w, out_float32=True).double()
    assert ((out - want).abs() <= bound).all()
    part = ops.linear(x, w, allow_partials=True)
    assert isinstance(part, ops.SplitPartials) and part.splits == 1
    assert ((part.materialize().double() - want).abs() <= bound + U * want.abs()).all()
    assert ((ops.linear(x, w).double() - want).abs() <= bound + U * want.abs()).all()


@pytest.mark.parametrize("M", [1, 3, 8])
@pytest.mark.parametrize("N,K,F", [(128, 256, 128), (1024, 2048, 384), (1024, 3072, 3072), (96, 512, 192), (1008, 1000, 64)])
def test_residual_then_scaled_and_gated(M, N, K, F):
    """residual += x w^T, then the norm's product and the gated product of the new residual."""
    from tinyserve_b200.kernels import ops
    x, w = operands(M, N, K, 1)
    g = torch.Generator().manual_seed(5)
    res = torch.randn(M, N, generator=g).cuda()
    norm = (1 + 0.1 * torch.randn(N, generator=g)).bfloat16().cuda()
    want = res.double() + x.double() @ w.double().T
    pending = ops.linear(x, w, allow_pending=True)
    scaled = ops.add_rmsnorm(pending, res, norm, 1e-6, torch.bfloat16, scaled_ok=True)
    assert isinstance(scaled, ops.ScaledRows) and scaled.tiles == N // 16
    assert (res.double() - want).abs().max() <= 2.0 ** -20 * (want.abs().max() + K ** 0.5)
    normed = want * (want.square().mean(1, keepdim=True) + 1e-6).rsqrt() * norm.double()
    assert (scaled.materialize().double() - normed).abs().max() <= 2 * U * normed.abs().max()
    w2 = (torch.randn(2 * F, N, generator=g) / N ** 0.5).bfloat16().cuda()
    full = normed @ w2.double().T
    # every normed element carries one rounding to bfloat16
    slack = U * (normed.abs() @ w2.double().abs().T)
    y = ops.linear(scaled, w2, out_float32=True).double()
    assert ((y - full).abs() <= slack + 1e-5).all()
    if F % 64 == 0:
        act = ops.gated_linear(scaled, w2, "silu", ops.GATED_BLOCK).double()
        parts = full.view(M, F // 64, 2, 64)
        gate, up = parts[:, :, 0].reshape(M, F), parts[:, :, 1].reshape(M, F)
        want2 = torch.nn.functional.silu(gate) * up
        s = slack.view(M, F // 64, 2, 64)
        # |silu'| <= 1.1
        tol = 1.1 * s[:, :, 0].reshape(M, F) * (up.abs() + 1) + s[:, :, 1].reshape(M, F) * gate.abs() + U * want2.abs() + 1e-5
        assert ((act - want2).abs() <= tol).all()


def test_range():
    """What lies outside goes to the other kernels."""
    from tinyserve_b200.kernels import ops
    assert not ops._gemv_fits(9, 128, 128) and not ops._gemv_fits(1, 16, 4104) and not ops._gemv_fits(1, 8193, 1024)
    assert not ops._gemv_fits(1, 128, 2056, gated=True) and not ops._gemv_fits(1, 192, 128, gated=True)
    assert not ops._gemv_fits(1, 1040, 128, residual=True) and not ops._gemv_fits(1, 1000, 128, residual=True)


def test_blocks_that_have_a_place():
    """A block is four warps and more, 16 warps of them a multiprocessor: rows of a short K, blocks of a long one."""
    from tinyserve_b200.kernels import ops
    if ops.num_sms() != 148:
        pytest.skip("the numbers are those of 148 multiprocessors")
    fits = ops._gemv_fits
    assert fits(1, 9472, 256) and not fits(1, 9488, 256) and not fits(1, 65536, 64)
    assert fits(1, 16384, 512) and fits(1, 8192, 1024)                      # (a second wave of small blocks)
    assert fits(1, 4736, 1536) and not fits(1, 4752, 1536) and not fits(1, 2384, 3072)
    assert fits(1, 9472, 512, gated=True) and not fits(1, 9600, 512, gated=True) and not fits(1, 4864, 1536, gated=True)
    assert fits(1, 2048, 4096, residual=True) and not fits(1, 2064, 2048, residual=True) and not fits(1, 2048, 256, residual=True)


# sums of squares of 64, 65, 96 and 128 tiles, which come 32 at a time
@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K", [(1024, 3072), (1040, 512), (1536, 1536), (2048, 1024)])
def test_residual_then_a_product_by_tcgen05(M, N, K):
    """The next product's weights are too large for this kernel; the norm factor comes from the sums per 16 columns."""
    from tinyserve_b200.kernels import ops
    F = (1 << 23) // N // 64 * 64
    assert ops._gemv_fits(M, N, K, residual=True) and not ops._gemv_fits(M, 2 * F, N) and not ops._gemv_fits(M, 2 * F, N, gated=True)
    x, w = operands(M, N, K, 2)
    g = torch.Generator().manual_seed(6)
    res = torch.randn(M, N, generator=g).cuda()
    norm = (1 + 0.1 * torch.randn(N, generator=g)).bfloat16().cuda()
    want = res.double() + x.double() @ w.double().T
    scaled = ops.add_rmsnorm(ops.linear(x, w, allow_pending=True), res, norm, 1e-6, torch.bfloat16, scaled_ok=True)
    assert isinstance(scaled, ops.ScaledRows) and scaled.tiles == N // 16
    normed = want * (want.square().mean(1, keepdim=True) + 1e-6).rsqrt() * norm.double()
    w2 = (torch.randn(2 * F, N, generator=g) / N ** 0.5).bfloat16().cuda()
    full = normed @ w2.double().T
    # every normed element carries one rounding to bfloat16
    slack = U * (normed.abs() @ w2.double().abs().T)
    assert ((ops.linear(scaled, w2, out_float32=True).double() - full).abs() <= slack + 1e-5).all()
    act = ops.gated_linear(scaled, w2, "silu", ops.GATED_BLOCK).double()
    parts, s = full.view(M, F // 64, 2, 64), slack.view(M, F // 64, 2, 64)
    gate, up = parts[:, :, 0].reshape(M, F), parts[:, :, 1].reshape(M, F)
    want2 = torch.nn.functional.silu(gate) * up
    tol = 1.1 * s[:, :, 0].reshape(M, F) * (up.abs() + 1) + s[:, :, 1].reshape(M, F) * gate.abs() + U * want2.abs() + 1e-5
    assert ((act - want2).abs() <= tol).all()
    assert ops.gemm_tcgen05_error() == 0

"""The scratch of the paired product: captured graphs hold its address, so no later product may replace it, and it has
to hold what any product needs.  The sizes come from the kernel's own plan, which runs on the host."""
import random

import pytest
import torch


@pytest.fixture
def lib(monkeypatch):
    from tinyserve_b200.kernels import ops
    monkeypatch.setattr(ops, "_pair_scratch", {})
    monkeypatch.setattr(ops, "gemm_pairs", lambda: 74)
    monkeypatch.setattr(ops, "num_sms", lambda: 148)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return ops._gemm_pair()


def test_a_larger_need_leaves_the_scratch_where_it_is(lib):
    """51200 x 5120: 2,816 tokens need three times what 4,096 need."""
    from tinyserve_b200.kernels import ops
    first = ops._pair_workspace(lib, 4096, 51200, 5120, 74, 0, False, "cpu")
    for tokens in (2048, 3072, 2816, 6144):
        again = ops._pair_workspace(lib, tokens, 51200, 5120, 74, 0, False, "cpu")
        assert again[0] is first[0] and again[1] is first[1]
    more = ops._pair_workspace(lib, 4096, 51200, 5120, 80, 0, False, "cpu")
    assert more[0] is not first[0]
    assert ops._pair_workspace(lib, 4096, 51200, 5120, 74, 0, False, "cpu")[0] is first[0]


@pytest.mark.parametrize("pairs", [1, 3, 5, 20, 66, 74, 75, 148])
def test_every_plan_fits(lib, pairs):
    """(a product that needed more would raise)"""
    from tinyserve_b200.kernels import ops
    rng = random.Random(pairs)
    for _ in range(400):
        M, N, K = rng.randint(65, 8192), 8 * rng.randint(1, 8000), 8 * rng.randint(1, 3200)
        ops._pair_workspace(lib, M, N, K, pairs, rng.randint(0, 2), rng.random() < 0.3, "cpu")

"""How many cuts along K the gated product of a few tokens gets, against measured times."""
import pytest

# us on a B200 by number of cuts; clusters of 2 .. 8 blocks that the device holds at once
TIMES = {
    (1, 512, 2048): {1: 8.13, 2: 5.78, 4: 4.08, 8: 3.44}, (64, 512, 2048): {1: 14.67, 2: 19.58, 4: 11.38, 8: 7.25},
    (1, 6144, 1024): {1: 5.63, 2: 5.46, 3: 4.75, 4: 4.63, 5: 4.78, 6: 8.31, 8: 8.29}, (48, 6144, 1024): {1: 10.45, 2: 15.58, 4: 10.2, 5: 9.72, 6: 15.45, 8: 14.17},
    (1, 12288, 2048): {1: 11.28, 2: 11.3, 3: 14.49, 4: 13.8, 8: 15.65}, (64, 12288, 2048): {1: 17.72, 2: 24.84, 3: 32.87, 4: 28.0, 8: 28.25},
    (1, 9216, 4096): {1: 17.6, 2: 15.16, 3: 14.38, 4: 19.33, 8: 20.57}, (64, 9216, 4096): {1: 26.98, 2: 29.5, 3: 24.08, 4: 33.93, 8: 31.84},
    (1, 18816, 5120): {1: 32.97, 2: 30.84, 3: 33.85, 8: 38.17}, (64, 18816, 5120): {1: 40.57, 2: 45.79, 3: 54.29, 8: 63.83},
    (8, 24576, 4096): {1: 34.42, 2: 38.95, 3: 40.89, 8: 45.62},
}

PLACES = {2: 148, 3: 90, 4: 66, 5: 52, 6: 44, 7: 30, 8: 30}


@pytest.fixture(autouse=True)
def nothing_remembered():
    from tinyserve_b200.kernels import ops
    ops.gated_splits.cache_clear()
    yield
    ops.gated_splits.cache_clear()


@pytest.mark.parametrize("shape", TIMES)
def test_choice_is_close_to_the_best(shape, monkeypatch):
    from tinyserve_b200.kernels import ops
    monkeypatch.setattr(ops, "gemm_max_clusters", lambda M, splits: PLACES[splits])
    times, splits = TIMES[shape], ops.gated_splits(*shape)
    assert times[splits] <= 1.1 * min(times.values())


def test_cuts_have_slices_and_places(monkeypatch):
    from tinyserve_b200.kernels import ops
    monkeypatch.setattr(ops, "gemm_max_clusters", lambda M, splits: PLACES[splits])
    for K in (8, 64, 72, 128, 136, 192, 1024, 8192):
        for N in range(128, 40000, 640):
            for M in (1, 16, 17, 64):
                splits = ops.gated_splits(M, N, K)
                assert 1 <= splits <= ops.FUSED_MAX_SPLITS and (splits == 1 or (2 * splits <= -(-K // 64) and N // 128 <= PLACES[splits]))
    ops.gated_splits.cache_clear()
    monkeypatch.setattr(ops, "gemm_max_clusters", lambda M, splits: 0)          # a device that does not say
    assert ops.gated_splits(1, 512, 2048) == 1

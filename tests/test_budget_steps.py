"""Which steps with prompt portions are padded to a captured shape, and what the cache leaves free for their graphs.
The runner's rules alone, on the host."""
from types import SimpleNamespace as NS

import pytest

from tinyserve_b200.engine.batch import StepEntry
from tinyserve_b200.engine.runner import MIXED_GRAPH_TOKENS, ModelRunner


def runner(budget=2048, seqs=128, longest=16384, **more):
    r = ModelRunner.__new__(ModelRunner)
    r.cfg = NS(max_num_batched_tokens=budget, max_num_seqs=seqs, max_model_len=longest, **more)
    r.manager = NS(num_computed=lambda rid: 100)
    r.mixed_graphs_enabled = r.budget_graphs_enabled = True
    return r


def step(tokens, wants=None):
    """Entries of so many tokens; ``wants``: places wanted of each (default: the last)."""
    return [StepEntry(f"r{i}", [1] * n, [n - 1] if wants is None else list(range(wants[i]))) for i, n in enumerate(tokens)]


@pytest.mark.parametrize("budget", [300, 512, 700, 2048, 4096])
def test_a_step_of_the_whole_budget(budget):
    r = runner(budget)
    listed = budget in MIXED_GRAPH_TOKENS
    assert r._mixed_shape_for(step([1, budget - 1]))[:3] == (budget, 4, 4)
    assert r._mixed_shape_for(step([1, 1, 1, budget - 3]))[:3] == (budget, 8, 8)
    # portions alone, and steps that leave some of a large budget
    assert (r._mixed_shape_for(step([budget])) is not None) == listed
    if budget - 1 > MIXED_GRAPH_TOKENS[-1]:
        assert r._mixed_shape_for(step([1, budget - 2])) is None
    assert r._mixed_shape_for(step([1, 39]))[:3] == (48, 4, 4)


@pytest.mark.parametrize("budget", [300, 700, 2048, 4096])
def test_a_whole_budget_with_more_places_than_requests_runs_as_it_is(budget):
    """Padded it would take a row of logits for every token (4,096 x 151,936 floats are 2.5 GB)."""
    r = runner(budget)
    assert r._mixed_shape_for(step([1, budget - 1], [1, 3]))[:3] == (budget, 4, 4)
    assert r._mixed_shape_for(step([1, budget - 1], [1, 4])) is None
    assert r._mixed_shape_for(step([1, budget - 1], [1, budget - 1])) is None
    # smaller steps are padded to a row per token, as they always were
    assert r._mixed_shape_for(step([1, 39], [1, 39]))[:3] == (48, 4, 48)


@pytest.mark.parametrize("graphs", [False, True])
def test_the_cache_leaves_room_for_the_graphs_of_a_whole_budget(graphs, monkeypatch):
    """The captured step's activations and the kept logits beside those of an eager step; a cache that just holds the longest
    request is not refused for it."""
    import torch
    from tinyserve_b200.cache.device import DeviceCache
    per_page, page = 1 << 20, 64
    r = runner(4096, 64, 4096, num_blocks=0, gpu_memory_utilization=0.9, use_cuda_graphs=graphs)
    r.page_size, r.max_blocks, r.device, r.dtype = page, 1 << 20, "cuda:0", torch.bfloat16
    r.model = NS(vocab_size=151936, capturable=True)
    r._activation_bytes_per_token = lambda: 400_000
    monkeypatch.setattr(DeviceCache, "bytes_per_page", staticmethod(lambda *a: [per_page]))
    total = 180 << 30
    step, logits = 4096 * 400_000, 64 * 151936 * 4

    def pages(free):
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (free, total))
        return r._size_cache()

    left = int(0.9 * total) - (1 << 30)          # (a card with nothing on it)
    assert pages(total) * per_page + step + 2 * logits + (step + 16 * logits if graphs else 0) <= left
    # little room: as many pages as without graphs, up to those of the longest request
    few = int(0.1 * total) + step + 2 * logits + (1 << 30)
    assert pages(few + 65 * per_page + 4096) == 65
    assert pages(few + 80 * per_page + 4096) == (65 if graphs else 80)
    from tinyserve_b200.cache.manager import CacheError
    with pytest.raises(CacheError):
        pages(few + 64 * per_page + 4096)

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

"""Steps that use up the token budget with decoded tokens beside portions, replayed from graphs above the listed token counts:
library products, tcgen05 prefill over a padded work list and the paired product inside the capture, against the plain
implementation; and a capture of such a step that finds no memory."""
import pytest
import torch

import plain_qwen3 as plain
from helpers import make_model_dir, random_ids
from test_real_shapes_gpu import TOLERANCE, assert_no_kernel_gave_up, errors, make_folder

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def flagship(tmp_path_factory):
    folder = make_folder(tmp_path_factory.mktemp("flagship"), "flagship_layers", seed=31)
    cfg, weights = plain.load_folder(folder)
    return folder, cfg, {k: v.cuda() for k, v in weights.items()}


# 700 tokens: library products only; 2,048 and 3,456: the paired gate/up product, at 3,456 with less scratch (0.8 M floats)
# than the step of 3,000 that comes between the replays takes (2.8 M)
@pytest.mark.parametrize("budget,page,between", [(700, 16, 60), (2048, 64, 1500), (3456, 16, 3000)])
def test_replays_of_the_whole_budget(flagship, budget, page, between):
    from tinyserve_b200.config.engine_config import EngineConfig
    from tinyserve_b200.engine.batch import StepEntry
    from tinyserve_b200.engine.runner import ModelRunner
    from tinyserve_b200.kernels import ops
    folder, cfg, weights = flagship
    vocab, turns = cfg["vocab_size"], 7
    cut = (budget - 2) // 3
    lengths = {"long": budget - 2 - cut, "short": cut, "alone": between // 2, "rest": between - between // 2}
    prompts = {name: random_ids(vocab, n, seed=n) for name, n in lengths.items()}
    decoded = {"d0": random_ids(vocab, 40 + turns, seed=5), "d1": random_ids(vocab, 3 + turns, seed=6)}
    with torch.no_grad():
        ref = {name: plain.logits(cfg, weights, ids).cpu() for name, ids in {**prompts, **decoded}.items()}
    runner = ModelRunner(EngineConfig(model=folder, dtype="bfloat16", max_model_len=4096, block_size=page, max_num_seqs=8,
                                      max_num_batched_tokens=budget, num_blocks=8 * 4096 // page, use_cuda_graphs=True))
    runner.capture_decode_graphs([1, 8])
    tol_max, tol_rms = TOLERANCE[("flagship_layers", "bfloat16")]

    def check(entries, names):
        logits = runner.step(entries).cpu()
        for row, (e, name) in enumerate(zip(entries, names)):
            place = runner.manager.num_computed(e.rid) - 1
            e_max, e_rms = errors(logits[row], ref[name][place], ref[name].abs().max().item())
            assert e_max.item() <= tol_max and e_rms.item() <= tol_rms, f"{name} at place {place} of {len(ref[name])}"

    for rid in decoded:
        runner.manager.begin(rid)
    check([StepEntry(rid, ids[:-turns], [len(ids) - turns - 1]) for rid, ids in decoded.items()], list(decoded))
    at = {rid: len(ids) - turns for rid, ids in decoded.items()}
    for turn in range(turns):
        names = ["long", "short"]
        for name in names:
            runner.manager.begin(f"{name}{turn}")
        entries = [StepEntry(rid, [decoded[rid][at[rid] + turn]], [0]) for rid in decoded]
        entries += [StepEntry(f"{name}{turn}", prompts[name], [lengths[name] - 1]) for name in names]
        assert runner._mixed_shape_for(entries)[:3] == (budget, 8, 8)
        check(entries, list(decoded) + names)
        if turn == 4:
            for name in ("alone", "rest"):
                runner.manager.begin(f"{name}{turn}")
            check([StepEntry(f"{name}{turn}", prompts[name], [lengths[name] - 1]) for name in ("alone", "rest")], ["alone", "rest"])
            names += ["alone", "rest"]
        for name in names:
            runner.manager.free(f"{name}{turn}")
    captured = [k for k, v in runner.mixed_graphs.items() if not isinstance(v, int)]
    assert [k[0] for k in captured] == [budget] and runner.mixed_graph_replays == turns - 2
    assert_no_kernel_gave_up(cfg["head_dim"])
    assert ops.gemm_pair_error() == 0


def test_a_whole_budget_without_memory_leaves_the_smaller_graphs(tmp_path, monkeypatch):
    """A capture of a step of the whole budget that runs out of memory gives up those shapes; the listed ones are captured on."""
    from test_engine_gpu import greedy, llm_for
    from tinyserve_b200.engine.runner import MIXED_GRAPH_TOKENS, ModelRunner
    folder = make_model_dir(tmp_path, "A", seed=33)
    prompts = [random_ids(256, n, seed=n) for n in (30, 28, 26, 31, 29, 27, 45, 44, 43, 21)] * 3
    want = llm_for(folder, "float32", async_scheduling=False).generate(prompts, greedy(12))
    llm = llm_for(folder, "float32", use_cuda_graphs=True, max_num_batched_tokens=40, max_num_seqs=4)
    assert 40 not in MIXED_GRAPH_TOKENS
    shapes, tried = [], []
    graph_of, begin = ModelRunner._mixed_graph, torch.cuda.CUDAGraph.capture_begin

    def watched(self, prep):
        shapes.append(prep.mixed)
        return graph_of(self, prep)

    def no_memory(self, *args, **kwargs):
        if shapes and shapes[-1][0] == 40:
            tried.append(shapes[-1])
            raise torch.cuda.OutOfMemoryError("no memory for this capture (simulated)")
        return begin(self, *args, **kwargs)

    monkeypatch.setattr(ModelRunner, "_mixed_graph", watched)
    monkeypatch.setattr(torch.cuda.CUDAGraph, "capture_begin", no_memory)
    outs = llm.generate(prompts, greedy(12))
    assert len(tried) == 1 and not llm.runner.budget_graphs_enabled
    assert llm.runner.mixed_graphs_enabled and llm.runner.mixed_graph_replays > 0
    assert all(k[0] in MIXED_GRAPH_TOKENS for k in llm.runner.mixed_graphs)
    assert [o.token_ids for o in outs] == [o.token_ids for o in want]

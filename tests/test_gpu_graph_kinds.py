"""One decode graph serves steps that ask for token ids and steps that ask for logits alone, whichever kind it was captured for."""
import pytest
import torch

from helpers import make_model_dir, plain_inputs, random_tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first_asks_for_ids", [True, False])
def test_both_kinds_of_step_share_a_graph(tmp_path, first_asks_for_ids):
    from inf_engine_b200 import ModelRunner, StepEntry
    from inf_engine_b200.sampling.sampler import SamplingConfig, SamplingMode, pack_rows
    d = make_model_dir(tmp_path, "tiny_a")
    vocab = plain_inputs(d)[0]["vocab_size"]
    runner = ModelRunner.from_dir(d, dtype="float32", page_size=8, n_pages=64, max_requests=4)
    configs = [SamplingConfig(), SamplingConfig(mode=SamplingMode.TOP_K, temperature=0.8, top_k=20, seed=3), SamplingConfig()]
    for i in range(3):
        runner.open(i)
    runner.step([StepEntry(i, random_tokens(vocab, 4 + i, i), []) for i in range(3)])
    alone = ModelRunner.from_dir(d, dtype="float32", page_size=8, n_pages=64, max_requests=4, use_graphs=False)
    for i in range(3):
        alone.open(i)
    alone.step([StepEntry(i, random_tokens(vocab, 4 + i, i), []) for i in range(3)])
    tokens = [5, 6, 7]
    for step in range(6):
        entries = [StepEntry(i, [t], [0]) for i, t in enumerate(tokens)]
        rows = pack_rows(configs, [100 * step + i for i in range(3)], vocab)
        asks = (step % 2 == 0) == first_asks_for_ids
        logits, ids = runner.step_and_sample(entries, rows if asks else None)
        want_logits, want_ids = alone.step_and_sample(entries, rows)
        assert torch.equal(logits, want_logits) and (ids is None) == (not asks)
        if asks:
            assert ids.tolist() == want_ids.tolist()
        tokens = want_ids.tolist()
    assert runner.graphs.captures == 1 and runner.graphs.replays == 5

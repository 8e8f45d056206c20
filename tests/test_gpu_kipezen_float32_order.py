"""The 32-bit path of a model with both recurrences, gates and experts gives a sequence the same bits whatever else the step
holds and however it was cut into steps: its sums have one order each (sizes here reach every other form that bfloat16 steps
take: chunks of the delta rule, runs of the recurrence, gate products of a few rows)."""
import pytest
import torch

from helpers import random_tokens
from kipezen_models import _delta, _model, _moe, _par, make_kipezen_dir

pytestmark = pytest.mark.gpu
CONFIG = _model(300, 256, 1e-5, [
    _delta(4, 2, 64, 64, 4, _moe(64, 8, 2, 2, 1, 1.5, 64)),
    _par(4, 2, 64, 64, 0.125, (10000.0, 32), 90, 4, 256, 4, 4, 1.0, 1.0, _moe(64, 4, 2, 2, 2, 2.0, None)),
])


def test_float32_bits_depend_neither_on_the_step_nor_on_the_cut(tmp_path):
    from inf_engine_b200 import ModelRunner, StepEntry
    r = ModelRunner.from_dir(make_kipezen_dir(tmp_path, "float32_order", config=CONFIG), dtype="float32", page_size=16, n_pages=128,
                             max_requests=40)
    long, short = random_tokens(300, 300, 1), random_tokens(300, 16, 2)
    others = [(("other", i), random_tokens(300, 3 + i, 10 + i)) for i in range(20)]

    def run(rid, tokens, sizes, beside):
        """Logits of every place of ``tokens``; with ``beside`` each step also decodes a token of twenty requests and runs a prompt."""
        r.open(rid)
        out, at = [], 0
        for i, n in enumerate(sizes):
            es = [StepEntry(rid, tokens[at:at + n], list(range(n)))]
            if beside:
                es += [StepEntry(o, [7 + i], [0]) for o, _ in others]
                r.open(("prompt", i))
                es.append(StepEntry(("prompt", i), random_tokens(300, 70, 50 + i), [69]))
            out.append(r.step(es)[:n].clone())
            if beside:
                r.close(("prompt", i))
            at += n
        r.close(rid)
        return torch.cat(out)

    for o, toks in others:
        r.open(o)
    r.step([StepEntry(o, toks, []) for o, toks in others])
    want = run("a", long, [300], False)
    assert torch.equal(run("b", long, [300], True), want)
    assert torch.equal(run("c", long, [200, 17, 83], False), want)
    assert torch.equal(run("d", long, [120, 180], True), want)
    assert torch.equal(run("e", short, [16], True), run("f", short, [16], False))

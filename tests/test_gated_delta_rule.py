"""When a step of the gated delta rule goes in chunks: the choice follows what both forms were measured to take, and
a step that finds no memory for chunks goes token after token."""
import pytest
import torch

from inf_engine_b200.parts import gated_delta
from inf_engine_b200.parts.gated_delta import chunks_pay


# us measured on a B200: (tokens of each request, heads, key size, value size, token after token, in chunks)
MEASURED = [
    ([64], 32, 64, 64, 41, 52), ([128], 32, 64, 64, 79, 55), ([512], 32, 64, 64, 307, 73), ([2048], 32, 64, 64, 1224, 292),
    ([512], 64, 64, 64, 309, 133), ([512], 4, 64, 64, 304, 58), ([200] + [1] * 32, 32, 64, 64, 144, 278),
    ([128] * 8, 32, 64, 64, 104, 138), ([300] * 3, 32, 64, 64, 183, 130), ([512] * 8, 32, 64, 64, 411, 531),
    ([33, 400, 1], 32, 64, 64, 243, 77), ([300] * 3, 32, 64, 128, 196, 225), ([200] + [1] * 32, 32, 64, 128, 158, 453),
    ([512], 64, 128, 64, 351, 220), ([300] * 3, 32, 128, 64, 209, 217), ([128], 32, 96, 96, 89, 71), ([300] * 3, 32, 96, 96, 204, 243),
    ([128], 32, 128, 128, 116, 77), ([300] * 3, 32, 128, 128, 268, 367), ([200] + [1] * 32, 32, 128, 128, 214, 727),
    ([200] + [1] * 32, 32, 48, 48, 150, 203), ([300] * 3, 32, 80, 80, 185, 214), ([512] * 8, 32, 80, 80, 624, 821),
    ([200] + [1] * 32, 32, 128, 32, 160, 298), ([128], 32, 128, 32, 89, 66), ([128] * 8, 32, 32, 32, 114, 80),
]


@pytest.mark.parametrize("q_lens,heads,dk,dv,chain,chunks", MEASURED)
def test_the_faster_form_is_taken(q_lens, heads, dk, dv, chain, chunks):
    assert chunks_pay(q_lens, heads, dk, dv) == (chunks < chain)


def test_decode_tokens_count_as_chunks():
    assert chunks_pay([200], 32, 64, 64) and not chunks_pay([200] + [1] * 32, 32, 64, 64)
    assert not chunks_pay([1] * 64, 32, 64, 64)


def test_no_memory_for_chunks_is_no_error(monkeypatch):
    got = gated_delta.chunk_scratch(1000, "cpu")
    assert got.numel() == 1000 and got.dtype is torch.float32
    assert gated_delta.chunk_scratch(0, "cpu") is None and gated_delta.chunk_scratch(gated_delta.CHUNK_MAX_SCRATCH + 1, "cpu") is None

    def full(*args, **kw):
        raise torch.OutOfMemoryError("CUDA out of memory")

    monkeypatch.setattr(torch, "empty", full)
    assert gated_delta.chunk_scratch(1000, "cpu") is None

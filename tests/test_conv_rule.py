"""When the short convolution takes runs of tokens: the choice follows what both forms were measured to take."""
import pytest

from inf_engine_b200.kernels import conv_runs_pay

# us measured on a B200: (channels, taps, tokens of each request, a thread a token, runs)
MEASURED = [
    (64, 4, [8], 3.2, 7.7), (3072, 4, [16], 4.6, 7.7), (2048, 4, [32], 6.4, 7.6), (512, 4, [61], 9.7, 7.7), (3072, 4, [61], 10.1, 7.8),
    (2048, 4, [2048], 47.4, 15.6), (3072, 4, [2048], 67.6, 23.1), (2048, 4, [8] * 8, 6.0, 8.3), (2048, 4, [24] * 8, 10.5, 7.7),
    (1024, 4, [24] * 8, 6.0, 7.8), (3072, 4, [40] * 8, 15.1, 8.2), (3072, 4, [200] + [1] * 32, 33.5, 35.6),
    (2048, 4, [100] + [1] * 60, 30.0, 40.9), (3072, 4, [64] + [1] * 63, 40.0, 60.8), (6144, 4, [61] + [1] * 7, 14.7, 20.6),
    (3072, 4, [600] + [1] * 60, 91.5, 71.8), (2048, 4, [2000] + [1] * 32, 96.5, 49.5), (3072, 2, [61], 8.1, 8.7),
    (1024, 2, [300], 8.4, 9.2), (2048, 2, [2048], 37.9, 8.3), (512, 2, [300, 5, 1, 1], 8.5, 11.2), (6144, 2, [40] * 8, 22.4, 7.9),
]


@pytest.mark.parametrize("channels,taps,q_lens,tokens,runs", MEASURED)
def test_the_faster_form_is_taken(channels, taps, q_lens, tokens, runs):
    assert conv_runs_pay(sum(q_lens), len(q_lens), max(q_lens), channels, taps) == (runs < tokens)

"""RoutedExperts: which kernel takes a step is a function of the block's sizes and the number of tokens alone.  No GPU: nothing is launched."""
import pytest
import torch

from mistralrs_b200 import mixers, seq_ops


def _block(E=16, top=4, W=2048, ff=2048):
    weights = torch.empty(E, 2 * ff, W, dtype=torch.bfloat16), torch.empty(E, W, ff, dtype=torch.bfloat16)      # never read
    return mixers.RoutedExperts(torch.zeros(E, W), torch.zeros(E), *weights, top, 1, 1, seq_ops.ACT_SILU)


@pytest.mark.parametrize("tokens", [1, 3, 4, 7, 8, 16])
def test_streams_weights_does_not_depend_on_earlier_questions(tokens):
    fresh, asked = _block(), _block()
    asked.groups_weights(tokens)
    assert fresh.streams_weights(tokens) == asked.streams_weights(tokens)
    if tokens == 8:      # 32 pairs of 25 MB: the one-launch products' work, not the streaming kernels'
        assert not _block().streams_weights(tokens)

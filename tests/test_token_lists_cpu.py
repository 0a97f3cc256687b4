"""Token lists that the extension reads directly and those it leaves to the general caster give the same results."""
import numpy as np
import pytest
import torch

from chunk_attn import PrefixTree, SpanBatch

IDS = [3, 0, -5, 2 ** 31 - 1, -2 ** 31]


@pytest.mark.parametrize("given", [IDS, tuple(IDS), np.array(IDS, np.int32), [np.int64(x) for x in IDS], [3, np.int32(0)] + IDS[2:]])
def test_same_ids(given):
    t = PrefixTree(8, 16)
    t.add_seq(given)
    assert t.tails[0].tokens == IDS


@pytest.mark.parametrize("given", [[1, 2.5], ["a"], [2 ** 31], [-2 ** 31 - 1], "12", 5, [None], [[1]]])
def test_refused(given):
    t = PrefixTree(8, 16)
    with pytest.raises(TypeError):
        t.add_seq(given)
    assert len(t.tails) == 0
    with pytest.raises(TypeError):
        SpanBatch([[1], given], [0, 0], [0, 1], torch.device("cpu"))
    assert t.add_seq([True, 7]) == 0 and t.tails[0].tokens == [1, 7]

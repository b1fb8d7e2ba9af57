"""What a step refuses before anything reaches the device (no device)."""

from array import array
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import tesseract_b200.parts  # noqa: F401
from tesseract_b200.cache import CacheManager
from tesseract_b200.engine.step import StepEntry, StepError, Stepper
from tesseract_b200.parts import PagedKVNeed


def stepper():
    cache = CacheManager([PagedKVNeed(2, 16)], [None], num_pages=8, page_size=16, max_requests=2, dtype=torch.float32,
                         device="cpu", max_step_tokens=8, allocate_storage=False)
    assert cache.admit("a")
    return Stepper(SimpleNamespace(runtime=SimpleNamespace(device=torch.device("cpu")),
                                   spec=SimpleNamespace(vocab_size=100, max_positions=64)), cache)


@pytest.mark.parametrize("tokens", [{5}, {0: 5}, b"\x05", "5", [5.0], [True], [[5]], [None], [100], [-1], (2 ** 40,)])
def test_a_single_token_that_is_no_list_of_integers_is_refused_with_the_step(tokens):
    with pytest.raises(StepError):
        stepper()._validate([StepEntry("a", tokens, [0])])


@pytest.mark.parametrize("tokens", [[5], (5,), range(5, 6), np.array([5]), torch.tensor([5]), array("i", [5]), bytearray(b"\x05"),
                                    [np.int64(5)]])
def test_a_single_token_of_any_sequence_of_integers_is_taken(tokens):
    assert [int(t) for t in stepper()._validate([StepEntry("a", tokens, [0])])[0]] == [5]

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


ROWS, HEADS, KV, DIM, RANK, PAGE = 3, 4, 2, 64, 128, 16


def index_readers(kernels):
    """Calls of the functions whose kernels read the step's index arrays in front of the wait for the kernel before them."""
    positions, of_row, table = torch.zeros(ROWS, dtype=torch.int32), torch.zeros(ROWS, dtype=torch.int32), torch.zeros(1, 1, dtype=torch.int32)

    def bf16(*shape):
        return torch.zeros(shape, dtype=torch.bfloat16)

    cache, entry = bf16(2, PAGE * 1024), RANK + 32
    return {
        "pair_rope_cache": lambda **kw: kernels.pair_rope_cache(
            bf16(ROWS, (HEADS + 2 * KV) * DIM), bf16(ROWS, HEADS * DIM), cache, positions, of_row, table, None, q_heads=HEADS, key_heads=KV,
            value_heads=KV, dim=DIM, vdim=DIM, rot_dims=0, page_size=PAGE, **kw),
        "latent_rope_cache": lambda **kw: kernels.latent_rope_cache(
            torch.zeros(ROWS, entry), bf16(ROWS, HEADS * (DIM + 32)), bf16(ROWS, HEADS * entry), cache, torch.ones(RANK), positions, of_row,
            table, None, heads=HEADS, dim=DIM, rank=RANK, rot_width=32, rot_dims=0, page_size=PAGE, eps=1e-5, **kw),
        "attention_rows_mma": lambda **kw: kernels.attention_rows_mma(
            bf16(ROWS, HEADS * DIM), bf16(ROWS, HEADS * DIM), cache, positions, of_row, table, heads=HEADS, kv_heads=KV, dim=DIM, vdim=DIM,
            page_size=PAGE, mask_kind=kernels.MASK_CAUSAL, mask_size=0, scale=1.0, **kw),
        "attention_latent_mma": lambda **kw: kernels.attention_latent_mma(
            bf16(ROWS, HEADS * entry), bf16(ROWS, HEADS * RANK), cache, positions, of_row, table, heads=HEADS, dim=entry, vdim=RANK,
            page_size=PAGE, mask_kind=kernels.MASK_CAUSAL, mask_size=0, scale=1.0, **kw),
    }


@pytest.mark.parametrize("name", ["pair_rope_cache", "latent_rope_cache", "attention_rows_mma", "attention_latent_mma"])
def test_a_kernel_reads_index_arrays_early_only_where_its_caller_vouches_for_them(name, monkeypatch):
    """The last number in front of the stream says whether the kernel may begin while the one in front of it still runs: by default it
    may not, for that one may be what writes the positions or the block table."""
    from tesseract_b200 import kernels

    early = []

    class Library:
        def tb_attention_latent_mma_splits(self, rows, heads):
            return 1

        def __getattr__(self, entry):
            assert entry == "tb_" + name
            return lambda *args: early.append(args[-2].value) or 0

    monkeypatch.setattr(kernels, "load_library", lambda source: Library())
    monkeypatch.setattr(kernels, "_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_stream", lambda: None)
    call = index_readers(kernels)[name]
    call()
    call(indices_copied=False)
    call(indices_copied=True)
    assert early == [0, 0, 1]

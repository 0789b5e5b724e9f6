"""What the sampler hands to its kernel: one number a row, whatever rows share the step, and errors for what does not fit.
On the CPU, with the kernel replaced by one that keeps its arguments."""
import pytest
import torch

from spyinfer_b200 import kernels
from spyinfer_b200.sampling import Sampler, SamplingParams


@pytest.fixture
def handed_over(monkeypatch):
    calls = []

    def sample(logits, tokens, *rest):
        calls.append([None if r is None else r.tolist() for r in rest])
        return tokens

    monkeypatch.setattr(kernels, "sample", sample)
    return calls


def test_every_row_gets_its_own_numbers(handed_over):
    params = [SamplingParams(temperature=0.5 * r, seed=2 ** 62 + r - 3, top_k=3 * (r % 2)) for r in range(5)]
    Sampler("cpu").sample(torch.zeros(5, 8), params, range(10, 15))
    temperatures, seeds, draws, top_k = handed_over[0]
    assert temperatures == [0.0, 0.5, 1.0, 1.5, 2.0] and seeds == [2 ** 62 + r - 3 for r in range(5)] and draws == list(range(10, 15)) and top_k == [0, 3, 0, 3, 0]
    Sampler("cpu").sample(torch.zeros(1, 8), [SamplingParams(temperature=1.0, seed=-1)], [2 ** 63 - 1])
    assert handed_over[1] == [[1.0], [-1], [2 ** 63 - 1], None]


def test_top_k_that_no_row_uses_may_be_of_any_size(handed_over):
    params = [SamplingParams(top_k=2 ** 40), SamplingParams(temperature=1.0)]
    Sampler("cpu").sample(torch.zeros(2, 8), params, [0, 0])
    assert handed_over[0][3] is None
    with pytest.raises(RuntimeError):
        Sampler("cpu").sample(torch.zeros(3, 8), params + [SamplingParams(temperature=1.0, top_k=4)], [0, 0, 0])


@pytest.mark.parametrize("rows,given,draws", [(3, 1, 3), (3, 3, 1), (2, 3, 2), (1, 2, 2)])
def test_one_entry_a_row(handed_over, rows, given, draws):
    with pytest.raises(kernels.KernelError):
        Sampler("cpu").sample(torch.zeros(rows, 8), [SamplingParams(temperature=1.0)] * given, [0] * draws)


@pytest.mark.parametrize("seed", [2 ** 63, -2 ** 63 - 1])
def test_a_seed_beyond_64_bits_is_a_value_error(handed_over, seed):
    with pytest.raises(ValueError):
        Sampler("cpu").sample(torch.zeros(2, 8), [SamplingParams(temperature=1.0), SamplingParams(temperature=1.0, seed=seed)], [0, 0])

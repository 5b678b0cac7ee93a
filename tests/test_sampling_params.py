"""Sampling parameters on their way to the kernels, which count in 32 bits."""
import numpy as np
import pytest

from pulsar_b200.sampling.sampler import GenerationParams


@pytest.mark.parametrize("top_k", [2 ** 31, 2 ** 32 + 5, 3e9, float("nan"), float("inf"), np.int64(2 ** 33)])
def test_a_top_k_beyond_32_bits_is_refused_and_not_cut(top_k):
    with pytest.raises(ValueError):
        GenerationParams(temperature=0.8, top_k=top_k).validate()
    with pytest.raises((ValueError, OverflowError)):
        GenerationParams(temperature=0.8, top_k=top_k).device_top_k()
    greedy = GenerationParams(temperature=0.0, top_k=top_k)              # no use for it: taken as before, and kept from the rows beside it
    greedy.validate()
    assert greedy.device_top_k() == 0


@pytest.mark.parametrize("top_k,number", [(0, 0), (40, 40), (40.0, 40), (40.7, 40), (True, 1), (np.int64(7), 7), (np.float32(9), 9), (2 ** 31 - 1, 2 ** 31 - 1)])
def test_a_top_k_that_fits_is_taken_whatever_its_type(top_k, number):
    p = GenerationParams(temperature=0.8, top_k=top_k)
    p.validate()
    assert p.device_top_k() == number and type(p.device_top_k()) is int


@pytest.mark.gpu
def test_rows_take_their_own_top_k():
    """A whole number given as a float is the same filter; a greedy row's number beyond 32 bits disturbs nobody."""
    import torch
    from pulsar_b200.sampling.sampler import Sampler
    logits = torch.randn(3, 500, generator=torch.Generator().manual_seed(1)).cuda() * 2
    first = None
    for k, beside in ((3, 0), (3.0, 2 ** 40)):
        params = [GenerationParams(temperature=0.9, top_k=k), GenerationParams(temperature=0.0, top_k=beside), GenerationParams(temperature=0.9, top_k=k)]
        got = Sampler("cuda:0").sample_on_device(logits, params, (), [0.3, 0.0, 0.9]).tolist()
        assert first is None or got == first
        first = got
    assert first[1] == int(logits[1].argmax())
    for row in (0, 2):
        assert first[row] in logits[row].topk(3).indices.tolist()

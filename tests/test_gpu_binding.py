"""GPU: arguments that the CPython binding passes on directly and arguments that are converted first give the same results."""
import pytest
import torch

from tallax_b200 import sampling, tax, tumpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["strided", "lists", "other_types", "numpy_key"])
def test_converted_arguments_give_the_same_results(cuda, how):
    gen = torch.Generator(device=cuda).manual_seed(5)
    x = torch.randn((6, 3000), generator=gen, device=cuda)
    top_k = torch.tensor([1, 5, 0, 50, 700, 2], dtype=torch.int32, device=cuda)
    top_p, temperature = torch.full((6,), 0.9, device=cuda), torch.full((6,), 0.8, device=cuda)
    index = torch.randint(0, 3000, (6, 40), generator=gen, device=cuda, dtype=torch.int32)
    key, y, i = (3, 4), x, index
    md = sampling.SamplingMetadata(top_k, top_p, temperature)
    if how == "strided":
        y = torch.stack([x, x], dim=2)[:, :, 0]
        assert not y.is_contiguous()
    elif how == "lists":
        md = sampling.SamplingMetadata(top_k.tolist(), 0.9, temperature.tolist())
    elif how == "other_types":
        md = sampling.SamplingMetadata(top_k.long(), top_p.double(), temperature)
        i = index.long()
    else:
        import numpy as np
        key = np.array(key, np.uint32)
    want = sampling.sample((3, 4), x, sampling.SamplingMetadata(top_k, top_p, temperature))
    assert torch.equal(sampling.sample(key, y, md), want)
    for a, b in zip(tax.top_k(y, 9, block_token=1), tax.top_k(x, 9, block_token=1)):
        assert torch.equal(a, b)
    for a, b in zip(tax.sort([y], num_keys=1, return_argsort=True), tax.sort([x], num_keys=1, return_argsort=True)):
        assert torch.equal(a, b)
    assert torch.equal(tumpy.take_along_axis(y, i, 1), tumpy.take_along_axis(x, index, 1))
    assert torch.equal(tax.cumsum(y, 1), tax.cumsum(x, 1))


def test_errors_keep_their_classes(cuda):
    x = torch.randn((4, 100), device=cuda)
    with pytest.raises(ValueError):
        tax.top_k(x, 101, block_token=1)
    with pytest.raises(NotImplementedError):
        tax.cumsum(x.half(), 1)
    with pytest.raises(ValueError):
        tumpy.take_along_axis(x, torch.zeros((3, 2), dtype=torch.int32, device=cuda), 1)

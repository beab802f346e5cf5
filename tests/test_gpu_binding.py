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


@pytest.mark.parametrize("op", ["sample", "top_k", "sort", "take_along_axis", "cumsum"])
def test_declined_allocation_is_torchs_own_error(cuda, op):
    x = torch.zeros((128, 1 << 17), device=cuda)               # 64 MB; every call below wants more than 8 MB
    index = torch.zeros((128, 1 << 17), dtype=torch.int32, device=cuda)
    md = sampling.SamplingMetadata(torch.full((1024,), 5, dtype=torch.int32, device=cuda), torch.ones(1024, device=cuda),
                                   torch.ones(1024, device=cuda))
    logits = torch.zeros((1024, 1 << 15), dtype=torch.bfloat16, device=cuda)
    call = {"sample": lambda: sampling.sample((1, 2), logits, md),
            "top_k": lambda: tax.top_k(x.reshape(-1, 1 << 11), 1 << 11, block_token=1),
            "sort": lambda: tax.sort([x], num_keys=1),
            "take_along_axis": lambda: tumpy.take_along_axis(x, index, 1),
            "cumsum": lambda: tax.cumsum(x, 1)}[op]
    call()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (1 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    call()

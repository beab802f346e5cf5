"""GPU: the radix sort at the edges of its CTAs and clusters, with ties, -0, NaNs, infinities and small integers."""
import numpy as np
import pytest

from oracle import tallax_oracle as o
from tallax_b200 import tax
from tests.conftest import exact_match, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1025, 8192, 8193, 16384, 16385, 32769, 131072, 131073])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16", "i32"])
@pytest.mark.parametrize("descending", [False, True])
def test_radix_sort_sizes(cuda, dtype, n, descending):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((4, n)).astype(np.float32) * 3
    x[1] = np.round(x[1])
    x[2] = 1.0
    if dtype == "i32":
        x = (x * 1000).astype(np.int32)
        x[3] = rng.integers(-2**31, 2**31 - 1, n)
    else:
        x[3, ::7] = 0.0
        x[3, 1::7] = -0.0
        x[3, 2::7] = np.nan
        x[3, 3::7] = np.inf
        x[3, 4::7] = -np.inf
        x = x.astype({"f32": np.float32, "f16": np.float16, "bf16": o.bfloat16}[dtype])
    first = rng.integers(0, 5, x.shape).astype(np.int32)
    for operands, keys in (([x], 1), ([first, x], 2)):
        got = tax.sort([to_dev(a, cuda) for a in operands], num_keys=keys, is_stable=True, return_argsort=True, descending=descending)
        exp = o.sort(operands, keys, is_stable=True, return_argsort=True, descending=descending)
        for g, e in zip(got, exp):
            assert exact_match(to_np(g), e)


@pytest.mark.parametrize("rows", [1, 300])
def test_radix_sort_row_counts(cuda, rows):
    x = np.random.default_rng(rows).standard_normal((rows, 3001)).astype(np.float32)
    keys, perm = tax.sort([to_dev(x, cuda)], num_keys=1, return_argsort=True)
    assert np.array_equal(to_np(perm), np.argsort(x, axis=1, kind="stable")) and np.array_equal(to_np(keys), np.sort(x, axis=1))


# many rows: clusters of CTAs of 8192 elements (three become four), and of 16384 for the longest rows
@pytest.mark.parametrize("dtype,rows,n", [("f32", 160, 8193), ("bf16", 80, 20001), ("f32", 40, 65536), ("i32", 24, 65537)])
def test_radix_sort_many_rows(cuda, dtype, rows, n):
    rng = np.random.default_rng(n)
    x = np.round(rng.standard_normal((4, n)).astype(np.float32) * 300)
    x = x.astype({"f32": np.float32, "bf16": o.bfloat16, "i32": np.int32}[dtype])
    v, i = tax.sort([to_dev(np.tile(x, (rows // 4, 1)), cuda)], num_keys=1, is_stable=True, return_argsort=True)
    ev, ei = o.sort([x], 1, is_stable=True, return_argsort=True)
    assert np.array_equal(to_np(i), np.tile(ei, (rows // 4, 1)))
    assert exact_match(to_np(v), np.tile(ev, (rows // 4, 1)))


# many rows in one CTA each: rows that end in the first, a middle and the last warp, inside a group of 32 and at its end
@pytest.mark.parametrize("dtype", ["f32", "bf16", "i32"])
@pytest.mark.parametrize("n", [1025, 1057, 1500, 2048, 2049, 3000, 3073, 4096, 4097])
def test_radix_sort_places_past_the_end(cuda, dtype, n):
    rng = np.random.default_rng(n)
    x = np.round(rng.standard_normal((4, n)).astype(np.float32) * 300)
    x[1] = x[1, 0]
    if dtype == "i32":
        x = x.astype(np.int32)
        x[2, ::5] = 2**31 - 1                                  # the key that the places past the end carry
        x[3, ::3] = -2**31
    else:
        x[2, ::5] = np.nan
        x[3, ::3] = -np.inf
        x = x.astype({"f32": np.float32, "bf16": o.bfloat16}[dtype])
    rows = 300
    payload = rng.integers(0, 1 << 30, x.shape).astype(np.int32)
    for descending in (False, True):
        got = tax.sort([to_dev(np.tile(a, (rows // 4, 1)), cuda) for a in (x, payload)], num_keys=1, is_stable=True,
                       return_argsort=True, descending=descending)
        exp = o.sort([x, payload], 1, is_stable=True, return_argsort=True, descending=descending)
        for g, e in zip(got, exp):
            assert exact_match(to_np(g), np.tile(e, (rows // 4, 1)))


# no scratch is allocated that no kernel touches, by the binding or by the wrapper behind it; beyond 131072 elements it is needed
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("rows,n,copies", [(64, 65536, 0), (32, 131072, 0), (8, 131073, 4)])
def test_sort_allocates_what_it_uses(cuda, rows, n, copies, strided):
    import torch

    from tallax_b200._src import ops
    x = torch.randn((rows, n), device=cuda)
    if strided:
        x = x.t().contiguous().t()
    one = rows * n * 4
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    keys, perm = ops.argsort_rows(x)
    used = torch.cuda.max_memory_allocated() - before
    # keys, permutation, the contiguous copy of a strided operand, and the composites (8 bytes each, padded to a power of two)
    assert (2 + strided + copies) * one <= used + 4096 and used <= (2 + strided + copies) * one * 1.01 + (1 << 20)
    assert np.array_equal(to_np(perm), np.argsort(to_np(x), axis=1, kind="stable"))

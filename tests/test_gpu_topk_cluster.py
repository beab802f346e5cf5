"""GPU: top-k of fewer than 256 rows (a row over a cluster's shared memory) at the edges of its parts and lists."""
import numpy as np
import pytest

from oracle import tallax_oracle as o
from tallax_b200 import tax
from tests.conftest import exact_match, to_dev, to_np

pytestmark = pytest.mark.gpu


# all elements candidates (<= 2048) and just not; parts that end inside a vector; odd row starts; sixteen CTAs; more
# candidates than are ordered by counting; fewer finite elements than k; ties, NaNs, sorted rows
@pytest.mark.parametrize("n,k", [(1, 1), (7, 3), (2048, 1000), (2049, 64), (4099, 128), (40961, 1024), (70001, 200), (262147, 50)])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
def test_cluster_top_k_sizes(cuda, dtype, n, k):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((9, n)).astype(np.float32) * 2
    x[1] = np.round(x[1])
    x[2] = 1.5
    x[3] = np.sort(x[3])
    x[4, max(1, k // 2):] = -np.inf
    x[5, ::max(1, n // 5)] = np.nan
    x[6, ::2] = 0.0
    x[6, 1::2] = -0.0
    x[7] = np.sort(x[7])[::-1]
    x = x.astype({"f32": np.float32, "f16": np.float16, "bf16": o.bfloat16}[dtype])
    v, i = tax.top_k(to_dev(x, cuda), k, block_token=1)
    ev, ei = o.top_k(x, k)
    assert np.array_equal(to_np(i), ei)
    assert exact_match(to_np(v), ev)


# the lines between the cluster form and the one-pass kernel: lists of 128, 256, 512 and more candidates to order
@pytest.mark.parametrize("rows,n,k", [(3, 256, 256), (3, 257, 256), (3, 2048, 128), (3, 2049, 128), (200, 2050, 200), (5, 11999, 201), (5, 12000, 201), (5, 12001, 440),
                                      (8, 20 * 441 - 1, 441), (8, 20 * 441, 441), (9, 40 * 500 - 1, 500), (9, 40 * 500, 500)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_top_k_at_the_lines_of_the_cluster_form(cuda, dtype, rows, n, k):
    x = np.random.default_rng(n).standard_normal((rows, n)).astype(np.float32) * 2
    x[1] = np.round(x[1])
    x = x.astype({"f32": np.float32, "bf16": o.bfloat16}[dtype])
    v, i = tax.top_k(to_dev(x, cuda), k, block_token=1)
    ev, ei = o.top_k(x, k)
    assert np.array_equal(to_np(i), ei)
    assert exact_match(to_np(v), ev)

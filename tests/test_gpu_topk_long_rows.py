"""GPU: top-k of many rows of more than 128 KB (bound from an eighth of the row, noted vectors) at its edges."""
import numpy as np
import pytest

from oracle import tallax_oracle as o
from tallax_b200 import tax
from tests.conftest import exact_match, to_dev, to_np

pytestmark = pytest.mark.gpu


# just past 128 KB, whole groups of eight pieces and one vector more, odd row starts, the longest row whose vectors
# have 16-bit numbers and one vector more; ties, NaNs, sorted rows, everything large in or outside the sampled pieces,
# the greatest elements many octaves apart
@pytest.mark.parametrize("dtype,n,k", [("f32", 32769, 128), ("f32", 40964, 1), ("f32", 262144, 128), ("f32", 262148, 50),
                                       ("bf16", 65537, 128), ("bf16", 81920, 64), ("f16", 65541, 128), ("f16", 98312, 20)])
def test_long_row_top_k_sizes(cuda, dtype, n, k):
    rng = np.random.default_rng(n)
    x = np.tile(rng.standard_normal((16, n)).astype(np.float32) * 2, (16, 1))
    piece = np.arange(n) * (4 if dtype == "f32" else 2) // 4096 % 8
    x[1] = np.round(x[1])
    x[2] = 1.5
    x[3] = np.sort(x[3])
    x[4, max(1, k // 2):] = -np.inf
    x[5, ::n // 5] = np.nan
    x[6, ::2] = 0.0
    x[6, 1::2] = -0.0
    x[7] = np.sort(x[7])[::-1]
    x[8] += 9 * (piece == 0)
    x[9] += 9 * (piece == 3)
    x[10, :3000] = 50
    x[11] = np.minimum(np.exp(2 * x[11]), 6e4)
    x[12] = -np.minimum(np.exp(2 * x[12]), 6e4)
    x = x.astype({"f32": np.float32, "f16": np.float16, "bf16": o.bfloat16}[dtype])
    v, i = tax.top_k(to_dev(x, cuda), k, block_token=1)
    ev, ei = o.top_k(x[:32], k)
    ev, ei = (np.concatenate([a[:16], np.tile(a[16:], (15, 1))]) for a in (ev, ei))
    assert np.array_equal(to_np(i), ei)
    assert exact_match(to_np(v), ev)

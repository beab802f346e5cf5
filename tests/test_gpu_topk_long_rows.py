"""GPU: top-k of many rows of more than 128 KB (bound from an eighth of the row, noted vectors) at its edges."""
import numpy as np
import pytest

from oracle import tallax_oracle as o
from tallax_b200 import tax
from tests.conftest import exact_match, to_dev, to_np

pytestmark = pytest.mark.gpu


# CTAs of 1024 threads (up to 148 rows), 512, 256 and 128; whole groups of eight pieces and one vector
# more, odd row starts, the longest row whose vectors have 16-bit numbers and one vector more; ties, NaNs, sorted rows,
# everything large in or outside the sampled pieces, the greatest elements many octaves apart
@pytest.mark.parametrize("dtype,rows,n,k", [
    ("f32", 64, 65536, 128), ("f32", 144, 32769, 5), ("f32", 16, 262144, 128), ("f32", 256, 262148, 50),
    ("bf16", 144, 65543, 100), ("f16", 112, 65541, 128),
    ("f32", 256, 32769, 128), ("f32", 288, 40964, 1), ("bf16", 160, 65537, 128), ("f16", 256, 65541, 128),
    ("f32", 400, 20484, 128), ("bf16", 304, 81920, 64), ("f16", 608, 49201, 20),
    ("f32", 608, 24584, 64), ("bf16", 1184, 41001, 64), ("f32", 608, 30001, 65),
    # the shortest rows that the long-row kernel does not number: the bound from a quarter of the row
    ("bf16", 304, 524296, 64), ("f16", 304, 524299, 128), ("f32", 304, 262149, 128)])
def test_long_row_top_k_sizes(cuda, dtype, rows, n, k):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((16, n)).astype(np.float32) * 2
    threads = 1024 if rows <= 148 else 512 if rows <= 296 else 128 if rows > 592 and k <= 64 else 256
    piece = np.arange(n) * (4 if dtype == "f32" else 2) // (16 * threads) % 8
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
    v, i = tax.top_k(to_dev(np.tile(x, (rows // 16, 1)), cuda), k, block_token=1)
    ev, ei = (np.tile(a, (rows // 16, 1)) for a in o.top_k(x, k))
    assert np.array_equal(to_np(i), ei)
    assert exact_match(to_np(v), ev)

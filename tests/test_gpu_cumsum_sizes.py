"""GPU: cumsum at the edges of its tiles, rings and clusters (odd row starts, one element over a tile, several turns)."""
import numpy as np
import pytest

from tallax_b200 import tax
from tests.conftest import to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,axis", [((5, 1021), 1), ((5, 1022), 1), ((3, 4095), 1), ((2, 4098), 1), ((7, 16385), 1), ((3, 70001), 1),
                                        ((400, 5003), 1), ((1, 1), 1), ((256, 33), 0), ((257, 31), 0), ((2049, 5), 0), ((5000, 70), 0),
                                        # a warp per row and just not; a thread per column and just not
                                        ((9, 125), 1), ((9, 126), 1), ((1, 7), 0), ((40, 129), 0), ((41, 129), 0), ((48, 8192), 0), ((49, 8192), 0),
                                        ((128, 65537), 0)])
@pytest.mark.parametrize("reverse", [False, True])
def test_cumsum_sizes(cuda, shape, axis, reverse):
    rng = np.random.default_rng(shape[1])
    x = rng.integers(-1000, 1000, shape).astype(np.int32)
    y = np.flip(np.cumsum(np.flip(x, axis), axis=axis, dtype=np.int32), axis) if reverse else np.cumsum(x, axis=axis, dtype=np.int32)
    assert np.array_equal(to_np(tax.cumsum(to_dev(x, cuda), axis, reverse=reverse)), y)
    # whole numbers, so that f32 sums are exact in any order
    f = (x % 8).astype(np.float32)
    g = np.flip(np.cumsum(np.flip(f, axis), axis=axis), axis) if reverse else np.cumsum(f, axis=axis)
    assert np.array_equal(to_np(tax.cumsum(to_dev(f, cuda), axis, reverse=reverse)), g)


# rows over clusters, a turn ahead and (too many of them) not: one turn, several, one that ends with a vector's first element; rows
# that begin at any element
@pytest.mark.parametrize("shape", [(1, 4097), (65, 33001), (66, 33001), (260, 9001), (261, 9001), (2, 131075), (3, 32765), (5, 65537)])
@pytest.mark.parametrize("reverse", [False, True])
def test_cumsum_over_clusters(cuda, shape, reverse):
    test_cumsum_sizes(cuda, shape, 1, reverse)


# rounding errors along columns.  A large first element and ones that round up every time they are added to it alone: a running sum is off by
# 0.4 units in the last place of the sum a row.  Sums of at most 16 rows, added up: their own additions, and those of their totals,
# lose at most half a unit each, 2^-24 of the sum
@pytest.mark.parametrize("rows,cols", [(9, 600), (40, 129), (41, 129), (48, 9000), (64, 33000), (128, 65537), (129, 65537)])
@pytest.mark.parametrize("reverse", [False, True])
def test_cumsum_of_few_rows_rounds_like_short_sums(cuda, rows, cols, reverse):
    x = np.full((rows, cols), 1.2 * 2.0 ** -24, np.float32)
    x[-1 if reverse else 0] = 1.0
    got = to_np(tax.cumsum(to_dev(x, cuda), 0, reverse=reverse)).astype(np.float64)
    want = np.cumsum(x[::-1] if reverse else x, axis=0, dtype=np.float64)
    want = want[::-1] if reverse else want
    assert np.abs(got - want).max() <= (16 + -(-rows // 8) + 1) * 2.0 ** -24 * want.max()

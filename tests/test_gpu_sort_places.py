"""GPU: the sort by estimated places, one row of every kind that its branches tell apart, at the edges of its kernels' sizes.

The expectation is numpy's stable argsort: sorting is exact, so there is no tolerance.
"""
import numpy as np
import pytest
import torch

from tallax_b200 import tax

pytestmark = pytest.mark.gpu


def _rows(n, rng):
    """Even keys; few values (the radix passes from the start); one value; a third of the row one value (more than its owner
    has room for); in order, and in reverse order; keys over the whole range of exponents; values that occur dozens and
    hundreds of times (large groups); every other element the same; a mask; two outliers that leave the rest one range."""
    z = rng.standard_normal(n).astype(np.float32)
    rare = np.clip(z, -4, 4) * np.float32(1e-6) + 1
    rare[0], rare[-1] = 3e38, -3e38
    return np.stack([z, np.round(z * 3), np.zeros(n, np.float32), np.where(rng.random(n) < 0.3, np.float32(np.inf), z),
                     np.sort(z), -np.sort(z), np.exp(np.clip(z, -4, 4) * 20).astype(np.float32),
                     rng.choice(z[:max(1, n // 40)], n), rng.choice(z[:max(1, n // 300)], n),
                     np.where(np.arange(n) % 2 == 0, np.float32(3), z),
                     np.where(np.arange(n) > n // 3, np.float32(-np.inf), z), rare])


# (copies of the rows, elements): four, eight and sixteen elements a thread, warps past the end; clusters of CTAs of 4096, 8192
# and 16384 elements; the rows that are too many for the shortest lengths
@pytest.mark.parametrize("copies,n", [(1, 65), (1, 1024), (50, 65), (50, 256), (50, 257), (1, 1025), (30, 1792), (30, 1793), (30, 2049),
                                      (1, 8192), (20, 8192), (1, 10000), (1, 10001), (15, 16384), (1, 16385), (6, 20000), (10, 24577),
                                      (4, 65536), (12, 65536), (1, 131071), (2, 131072)])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "i32"])
def test_sort_by_places(cuda, dtype, copies, n):
    rng = np.random.default_rng(n)
    x = _rows(n, rng)
    if dtype == "i32":
        x = (np.clip(x, -1e4, 1e4) * 2e5).astype(np.int32)      # (the outliers are the type's limits, nearly)
        t, a = torch.from_numpy(x), x.astype(np.int64)
    else:
        t = torch.from_numpy(x).to(torch.bfloat16 if dtype == "bf16" else torch.float32)
        a = t.float().numpy()
    for descending in (False, True):
        v, p = tax.sort([t.to(cuda).repeat(copies, 1)], num_keys=1, is_stable=True, return_argsort=True, descending=descending)
        e = np.argsort(-a if descending else a, axis=1, kind="stable")
        assert np.array_equal(p.cpu().numpy(), np.tile(e, (copies, 1)))
        assert torch.equal(v.cpu(), torch.take_along_dim(t, torch.from_numpy(e), 1).repeat(copies, 1))


# through a permutation, which a second key does
@pytest.mark.parametrize("n", [1000, 4097, 20000])
def test_sort_by_places_of_two_keys(cuda, n):
    rng = np.random.default_rng(n)
    first, x = rng.integers(0, 3, (12, n)).astype(np.int32), _rows(n, rng)
    out = tax.sort([torch.from_numpy(first).to(cuda), torch.from_numpy(x).to(cuda)], num_keys=2, is_stable=True, return_argsort=True)
    e = np.stack([np.lexsort((x[r], first[r])) for r in range(12)])
    assert np.array_equal(out[-1].cpu().numpy(), e)


# operands beside the first key, moved by the kernel that ends the sort: two and four bytes an element, further keys (whose -0
# and NaNs become canonical), rows of the network, of the places and of the tiles; and the kinds that are gathered afterwards
@pytest.mark.parametrize("n", [40, 1000, 4097, 20000, 131073])
@pytest.mark.parametrize("payloads", [("i32",), ("bf16",), ("i32", "bf16", "f32", "f16"), ("i64",), ("i32",) * 5])
@pytest.mark.parametrize("key", ["f32", "bf16", "i32"])
def test_operands_beside_the_first_key(cuda, n, payloads, key):
    types = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i32": torch.int32, "i64": torch.int64}
    gen = torch.Generator().manual_seed(n)
    first = torch.randint(0, 3, (3, n), generator=gen, dtype=torch.int32)
    second = torch.randn((3, n), generator=gen) * 100
    if key != "i32":
        second[:, ::5], second[:, 1::5], second[:, 2::9] = 0.0, -0.0, float("nan")
    second = second.to(types[key])
    rest = [torch.randint(0, 1000, (3, n), generator=gen).to(types[t]) for t in payloads]
    out = tax.sort([t.to(cuda) for t in (first, second, *rest)], num_keys=2, is_stable=True)
    v = second.float().numpy().astype(np.float64)
    v = np.where(np.isnan(v), np.inf, v)
    perm = torch.from_numpy(np.stack([np.lexsort((v[r], first[r].numpy())) for r in range(3)]))
    want = [torch.take_along_dim(t, perm, 1) for t in (first, second, *rest)]
    assert len(out) == len(want)
    for i, (g, e) in enumerate(zip(out, want)):
        g = g.cpu()
        assert g.dtype == e.dtype
        if i == 1 and key != "i32":
            assert torch.equal(g.isnan(), e.isnan()) and not torch.signbit(g[g == 0]).any()
            g, e = g.nan_to_num(nan=1e9), e.nan_to_num(nan=1e9)
        assert torch.equal(g, e)


# keys of both signs whose lower digits only tell the sign (the passes leave them out), with the values whose bits are not their
# key's: -0, NaNs of both signs, infinities; and rows of one sign
@pytest.mark.parametrize("n", [300, 4097, 16385, 65536])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
def test_keys_of_few_digits_and_both_signs(cuda, dtype, n):
    rng = np.random.default_rng(n)
    z = rng.standard_normal((5, n)).astype(np.float32)
    z[0], z[1], z[2], z[3] = np.round(z[0] * 3), np.round(z[1] * 3) - 20, np.abs(np.round(z[2] * 3)), z[3].astype(np.float16)
    z[4] = np.where(rng.random(n) < 0.5, np.float32(1.5), np.float32(-1.5))
    z[::2, ::11], z[::2, 1::11], z[::4, 2::50], z[::4, 3::50] = 0.0, -0.0, np.inf, -np.inf
    z[0, 4::50] = np.array([0x7FC00000, 0xFFC12300], np.uint32).view(np.float32)[rng.integers(0, 2, len(z[0, 4::50]))]
    t = torch.from_numpy(z).to({"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype])
    a = t.float().numpy()
    nan = np.isnan(a)
    a = np.where(nan, 0, a)
    for descending in (False, True):
        p = tax.sort([t.to(cuda)], num_keys=1, is_stable=True, return_argsort=True, descending=descending)[1]
        e = np.lexsort((-a, ~nan) if descending else (a, nan), axis=1)
        assert np.array_equal(p.cpu().numpy(), e)


# rows of few values.  Near each other, they are numbered and sorted in one pass: two values, as many as fit one digit and one more; the
# frequent one the least or the greatest; values that one CTA of a cluster sees and another does not, more in all than fit; as
# far apart as the numbering's table reaches and further.  Others are sorted less the least one and without their common bits
@pytest.mark.parametrize("copies,n", [(1, 300), (1, 1024), (50, 1500), (1, 4097), (3, 16385), (6, 20000), (1, 65536), (1, 131072)])
@pytest.mark.parametrize("dtype", ["f32", "bf16", "i32", "f16"])
@pytest.mark.parametrize("spacing", ["scattered", "near", "far"])
def test_rows_of_few_values(cuda, dtype, copies, n, spacing):
    rng = np.random.default_rng(n)
    types = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i32": torch.int32}
    at = np.arange(-300, 300) if spacing != "scattered" else np.unique(rng.integers(-2**31, 2**31, 600))
    if dtype == "i32":
        pool = (at * {"scattered": 1, "near": 6, "far": 7 << 20}[spacing]).astype(np.int32)
    elif spacing == "scattered":
        bits = np.arange(1, 30001, 100, dtype=np.int16)        # (positive, finite, and the same negative)
        pool = torch.from_numpy(bits).view(types[dtype]).float().numpy() if dtype != "f32" else rng.random(300).astype(np.float32)
        pool = np.unique(np.concatenate([pool, -pool]))
    else:
        pool = at.astype(np.float32) if spacing == "near" else np.sign(at) * 2.0 ** (np.abs(at) % 12) * (1 + np.abs(at) // 12 / 32)
        pool = np.unique(torch.from_numpy(pool).to(types[dtype]).float().numpy())
    rows = []
    for count in (2, 3, 50, 200, 255, 256, 257, 258, 500):
        for frequent in (0, -1):
            v = pool[np.sort(rng.permutation(len(pool))[:count])]
            v = pool[len(pool) // 2:][:count] if spacing == "near" and count < 256 else v
            row = np.where(rng.random(n) < 0.5, v[frequent], rng.choice(v, n))
            row[rng.permutation(n)[:min(n, len(v))]] = v[:n]     # each occurs
            rows.append(row)
    half = np.where(rng.random(n) < 0.6, pool[5], np.where(np.arange(n) < n // 2, rng.choice(pool[:150], n), rng.choice(pool[150:300], n)))
    rows += [half, np.where(np.arange(n) < n // 2, pool[7], rng.choice(pool, n)), np.where(np.arange(n) % 2 == 0, pool[3], pool[4])]
    a = np.stack(rows)
    t, a = torch.from_numpy(a).to(types[dtype]), a.astype(np.float64)
    for descending in (False, True):
        v, p = tax.sort([t.to(cuda).repeat(copies, 1)], num_keys=1, is_stable=True, return_argsort=True, descending=descending)
        e = np.argsort(-a if descending else a, axis=1, kind="stable")
        assert np.array_equal(p.cpu().numpy(), np.tile(e, (copies, 1)))
        assert torch.equal(v.cpu(), torch.take_along_dim(t, torch.from_numpy(e), 1).repeat(copies, 1))

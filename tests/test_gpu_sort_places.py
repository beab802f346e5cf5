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


# ---- rows that get past the sample of equal keys: what the kernel decides later -------------------------------------------------
def _cluster(rows, n):
    """CTAs a row, as the dispatch chooses them; elements a thread; threads a CTA."""
    ctas, at_once = (lambda tile: -(-n // tile)), (lambda c, an_sm: 148 * an_sm if c == 1 else 8 * (18 * an_sm // c))
    least, half = ctas(16384), ctas(8192)
    c = 1
    if n > 10000:
        c = next((c for c in range(min(ctas(4096), 8), least - 1, -1) if rows <= at_once(c, 1)), 0)
        if c == 0:
            c = (1 if least == 1 else half if half <= 8 and rows <= at_once(half, 2) else (3 if half == 3 else 2) if least == 2
                 else half if half <= 6 else max(least, 4))
    if c > 1 or n > 8192:
        ipt = 16
    else:
        ipt = 4 if n <= 1024 else 8 if n <= 2048 or rows * ((n + 255) // 256 * 32) <= 148 * 1024 else 16
    return c, ipt, max(256, -(-n // (c * 32 * ipt)) * 32)


def _way(row, dtype, rows, descending):
    """The way that a row takes, from the rules of the kernel: by digits from the start; by digits because an owner has no room; or, per
    CTA, by places or by digits of its own elements."""
    n, half = len(row), dtype == "bf16"
    c, ipt, nt = _cluster(rows, n)
    pos = np.arange(n, dtype=np.int64)
    if dtype == "i32":
        key = row.astype(np.int64) + 2**31
    else:
        bits = (row if dtype == "f32" else torch.from_numpy(row).to(torch.bfloat16).float().numpy()).view(np.uint32).astype(np.int64)
        key = np.where(bits >> 31 == 1, bits ^ 0xFFFFFFFF, bits | 0x80000000)
    if descending:
        key = key ^ 0xFFFFFFFF
    if half:
        key = (key & 0xFFFF0000) | ((pos << 15) * (2 * (0xFFFFFFFF // n)) >> 32)
    upright = key if dtype == "i32" else np.where(key >> 31 == 1, key, key ^ 0x7FFFFFFF)
    diff = int(np.bitwise_or.reduce(upright ^ upright[0])) & (0xFFFF0000 if half else 0xFFFFFFFF)
    digits = sum((diff >> s & 255) != 0 for s in (0, 8, 16, 24))
    equal = 0
    for start in range(0, n, 32 * ipt):
        _, count = np.unique(key[start:start + 32] >> (16 if half else 0), return_counts=True)
        equal += int((count * (count - 1)).sum())
    if digits <= (1 if half else 2) or equal > (n // (2 * ipt) if half else 24 * 31 // ipt):
        return ["digits"]
    o = key - key.min()
    sh = max(int(o.max()).bit_length() - 11, 0)
    count = np.bincount(o >> sh, minlength=2049)
    before = np.concatenate([[0], np.cumsum(count)])
    at = before[o >> sh] + (((o << 1 & 0xFFFFFFFF) << (31 - sh) & 0xFFFFFFFF) * count[o >> sh] >> 32)
    per = -(-n // c)
    got = np.bincount(at // per, minlength=c)
    if c > 1 and (got > nt * (ipt + ipt // 16)).any():
        return ["no room"]
    ways = []
    for d in range(c):
        group = np.bincount(at[at // per == d])
        ways.append("own digits" if group.max(initial=0) > 512 or (np.minimum(group, 512)**2).sum() > 24 * got[d] else "places")
    return ways


def _crowded(n, dtype, rng):
    """Clumps of 40, of 480 and of 1500 elements next to each other in value, evenly spread; clumps in a part of the values only; one dense
    run, and nine tenths of the row a run.  Distinct keys; in bf16, of which there are not enough, equal ones side by side where the
    sample does not look."""
    rows, quiet = [], np.arange(n) % 128 >= 32
    for clump, share in ((40, 1.0), (480, 1.0), (1500, 1.0), (300, 0.5), (0, 1.0), (0, 0.9)):
        if dtype == "bf16":
            z, at = rng.standard_normal(n).astype(np.float32), np.arange(n) // max(clump, 1)
            v = rng.permutation(np.linspace(-9, 9, n // max(clump, 1) + 1).astype(np.float32))[at]
            rows.append(np.where(quiet & (np.arange(n) < n * share), v if clump else np.float32(0.5), z))
            continue
        most, m = 0x7F000000, int(n * share)
        k = 12345 + np.arange(m)
        if clump:
            k = (np.linspace(-most, most * (2 * share - 1) - 2 * clump, -(-m // clump)).astype(np.int64)[:, None] + np.arange(clump)).ravel()[:m]
        k = np.unique(np.concatenate([k[:n - 2], [-most, most]]))
        others = np.setdiff1d(rng.integers(-most, most, 2 * n), k)
        k = rng.permutation(np.concatenate([k, rng.permutation(others)[:n - len(k)]])).astype(np.int32)
        rows.append(k if dtype == "i32" else np.where(k < 0, -k | -2**31, k).astype(np.int32).view(np.float32))
    return rows


# a CTA, and clusters of two to eight; rows of which some CTAs' groups are large, on their own (the CTA's elements by digits), and rows
# of which one owner would get more than it has room for; through a permutation too, and with a payload
CROWDED = [(1, 700, 1), (1, 1500, 1), (1, 4097, 1), (80, 4097, 1), (11, 12000, 2), (1, 12000, 3), (1, 16384, 4), (1, 20000, 5),
           (1, 24000, 6), (1, 28001, 7), (1, 32768, 8), (1, 131072, 8)]


@pytest.mark.parametrize("copies,n,cluster", CROWDED)
@pytest.mark.parametrize("dtype", ["f32", "bf16", "i32"])
def test_crowded_keys(cuda, dtype, copies, n, cluster):
    rng = np.random.default_rng(n)
    a = np.stack(_crowded(n, dtype, rng))
    assert _cluster(copies * len(a), n)[0] == cluster
    t = torch.from_numpy(a).to(torch.bfloat16) if dtype == "bf16" else torch.from_numpy(a)
    a = t.float().numpy() if dtype == "bf16" else a.astype(np.float64)
    for descending in (False, True):
        ways = [_way(r, dtype, copies * len(a), descending) for r in (t.float() if dtype == "bf16" else t).numpy()]
        assert ["digits"] not in ways
        assert any("own digits" in w for w in ways) and (cluster == 1 or ["no room"] in ways), ways
        e = torch.from_numpy(np.argsort(-a if descending else a, axis=1, kind="stable"))
        v, p = tax.sort([t.to(cuda).repeat(copies, 1)], num_keys=1, is_stable=True, return_argsort=True, descending=descending)
        assert torch.equal(p.cpu().long(), e.repeat(copies, 1))
        assert torch.equal(v.cpu(), torch.take_along_dim(t, e, 1).repeat(copies, 1))
        # the second key brings the first one's row into this order before its pass
        second = torch.from_numpy(np.stack([rng.permutation(n) for _ in range(len(a))]).astype(np.int32))
        at = (n - 1 - second if descending else second).long()
        first, payload = torch.take_along_dim(t, at, 1), torch.randint(0, 1 << 30, t.shape, dtype=torch.int32)
        got = tax.sort([x.to(cuda).repeat(copies, 1) for x in (first, second, payload)], num_keys=2, is_stable=True, descending=descending)
        order = torch.empty_like(at).scatter_(1, at, torch.arange(n).repeat(len(a), 1))   # where the second key puts which element
        for g, x in zip(got, (first, second, payload)):
            assert torch.equal(g.cpu(), torch.take_along_dim(torch.take_along_dim(x, order, 1), e, 1).repeat(copies, 1))

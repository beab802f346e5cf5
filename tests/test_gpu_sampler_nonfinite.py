"""GPU: rows with NaNs and infinities get a token that exists, in every sampler.

An infinite logit has an infinite score and wins.  A row in which nothing has a score (its threshold, temperature or noise is a
NaN) gets the token of its greatest candidate, a NaN being greater than everything.
"""
import numpy as np
import pytest
import torch

from tallax_b200._src import ops

pytestmark = pytest.mark.gpu

KINDS = ["nan", "nans", "inf", "infs", "nan and inf", "masked", "all nan", "minus inf", "nan temperature", "nan noise", "plain"]


def _inputs(rows, vocab, dtype, seed):
    """Row r is of kind r % len(KINDS)."""
    g = torch.Generator().manual_seed(seed)
    x, noise = torch.randn((rows, vocab), generator=g), torch.rand((rows, vocab), generator=g)
    temperature = torch.rand(rows, generator=g) + 0.5
    nan, inf = float("nan"), float("inf")
    for r in range(rows):
        at = torch.randperm(vocab, generator=g)[:5]
        kind = KINDS[r % len(KINDS)]
        if kind == "nan":
            x[r, at[0]] = nan
        elif kind == "nans":
            x[r, at] = nan
        elif kind == "inf":
            x[r, at[0]] = inf
        elif kind == "infs":
            x[r, at] = inf
        elif kind == "nan and inf":
            x[r, at[0]], x[r, at[1]] = nan, inf
        elif kind == "masked":
            x[r] = -inf
        elif kind == "all nan":
            x[r] = nan
        elif kind == "minus inf":
            x[r, at] = -inf
        elif kind == "nan temperature":
            temperature[r] = nan
        elif kind == "nan noise":
            noise[r] = nan
    return x.to(dtype), noise, torch.rand(rows, generator=g) * 0.5 + 0.5, temperature


def _check(tokens, x, k):
    """tokens, x on the CPU; k: the rows' top-k, 0 for none.  Every token is one of the row's top-k set."""
    order = torch.sort(torch.where(x.isnan(), torch.full_like(x, float("inf")), x).float() + 0.0, dim=1, descending=True, stable=True)
    for r in range(x.shape[0]):
        kind, t = KINDS[r % len(KINDS)], int(tokens[r])
        assert 0 <= t < x.shape[1], (r, kind, t)
        if kind in ("inf", "infs"):
            assert x[r, t] == float("inf"), (r, kind, t)
        elif kind == "masked" and k[r] > 0:
            assert t < k[r], (r, kind, t)
        elif kind in ("nan", "nans", "all nan") and k[r] > 0:
            assert bool((order.indices[r, :k[r]] == t).any()), (r, kind, t)
        elif kind in ("minus inf", "plain"):
            assert x[r, t] > -float("inf"), (r, kind, t)


# both merges, every tail: one warp (up to 128 candidates kept), a block
@pytest.mark.parametrize("k", [1, 2, 50, 128, 200, 300])
@pytest.mark.parametrize("world", [1, 3])
def test_merge_of_vocabulary_shards(cuda, world, k):
    rows, vl, k_cand = 33, 2048, 128 if world > 1 else 300
    x, noise, top_p, temperature = _inputs(rows, vl * world, torch.bfloat16, k)
    tk = torch.full((rows,), k, dtype=torch.int32)
    args = [t.cuda() for t in (tk, top_p, temperature)]
    xs = [x[:, r * vl:(r + 1) * vl].contiguous().cuda() for r in range(world)]
    ns = [noise[:, r * vl:(r + 1) * vl].contiguous().cuda() for r in range(world)]
    blocks = torch.stack([ops.shard_candidates(xs[r], r * vl, k_cand, noise_shard=ns[r], vocab_total=vl * world) for r in range(world)])
    tokens = ops.merge_and_sample(blocks, *args).cpu()
    _check(tokens, x, [k] * rows)
    # what has no score: the greatest candidate, of equal ones the lowest token
    first = torch.where(x.isnan(), torch.full_like(x, 4.0), torch.where(x == float("inf"), torch.full_like(x, 3.9), x)).float()
    first = torch.sort(first, dim=1, descending=True, stable=True).indices[:, 0]
    for r in range(rows):
        if KINDS[r % len(KINDS)] in ("nan", "nans", "nan and inf", "all nan"):
            assert torch.isnan(x[r, int(tokens[r])]) and int(tokens[r]) == int(torch.isnan(x[r]).nonzero()[0]), r
    group = ops.Exchange.local_group(rows, k_cand, world, xs[0].device)
    try:
        for r in range(world):
            ops.exchange_shard_candidates(xs[r], r * vl, group[r], noise_shard=ns[r], vocab_total=vl * world)
        for r in range(world):
            assert torch.equal(ops.exchange_merge_and_sample(group[r], *args).cpu(), tokens)
    finally:
        for e in group:
            e.close()


# the cluster form, and the streaming one (more than 16 MB) with its classes of rows: normal, without top-k, everything else
@pytest.mark.parametrize("rows,vocab", [(55, 3000), (55, 40008), (550, 16384)])
@pytest.mark.parametrize("noise_kind", ["tensor", "rows at odd addresses", "key"])
def test_fused_sampler(cuda, rows, vocab, noise_kind):
    x, noise, top_p, temperature = _inputs(rows, vocab, torch.bfloat16, vocab)
    k = torch.tensor([0, 1, 2, 50, 700])[torch.arange(rows) // len(KINDS) % 5].to(torch.int32)
    if noise_kind == "rows at odd addresses":
        kw = dict(noise=torch.cat([noise, noise[:, :1]], 1).cuda())
    else:
        kw = dict(noise=noise.cuda()) if noise_kind == "tensor" else dict(rng_key=(3, 4))
    for p in (top_p, torch.ones(rows)):
        tokens = ops.sample(x.cuda(), k.cuda(), p.cuda(), temperature.cuda(), **kw).cpu()
        _check(tokens, x, k.tolist())


def test_candidate_sampler_and_gumbel_argmax(cuda):
    rows, k, vocab = 44, 96, 5000
    x, noise, top_p, temperature = _inputs(rows, vocab, torch.float32, 1)
    values, index = torch.sort(torch.where(x.isnan(), torch.full_like(x, float("inf")), x), dim=1, descending=True, stable=True)
    index = index[:, :k].contiguous()
    values = x.gather(1, index)
    tokens = ops.top_p_and_sample(values.cuda(), index.int().cuda(), top_p.cuda(), temperature.cuda(), vocab_size=vocab,
                                  replace_val=-1e12, noise=noise.cuda()).cpu()
    for r in range(rows):
        assert bool((index[r] == int(tokens[r])).any()), r
    lines = x[:, :k].contiguous()
    i0, i1 = (torch.arange(n, dtype=torch.int32) for n in lines.shape)
    i0, i1 = i0[:, None].expand(rows, k).contiguous(), i1[None].expand(rows, k).contiguous()
    got0, got1 = (t.cpu() for t in ops.gumbel_argmax((1, 2), lines.cuda(), i0.cuda(), i1.cuda(), k, 1))
    assert torch.equal(got0, torch.arange(rows, dtype=torch.int32))
    assert bool(((got1 >= 0) & (got1 < k)).all())

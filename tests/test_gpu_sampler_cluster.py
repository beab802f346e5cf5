"""GPU: the sampler's cluster kernel (a row resident in a cluster's shared memory) at the sizes where its parts, its lists
and its bound can go wrong, against the oracle."""
import numpy as np
import pytest

from oracle import tallax_oracle as o
from tallax_b200._src import ops
from tests.conftest import to_dev, to_np

pytestmark = pytest.mark.gpu


# one element; a vector and a remainder; all elements candidates (<= 2048) and just not; parts that end inside a vector;
# odd row starts; two, eight and sixteen CTAs; longer than a cluster holds
@pytest.mark.parametrize("V", [1, 2, 129, 2048, 2049, 8191, 40961, 131072, 327681, 800001])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("from_key", [False, True])
def test_cluster_sampler_sizes(cuda, dtype, V, from_key):
    B = 8 if V < 300000 else 4
    x, tk, tp, T, noise = o.make_sampling_inputs(B=B, V=max(V, 64), seed=V, dtype=dtype)
    x, noise = np.ascontiguousarray(x[:, :V]), np.ascontiguousarray(noise[:, :V])
    xf = x.astype(np.float32)
    tk[:] = ([1024, 0, 50, 257, 0, 1, 0, 1500])[:B]
    T[B - 3] = 0.0                                             # greedy
    if B == 8:
        xf[1] = 0.25 * (np.arange(V) % 3)                      # three values: far more survivors than the lists hold
        xf[2] = np.round(xf[2])                                # ties at the k-th value
        xf[3, V // 2:] = -np.inf                               # masked half
        xf[4] *= 0.01                                          # flat
        xf[6] = -np.inf
        xf[6, V // 3] = -3.0                                   # a single token left
        xf[7] = np.sort(xf[7])                                 # the set sits in one CTA's part
    x = xf.astype(x.dtype)
    key = (17, V)
    kw = dict(rng_key=key) if from_key else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = dict(rng_key=key) if from_key else dict(noise=to_dev(noise, cuda))
    tok, status = ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), return_status=True, **dkw)
    bad = (to_np(tok) != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), to_np(tok)[bad], exp[bad])
    assert (to_np(status) & 2 == 0).all()


# 1024 < top_k < vocab: the row is cut to its top-k set in the parts.  The smallest and the largest such k; one, two, eight and
# sixteen parts; parts that end inside a vector; ties at the k-th key that lie in one part, in several and in all of them
@pytest.mark.parametrize("V", [1026, 2049, 6000, 40961, 131072, 200003])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("from_key", [False, True])
def test_large_top_k_sizes(cuda, dtype, V, from_key):
    B = 10
    x, tk, tp, T, noise = o.make_sampling_inputs(B=B, V=V, seed=V, dtype=dtype)
    xf = x.astype(np.float32)
    tk[:] = [1025, V - 1, 1 + V // 2, 1025, 1025, V - 1, 1 + V // 2, 1025, 1 + V // 2, 1025]
    tk[:] = np.clip(tk, 1025, V - 1)
    xf[2] = np.round(xf[2])
    xf[3] = np.round(xf[3])
    xf[4] = 0.25 * (np.arange(V) % 2)                          # two values: the ties spread over all parts
    xf[5] = -1.0                                               # one value: all but the last column
    xf[6, V // 3:] = -np.inf                                   # fewer finite values than k
    xf[7] = np.sort(xf[7])                                     # the set sits in the last part
    xf[8] = 1.0 + 1e-3 * xf[8]                                 # (nearly) one bin of the first histogram
    xf[9, :1500] = 7.0                                         # the ties sit in the first part
    x = xf.astype(x.dtype)
    kw = dict(rng_key=(23, V)) if from_key else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = dict(rng_key=(23, V)) if from_key else dict(noise=to_dev(noise, cuda))
    tok, status = ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), return_status=True, **dkw)
    bad = (to_np(tok) != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), to_np(tok)[bad], exp[bad])
    assert (to_np(status) & 3 == 1).all()
    assert (to_np(status)[[0, 1, 2]] == 1).all()               # decided from the parts


# A call that needs a workspace for the form it would take has it reported: more scratch than that changes nothing.  Sizes
# around 16 MB of logits, the rule's line, and below it
@pytest.mark.parametrize("rows,V", [(33, 128256), (40, 128256), (48, 151936), (65, 128256), (66, 128256), (120, 128256)])
@pytest.mark.parametrize("from_key", [False, True])
def test_workspace_reported_is_the_workspace_used(cuda, rows, V, from_key):
    import torch

    from tallax_b200 import _lib
    lib = _lib.load()
    gen = torch.Generator(device=cuda).manual_seed(rows)
    x = (torch.randn((rows, V), generator=gen, device=cuda) * 3).to(torch.bfloat16)
    tk = torch.full((rows,), 50, dtype=torch.int32, device=cuda)
    tp, T = torch.full((rows,), 0.9, device=cuda), torch.full((rows,), 0.8, device=cuda)
    kw = dict(rng_key=(1, 2)) if from_key else dict(noise=torch.rand((rows, V), generator=gen, device=cuda))
    reported = lib.tlx_sample_workspace_bytes(rows, V)
    large = ops.SampleWorkspace(rows, V, cuda)
    large.ws = torch.empty(64 << 20, dtype=torch.uint8, device=cuda)
    launches, tokens = [], []
    for w in (None, ops.SampleWorkspace(rows, V, cuda), large):
        before = lib.tlx_kernel_launches()
        tokens.append(ops.sample(x, tk, tp, T, workspace=w, **kw).clone())
        launches.append(lib.tlx_kernel_launches() - before)
    assert launches == [3 if reported > 256 else 1] * 3
    assert torch.equal(tokens[0], tokens[1]) and torch.equal(tokens[0], tokens[2])


# rows with top-k whose candidates are hundreds of ties (cut by column) or more than the lists hold (cut in the parts)
@pytest.mark.parametrize("V", [300, 1509, 2048, 2049, 12032, 80129])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("from_key", [False, True])
def test_heavy_ties_and_masked_rows(cuda, dtype, V, from_key):
    B = 12
    x, tk, tp, T, noise = o.make_sampling_inputs(B=B, V=V, seed=V + 1, dtype=dtype)
    xf = x.astype(np.float32)
    tk[:] = np.minimum([50, 257, 1024, 50, 700, 1, 1024, 50, 1000, 3, 1024, 257], V - 1)
    xf[:3] = 0.0                                               # one value
    xf[3] = 0.5 * (np.arange(V) % 2)                           # two values, the cut inside the greater one's ties
    xf[4] = np.where(np.arange(V) % 100 < 3, 1.0, 0.25 * (np.arange(V) % 3))
    xf[5] = 2.0                                                # greedy: the first column of all
    T[5] = 0.0
    xf[6:9, V // 20:] = -np.inf                                # 95 % masked, together
    xf[9] = np.round(xf[9] / 4)
    xf[10, ::2] = -np.inf                                      # half masked, scattered
    xf[11] = -7.0
    x = xf.astype(x.dtype)
    kw = dict(rng_key=(29, V)) if from_key else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = dict(rng_key=(29, V)) if from_key else dict(noise=to_dev(noise, cuda))
    tok, status = ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), return_status=True, **dkw)
    bad = (to_np(tok) != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), to_np(tok)[bad], exp[bad])
    assert (to_np(status) & 2 == 0).all()


# flat rows without top-k: hundreds of elements of a part lie above the best-scored published one; the parts settle them all
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("from_key", [False, True])
def test_flat_rows_without_top_k(cuda, dtype, from_key):
    B, V = 32, 40001
    x, tk, tp, T, noise = o.make_sampling_inputs(B=B, V=V, seed=3, dtype=dtype)
    x = (x.astype(np.float32) * np.repeat(np.float32([0.1, 0.03, 0.01, 0.003]), B // 4)[:, None]).astype(x.dtype)
    tk[:] = 0
    kw = dict(rng_key=(31, 7)) if from_key else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = dict(rng_key=(31, 7)) if from_key else dict(noise=to_dev(noise, cuda))
    tok, status = ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), return_status=True, **dkw)
    bad = (to_np(tok) != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), to_np(tok)[bad], exp[bad])
    assert (to_np(status) & 6 == 0).all()                      # none was answered by passes over global memory


# rows without top-k whose values top-p bounds first: parts just long enough and just not, parts that end inside a vector, two
# to sixteen CTAs; top_p from the least to what rules nothing out; what that way leaves to the other one: a constant row, equal
# scores (constant noise), NaN, infinities; a threshold deep in the tail, several rounds (hot rows), a row in order
@pytest.mark.parametrize("V", [8192, 23999, 24001, 50257, 96001, 131072])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("noise_kind", ["key", "tensor", "constant"])
def test_rows_bounded_by_top_p(cuda, dtype, V, noise_kind):
    B = 16
    x, tk, tp, T, noise = o.make_sampling_inputs(B=B, V=V, seed=V + 3, dtype=dtype)
    xf = x.astype(np.float32)
    tk[:] = 0
    tp[:] = [0.0, 0.3, 0.6, 0.9, 0.95, 0.99, 0.9995, 0.99995, 1.0, 0.8, 0.8, 0.8, 0.8, 0.7, 0.9, 0.5]
    T[:] = np.linspace(0.4, 1.6, B)
    xf[9] = 0.5                                                # one value
    xf[10] = np.round(xf[10])                                  # many equal values at the threshold
    xf[11, V // 7:] = -np.inf                                  # masked
    xf[12] *= 0.01                                             # flat: everything is scored
    xf[13] = np.sort(xf[13])                                   # the kept ones sit in one part
    xf[14] = np.where(np.arange(V) % 2 == 0, xf[14], xf[14] - 30)
    T[15], tp[15] = 20.0, 0.2                                  # hot: the best score lies below the threshold, again and again
    x = xf.astype(x.dtype)
    if noise_kind == "constant":
        noise = np.full_like(noise, 0.5)
    kw = dict(rng_key=(41, V)) if noise_kind == "key" else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = dict(rng_key=(41, V)) if noise_kind == "key" else dict(noise=to_dev(noise, cuda))
    tok, status = ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), return_status=True, **dkw)
    bad = (to_np(tok) != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), to_np(tok)[bad], exp[bad])
    assert (to_np(status) & 2 == 0).all()
    # rows with NaNs and infinities are left to passes over the row in global memory.  A NaN has no score and makes every mass one, so that
    # top-p rules nothing out: the row's token is that of the others at top_p 1.  An infinite logit wins, the first token of a masked row does,
    # and one -inf is an element like others
    xf[:4] = xf[13:14]
    xf[0, 5], xf[1, V - 1], xf[2, 7], xf[3] = np.nan, np.inf, -np.inf, -np.inf
    x = xf[:4].astype(x.dtype)
    dkw = dict(rng_key=(41, V)) if noise_kind == "key" else dict(noise=to_dev(noise[:4], cuda))
    tok = to_np(ops.sample(to_dev(x, cuda), to_dev(tk[:4], cuda), to_dev(tp[:4], cuda), to_dev(T[:4], cuda), **dkw))
    xf[0, 5], tp[0] = -np.inf, 1.0
    x = xf[:4].astype(x.dtype)
    for r in (0, 2):
        kw = dict(noise=noise[r:r + 1]) if noise_kind != "key" else dict(rng_key=(41, V), dim0_offset=r)
        exp, flags = o.sample(x[r:r + 1], tk[r:r + 1], tp[r:r + 1], T[r:r + 1], return_flags=True, **kw)
        assert flags[0] or tok[r] == exp[0], r
    assert tok[1] == V - 1 and tok[3] == 0


# f32 rows next to the type's least value (masked with it, and not all equal): what top-p bounds them by stays finite, so that nothing
# outside the part, which holds -inf, is taken for an element; rows at every offset from a 16-byte boundary
@pytest.mark.parametrize("V", [50257, 96003, 131070])
@pytest.mark.parametrize("from_key", [False, True])
def test_rows_next_to_the_least_value(cuda, V, from_key):
    B = 16
    rng = np.random.default_rng(V)
    least = np.finfo(np.float32).max * np.float32(-1)
    x = least * (1 - rng.integers(0, 64, (B, V)).astype(np.float32) * np.float32(2**-24)).astype(np.float32)
    x[::2, V // 3] = least * np.float32(1 - 70 * 2.0**-24)     # the greatest once
    x[5] = np.where(np.arange(V) == V - 1, np.float32(-1e38), least)
    tk, tp = np.zeros(B, np.int32), np.linspace(0.05, 0.99, B).astype(np.float32)
    T = np.linspace(1.0, 2.0, B).astype(np.float32)            # (from 1 on: every score is finite)
    noise = rng.random((B, V), dtype=np.float32)
    kw = dict(rng_key=(43, V)) if from_key else dict(noise=noise)
    exp, flags = o.sample(x, tk, tp, T, return_flags=True, **kw)
    dkw = kw if from_key else dict(noise=to_dev(noise, cuda))
    tok = to_np(ops.sample(to_dev(x, cuda), to_dev(tk, cuda), to_dev(tp, cuda), to_dev(T, cuda), **dkw))
    bad = (tok != exp) & ~flags
    assert not bad.any(), (np.flatnonzero(bad), tok[bad], exp[bad])

"""GPU: calls launched as programmatic dependents keep the stream's order, whatever precedes them, eager and in a graph.

Every call reads what the operation before it on the stream has just written, over buffers that are used again at once: values,
parameters, noise, keys, indices and permutations.  The expectation is the same call made after a synchronisation.
"""
import pytest
import torch

from tallax_b200 import sampling, tax, tumpy
from tallax_b200._src import ops

pytestmark = pytest.mark.gpu

ROWS, N = 24, 40000


def _calls(index, metadata, shape):
    return {
        "sample": lambda x: sampling.sample((3, 5), x, metadata),
        "top_k": lambda x: tax.top_k(x, 20, block_token=1)[0],
        "sort": lambda x: tax.sort([x], num_keys=1)[0],
        "short_sort": lambda x: tax.sort([x[:, :40].contiguous()], num_keys=1)[0],
        "gather": lambda x: tumpy.take_along_axis(x, index, 1),
        "gather_rows": lambda x: tumpy.take_along_axis(x, index % ROWS, 0) if shape == index.shape else x,
        "cumsum": lambda x: tax.cumsum(x, 1),
        "cumsum_rows": lambda x: tax.cumsum(x, 0),
    }


def _setup(cuda):
    gen = torch.Generator(device=cuda).manual_seed(11)
    source = [torch.randn((ROWS, N), generator=gen, device=cuda) for _ in range(3)]
    index = torch.randint(0, N, (ROWS, N), generator=gen, device=cuda, dtype=torch.int32)
    metadata = sampling.SamplingMetadata(torch.full((ROWS,), 50, dtype=torch.int32, device=cuda), torch.full((ROWS,), 0.9, device=cuda),
                                         torch.ones(ROWS, device=cuda))
    return source, _calls(index, metadata, (ROWS, N))


# what writes the input just before: an elementwise kernel, a copy, a fill and a copy, another of these calls
def _write(x, source, how, calls):
    if how == "kernel":
        torch.add(source, 1.0, out=x)
    elif how == "copy":
        x.copy_(source)
    elif how == "fill":
        x.zero_()
        x[:, ::3].copy_(source[:, ::3])
    else:
        x.copy_(calls["cumsum"](calls["sort"](source)))


@pytest.mark.parametrize("how", ["kernel", "copy", "fill", "call"])
@pytest.mark.parametrize("name", ["sample", "top_k", "sort", "short_sort", "gather", "gather_rows", "cumsum", "cumsum_rows"])
def test_calls_wait_for_what_precedes_them(cuda, name, how):
    source, calls = _setup(cuda)
    x = torch.empty((ROWS, N), device=cuda)
    want = []
    for s in source:
        _write(x, s, how, calls)
        torch.cuda.synchronize()
        want.append(calls[name](x).clone())
        torch.cuda.synchronize()
    got = []
    for _ in range(3):
        for s in source:                      # no synchronisation: the next write overwrites what the call before it reads
            _write(x, s, how, calls)
            got.append(calls[name](x))
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert torch.equal(g, want[i % 3])


@pytest.mark.parametrize("how", ["kernel", "copy", "fill", "call"])
def test_captured_calls_wait_for_what_precedes_them(cuda, how):
    source, calls = _setup(cuda)
    x, s = torch.empty((ROWS, N), device=cuda), torch.empty((ROWS, N), device=cuda)
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    want = []
    for src in source:
        _write(x, src, how, calls)
        want.append([calls[c](x).clone() for c in ("top_k", "sort", "cumsum", "sample")])
    torch.cuda.synchronize()
    s.copy_(source[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        for _ in range(2):
            _write(x, s, how, calls)
            [calls[c](x) for c in ("top_k", "sort", "cumsum", "sample")]
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            _write(x, s, how, calls)
            first = calls["top_k"](x)
            other.wait_stream(side)            # a fork and a join: two predecessors of the calls after it
            with torch.cuda.stream(other):
                second = calls["sort"](x)
            third = calls["cumsum"](x)
            side.wait_stream(other)
            fourth = calls["sample"](x)
    for _ in range(2):
        for src, w in zip(source, want):
            s.copy_(src)
            graph.replay()
            torch.cuda.synchronize()
            for g, e in zip((first, second, third, fourth), w):
                assert torch.equal(g, e)


def test_steps_follow_each_other(cuda):
    """A large sampler call (three kernels), a call of one kernel on the same buffers, and again, as a decode loop queues them."""
    gen = torch.Generator(device=cuda).manual_seed(2)
    rows, vocab = 160, 65536
    logits = [(torch.randn((rows, vocab), generator=gen, device=cuda) * 3).bfloat16() for _ in range(2)]
    k = torch.randint(0, 300, (rows,), generator=gen, device=cuda, dtype=torch.int32)
    md = sampling.SamplingMetadata(k, torch.full((rows,), 0.9, device=cuda), torch.ones(rows, device=cuda))
    want = []
    for x in logits:
        t = sampling.sample((1, 9), x, md)
        torch.cuda.synchronize()
        want.append((t, tax.top_k(x, 8, block_token=1)[1]))
        torch.cuda.synchronize()
    got, x = [], torch.empty_like(logits[0])
    for i in range(12):
        x.copy_(logits[i % 2])
        got.append((sampling.sample((1, 9), x, md), tax.top_k(x, 8, block_token=1)[1]))
    torch.cuda.synchronize()
    for i, (t, v) in enumerate(got):
        assert torch.equal(t, want[i % 2][0]) and torch.equal(v, want[i % 2][1])


def _versions(cuda, rows, n, dtype, vocab=None):
    """Three sets of everything that a call reads."""
    gen = torch.Generator(device=cuda).manual_seed(rows)
    sets = []
    for i in range(3):
        k = torch.randint(1, 40, (rows,), generator=gen, device=cuda, dtype=torch.int32)
        k[i::5] = 0 if vocab is None else 7
        sets.append(dict(x=(torch.randn((rows, n), generator=gen, device=cuda) * 2).to(dtype), noise=torch.rand((rows, n), generator=gen, device=cuda),
                         top_k=k, top_p=torch.rand(rows, generator=gen, device=cuda) * 0.6 + 0.4,
                         temperature=(torch.rand(rows, generator=gen, device=cuda) + 0.5) * (torch.arange(rows, device=cuda) % 7 != i),
                         index=torch.randint(0, n, (rows, n), generator=gen, device=cuda, dtype=torch.int32),
                         perm=torch.argsort(torch.rand((rows, n), generator=gen, device=cuda), dim=1).int(),
                         key=torch.randint(0, 1 << 30, (2,), generator=gen, device=cuda, dtype=torch.int32),
                         offset=torch.tensor(3 * i, device=cuda, dtype=torch.int32)))
    return sets


# everything that a call reads is overwritten right before it, by kernels, the operand `last` at the very end; both forms of the sampler
# (the streaming one lists its rows by their parameters before it waits), both kinds of noise, and the pair of the vocabulary shards
READS = {"sample": "x noise top_k top_p temperature", "sample_key": "x key offset top_k top_p temperature", "gather": "x index",
         "sort_through": "x perm", "shard": "x noise top_k top_p temperature"}
READS["stream"], READS["stream_key"] = READS["sample"], READS["sample_key"]


@pytest.mark.parametrize("name,last", [(name, last) for name, reads in READS.items() for last in reads.split()])
def test_every_operand_may_change_between_queued_calls(cuda, name, last):
    names = READS[name].split()
    rows, n = (160, 65536) if name.startswith("stream") else (300, 4096) if name == "shard" else (24, 20000)
    sets = _versions(cuda, rows, n, torch.float32 if name in ("gather", "sort_through") else torch.bfloat16, n if name == "shard" else None)
    now = {k: torch.empty_like(v) for k, v in sets[0].items()}
    ex = ops.Exchange.local_group(rows, 40, 1, cuda)[0] if name == "shard" else None
    md = sampling.SamplingMetadata(now["top_k"], now["top_p"], now["temperature"])

    def write(i):
        for k in [k for k in names if k != last] + [last]:
            v = sets[i][k]
            if v.dtype in (torch.float32, torch.bfloat16):
                torch.mul(v, 1.0, out=now[k])
            else:
                torch.add(v, 0, out=now[k])

    def call():
        if name in ("sample", "stream"):
            return sampling.sample(None, now["x"], md, noise=now["noise"])
        if name in ("sample_key", "stream_key"):
            return ops.sample(now["x"], now["top_k"], now["top_p"], now["temperature"], rng_key=now["key"], dim0_offset=now["offset"])
        if name == "gather":
            return tumpy.take_along_axis(now["x"], now["index"], 1)
        if name == "sort_through":
            return ops.argsort_rows(now["x"], in_perm=now["perm"])[1]
        return sampling.sample_vocab_sharded(None, now["x"], md, noise_shard=now["noise"], k_cand=40, exchange=ex)

    try:
        want = []
        for i in range(3):
            write(i)
            torch.cuda.synchronize()
            want.append(call().clone())
            torch.cuda.synchronize()
        got = []
        for i in range(12):
            write(i % 3)
            got.append(call())
        torch.cuda.synchronize()
        for i, g in enumerate(got):
            assert torch.equal(g, want[i % 3]), i
    finally:
        if ex is not None:
            ex.close()


# parameters of other types, one number for all rows among them, are converted: before both stages of a step, and, where the second
# one is called by itself, in order with it
@pytest.mark.parametrize("by_stages", [False, True])
@pytest.mark.parametrize("kind", ["wider", "numbers", "of one row", "on the host"])
def test_shard_parameters_of_other_types(cuda, kind, by_stages):
    rows, n = 300, 4096
    sets = _versions(cuda, rows, n, torch.bfloat16, n)
    ex = ops.Exchange.local_group(rows, 40, 1, cuda)[0]
    try:
        for i in range(12):
            s = sets[i % 3]
            args = s["top_k"], s["top_p"], s["temperature"]
            if kind in ("numbers", "of one row"):
                args = [a[i:i + 1] for a in args]
            same = [a.expand(rows).contiguous() for a in args]
            if kind == "wider":
                args = args[0].long(), args[1].double(), args[2].double()
            elif kind == "numbers":
                args = int(args[0]), float(args[1]), float(args[2])
            elif kind == "on the host":
                args = [a.cpu() for a in args]
            if by_stages:
                ops.exchange_shard_candidates(s["x"], 0, ex, noise_shard=s["noise"])
                got = ops.exchange_merge_and_sample(ex, *args)
            else:
                got = ops.exchange_step(s["x"], 0, ex, *args, noise_shard=s["noise"])
            block = ops.shard_candidates(s["x"], 0, 40, noise_shard=s["noise"], vocab_total=n)
            torch.cuda.synchronize()
            assert torch.equal(got, ops.merge_and_sample(block[None], *same)), i
    finally:
        ex.close()

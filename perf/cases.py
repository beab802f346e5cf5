"""The calls that a serving program makes of this package, as a list of cases with their inputs, work and tolerance.

Most of a decode step's calls are the fused sampler on `[batch, vocab]` logits; beside it stand the operators that
such a program uses on their own: top-k (speculative decoding, log-probabilities of the best tokens), key/payload sort,
gather along an axis, prefix sums of probabilities, and one rank's share of a sampler whose vocabulary is split over
several GPUs.  Sizes are those of the benchmark configurations and of the test-suite, and generic ones between them.
"""
import math

import torch

from tallax_b200 import sampling, tax, tumpy

_DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "i32": torch.int32}
_BYTES = {"bf16": 2, "f16": 2, "f32": 4, "i32": 4}

# Upper limits of the drawn sizes, by operator: elements (bytes for the sampler) that the listed cases reach.
_SAMPLE_BYTES = 256 * 151936 * 2
_TOPK_BYTES = 1024 * 262144 * 4
_SORT_ELEMENTS = 128 * 65536
_CUMSUM_ELEMENTS = 256 * 128256
_SHARD_ELEMENTS = 1024 * 151936


def listed():
    return [
        # A single request being decoded: latency and launches are all there is.  The same three parameters for
        # every request, noise from a key.
        {"name": "sample_1", "op": "sample", "rows": 1, "vocab": 128256, "dtype": "bf16", "noise": "key",
         "params": "same"},
        # A small decode batch with every request's own parameters, noise handed in.
        {"name": "sample_32", "op": "sample", "rows": 32, "vocab": 128256, "dtype": "bf16", "noise": "dense",
         "params": "mixed"},
        # The benchmark's decode batch.
        {"name": "sample_256", "op": "sample", "rows": 256, "vocab": 128256, "dtype": "bf16", "noise": "dense",
         "params": "mixed"},
        # f32 logits with an odd vocabulary, requests that set no top-k, some of them greedy.
        {"name": "sample_64_f32_open", "op": "sample", "rows": 64, "vocab": 50257, "dtype": "f32", "noise": "key",
         "params": "open"},
        # A large decode batch on a large vocabulary, noise from a key (how a decode loop calls the sampler).
        {"name": "sample_256_key", "op": "sample", "rows": 256, "vocab": 151936, "dtype": "bf16", "noise": "key",
         "params": "mixed"},
        # Top-k of a handful of rows (the benchmark's first configuration).
        {"name": "topk_8", "op": "top_k", "rows": 8, "n": 32768, "k": 64, "dtype": "f32", "dynamic": False},
        # Top-k over a large matrix (the benchmark's fourth configuration).
        {"name": "topk_1024", "op": "top_k", "rows": 1024, "n": 262144, "k": 128, "dtype": "f32", "dynamic": False},
        # Short ragged rows, sorted descending with their permutation.
        {"name": "argsort_64", "op": "sort", "rows": 64, "n": 4097, "dtype": "bf16", "keys": 1, "payloads": 0,
         "descending": True, "argsort": True},
        # Stable sort of long rows with ties and a payload (the benchmark's second configuration).
        {"name": "sort_128", "op": "sort", "rows": 128, "n": 65536, "dtype": "f32", "keys": 1, "payloads": 1,
         "descending": False, "argsort": False},
        # A few thousand random columns of every row of a large matrix (the benchmark's fourth configuration).
        {"name": "gather_1024", "op": "gather", "rows": 1024, "n": 262144, "picks": 4096, "dtype": "f32", "axis": 1},
        # Cumulative probability over the vocabulary.
        {"name": "cumsum_64", "op": "cumsum", "rows": 64, "cols": 128256, "dtype": "f32", "axis": 1, "reverse": False},
        # One rank's share of an 8-way split vocabulary of 151936: candidates of 1024 rows, then merge and sample.
        {"name": "shard_1024", "op": "shard", "rows": 1024, "n": 18992, "k": 50, "dtype": "bf16"},
    ]


def _log_int(rng, low, high):
    """A whole number between the two, spread evenly over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    op = rng.choice(["sample"] * 5 + ["top_k"] * 3 + ["sort"] * 2 + ["gather", "cumsum", "shard"])
    if op == "sample":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        vocab = _log_int(rng, 32000, 201088)
        if rng.random() < 0.6:
            vocab = (vocab + 127) // 128 * 128      # most models pad their vocabulary
        rows = _log_int(rng, 1, min(512, _SAMPLE_BYTES // (vocab * _BYTES[dtype])))
        return {"op": op, "rows": rows, "vocab": vocab, "dtype": dtype, "noise": rng.choice(["key", "dense"]),
                "params": rng.choice(["mixed", "mixed", "same", "open"])}
    if op == "top_k":
        dtype = rng.choice(["f32", "f32", "bf16"])
        n = _log_int(rng, 2048, 262144)
        rows = _log_int(rng, 1, min(1024, _TOPK_BYTES // (n * _BYTES[dtype])))
        return {"op": op, "rows": rows, "n": n, "k": _log_int(rng, 1, 128), "dtype": dtype,
                "dynamic": rng.random() < 0.25}
    if op == "sort":
        n = _log_int(rng, 128, 131072)
        keys = rng.choice([1, 1, 1, 2])
        rows = _log_int(rng, 1, max(1, min(1024, _SORT_ELEMENTS // (n * 2 * keys))))
        return {"op": op, "rows": rows, "n": n, "dtype": rng.choice(["f32", "bf16", "i32"]), "keys": keys,
                "payloads": rng.choice([0, 1]), "descending": rng.random() < 0.5, "argsort": rng.random() < 0.5}
    if op == "gather":
        rows, n = _log_int(rng, 8, 1024), _log_int(rng, 2048, 262144)
        return {"op": op, "rows": rows, "n": n, "picks": _log_int(rng, 16, 4096), "dtype": rng.choice(["f32", "bf16"]),
                "axis": rng.choice([0, 1, 1])}
    if op == "cumsum":
        cols = _log_int(rng, 128, 128256)
        rows = _log_int(rng, 1, max(1, min(1024, _CUMSUM_ELEMENTS // cols)))
        axis = rng.choice([1, 1, 0])
        if axis == 0:                               # (candidates, batch): the layout of the sampler's own top-p
            rows, cols = _log_int(rng, 16, 2048), _log_int(rng, 8, 4096)
        return {"op": op, "rows": rows, "cols": cols, "dtype": rng.choice(["f32", "f32", "i32"]), "axis": axis,
                "reverse": rng.random() < 0.3}
    n = _log_int(rng, 4096, 151936)
    rows = _log_int(rng, 32, min(1024, _SHARD_ELEMENTS // n))
    return {"op": op, "rows": rows, "n": n, "k": _log_int(rng, 16, 128), "dtype": "bf16"}


def _logits(rows, vocab, dtype, gen, spread=3.0):
    """Normal logits with eight likely tokens a row."""
    x = torch.randn((rows, vocab), generator=gen, device="cuda") * spread
    at = torch.randint(0, vocab, (rows, 8), generator=gen, device="cuda")
    x.scatter_add_(1, at, torch.full((rows, 8), 10.0, device="cuda"))
    return x.to(_DTYPES[dtype])


def _params(kind, rows, gen):
    """The requests' parameters.  mixed: every request its own, a tenth of them without top-k; same: one usual
    setting for all; open: top-k left out, top-p set, a quarter of the requests greedy."""
    u = torch.rand((4, rows), generator=gen, device="cuda")
    if kind == "mixed":
        top_k = (1 + (u[0] * 1024).to(torch.int32)).clamp_(1, 1024)
        top_k[u[1] < 0.1] = 0
        top_p, temperature = 0.6 + 0.4 * u[2], 0.5 + u[3]
    elif kind == "same":
        top_k = torch.full((rows,), 50, dtype=torch.int32, device="cuda")
        top_p, temperature = torch.full_like(u[2], 0.95), torch.full_like(u[3], 0.8)
    else:
        top_k = torch.zeros(rows, dtype=torch.int32, device="cuda")
        top_p, temperature = 0.8 + 0.2 * u[2], 0.5 + 0.7 * u[3]
        temperature[u[1] < 0.25] = 0.0
    return sampling.SamplingMetadata(top_k=top_k, top_p=top_p.contiguous(), temperature=temperature.contiguous())


def _keys(rows, n, dtype, gen, values=None):
    """Sort keys: normal, one entry in a hundred a copy of another entry of its row; or few different values."""
    if values is not None:
        return torch.randint(0, values, (rows, n), generator=gen, device="cuda").to(_DTYPES[dtype])
    x = torch.randn((rows, n), generator=gen, device="cuda")
    m = max(1, n // 100)
    of = torch.randint(0, n, (rows, m), generator=gen, device="cuda")
    first = torch.randint(0, n, (rows, 1), generator=gen, device="cuda")
    at = (first + torch.arange(m, device="cuda") * (n // m)) % n      # different places of a row
    x.scatter_(1, at, x.gather(1, of))
    return (x * 1e6).to(torch.int32) if dtype == "i32" else x.to(_DTYPES[dtype])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op, rows = case["op"], case["rows"]
    s = {"op": op, "case": case}
    if op == "sample":
        s["logits"] = _logits(rows, case["vocab"], case["dtype"], gen)
        s["metadata"] = _params(case["params"], rows, gen)
        s["key"] = (int(seed) & 0xFFFFFFFF, 0x243F6A88) if case["noise"] == "key" else None
        s["noise"] = torch.rand((rows, case["vocab"]), generator=gen, device="cuda") if case["noise"] == "dense" else None
    elif op == "top_k":
        s["x"] = torch.randn((rows, case["n"]), generator=gen, device="cuda").to(_DTYPES[case["dtype"]])
        if case["dynamic"]:
            s["k"] = torch.randint(1, case["k"] + 1, (rows,), generator=gen, device="cuda", dtype=torch.int32)
    elif op == "sort":
        # of two keys the first has few different values, so that the second one decides
        first = _keys(rows, case["n"], case["dtype"], gen, values=50 if case["keys"] > 1 else None)
        s["operands"] = [first] + [_keys(rows, case["n"], case["dtype"], gen) for _ in range(case["keys"] - 1)]
        for _ in range(case["payloads"]):
            s["operands"].append(torch.randint(0, 1 << 30, (rows, case["n"]), generator=gen, device="cuda",
                                               dtype=torch.int32))
    elif op == "gather":
        s["x"] = torch.randn((rows, case["n"]), generator=gen, device="cuda").to(_DTYPES[case["dtype"]])
        shape, high = ((rows, case["picks"]), case["n"]) if case["axis"] == 1 else ((case["picks"], case["n"]), rows)
        if case["axis"] == 0:                       # as many outputs as the other direction has
            s["x"] = s["x"][:, : max(1, min(case["n"], 4096))].contiguous()
            shape = (max(1, case["picks"] // 4), s["x"].shape[1])
        s["indices"] = torch.randint(0, high, shape, generator=gen, device="cuda", dtype=torch.int32)
    elif op == "cumsum":
        shape = (rows, case["cols"])
        if case["dtype"] == "i32":
            s["x"] = torch.randint(0, 100, shape, generator=gen, device="cuda", dtype=torch.int32)
        else:
            s["x"] = torch.softmax(torch.randn(shape, generator=gen, device="cuda") * 3.0, dim=case["axis"])
    else:
        s["logits"] = _logits(rows, case["n"], case["dtype"], gen, spread=2.0)
        s["noise"] = torch.rand((rows, case["n"]), generator=gen, device="cuda")
        k = torch.full((rows,), case["k"], dtype=torch.int32, device="cuda")
        s["metadata"] = sampling.SamplingMetadata(top_k=k, top_p=torch.full((rows,), 0.95, device="cuda"),
                                                  temperature=torch.full((rows,), 0.8, device="cuda"))
        s["exchange"] = sampling.make_vocab_exchange(rows, case["k"])
    return s


def run(s):
    op, case = s["op"], s["case"]
    if op == "sample":
        return sampling.sample(s["key"], s["logits"], s["metadata"], noise=s["noise"])
    if op == "top_k":
        if case["dynamic"]:
            return tax.top_dynamic_k(s["x"], s["k"], case["k"], block_token=1, guarantee_convergence=True,
                                     replace_val=-1e12)
        return tax.top_k(s["x"], case["k"], block_token=1)
    if op == "sort":
        return tax.sort(s["operands"], num_keys=case["keys"], is_stable=True, descending=case["descending"],
                        return_argsort=case["argsort"])
    if op == "gather":
        return tumpy.take_along_axis(s["x"], s["indices"], case["axis"])
    if op == "cumsum":
        return tax.cumsum(s["x"], case["axis"], reverse=case["reverse"])
    return sampling.sample_vocab_sharded(None, s["logits"], s["metadata"], noise_shard=s["noise"], k_cand=case["k"],
                                         exchange=s["exchange"])


def work(case):
    op, rows = case["op"], case["rows"]
    size = _BYTES[case["dtype"]]
    if op == "sample":
        # logits once, three parameters and a token a row; noise is needed where a token is kept only
        return {"bytes": rows * (case["vocab"] * size + 16), "flops": 0}
    if op == "top_k":
        return {"bytes": rows * (case["n"] * size + case["k"] * (size + 4)), "flops": 0}
    if op == "sort":
        item = 2 * (case["keys"] * size + case["payloads"] * 4) + (4 if case["argsort"] else 0)
        return {"bytes": rows * case["n"] * item, "flops": 0}
    if op == "gather":
        if case["axis"] == 1:
            outputs, values = rows * case["picks"], rows * case["picks"]
        else:
            cols = max(1, min(case["n"], 4096))
            outputs, values = max(1, case["picks"] // 4) * cols, rows * cols
        return {"bytes": outputs * (4 + size) + min(values, outputs) * size, "flops": 0}
    if op == "cumsum":
        return {"bytes": 2 * rows * case["cols"] * size, "flops": rows * case["cols"]}
    # logits once, the noise of k candidates a row, three parameters and a token
    return {"bytes": rows * (case["n"] * size + case["k"] * 4 + 16), "flops": 0}


def tolerance(case):
    if case["op"] == "cumsum" and case["dtype"] == "f32":
        return {"rel": 1e-5}
    if case["op"] in ("sample", "shard"):
        # a row whose cumulative mass comes within 1e-6 of top_p at a token may keep one token more or fewer
        return {"differ": 0.004}
    return "exact"

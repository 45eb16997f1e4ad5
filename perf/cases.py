"""Workloads the engine is timed on: searches through its public entry points, over the range of
corpus sizes, row widths, k and batch sizes that its tests, benchmark and the reference's demos use.

listed() names them, draw() gives further ones of the same ranges, prepare() makes a case's inputs on
the GPU (or on the host for the host-buffer entry points), run() is one search, work() what it cannot
do without, exact() its distances from plain FP64 arithmetic.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "knn-toolbox_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "knn-toolbox_gb300"))

import cuknns  # noqa: E402

# Entry points ("call"):
#   search   cuknns.search on device tensors, every default: corpus and queries prepared in the call
#   index    Index.search on a corpus prepared once, into the caller's output tensors, without the
#            per-call device check: a program that keeps a corpus resident and queues batches
#   dropin   gpuknnsBitonic on page-locked host arrays (the reference's own C API)
#   double   the double library on host arrays
# Data ("data"): the benchmark's distributions -- "uniform" [0,1), "int" integer descriptors
# (clip(round(|N(0,40)|), 0, 255), 8 % zeros; exact in BF16), "mixture" L2-normalised Gaussian mixture,
# "aniso" coordinate j ~ N(0, 1/sqrt(1+j)).
# "form": exact, bf16 or fp8 keys ("c": shortlist factor of the latter two).


def _case(name, call, data, N, D, Q, k, form="exact", c=0):
    return {"name": name, "call": call, "data": data, "N": N, "D": D, "Q": Q, "k": k, "form": form, "c": c}


def listed():
    return [
        # the smallest calls: a handful of queries against a thousand short rows
        _case("tiny", "search", "uniform", 1_000, 32, 4, 5),
        # a small corpus of wide rows (document or image embeddings kept by a small program)
        _case("small_wide", "search", "uniform", 10_000, 300, 500, 10),
        # the benchmark's plain FP32 workload
        _case("uniform64k", "search", "uniform", 65_536, 128, 1_024, 16),
        # the reference demos' widest common shape: 32,768 rows of 1,024 columns, 256 queries
        _case("wide_rows", "search", "uniform", 32_768, 1_024, 256, 16),
        # the largest k of the reference (512) on odd sizes
        _case("large_k", "search", "uniform", 100_003, 43, 777, 512),
        # a million FP32 rows, ragged, one search of a fresh corpus
        _case("float_million", "search", "mixture", 1_000_003, 96, 2_000, 10),
        # the benchmark's headline: a million integer descriptors, 10,000 queries, k = 100
        _case("int_million", "search", "int", 1_000_000, 128, 10_000, 100),
        # a serving batch on the resident two-million-row corpus
        _case("serve_batch", "index", "int", 2_000_000, 128, 48, 10),
        # the precision forms on resident corpora: BF16 keys on 4M x 96, E4M3 keys on 256-column rows
        _case("bf16_form", "index", "mixture", 4_000_000, 96, 4_096, 10, "bf16", 4),
        _case("fp8_form", "index", "aniso", 2_000_000, 256, 2_048, 32, "fp8", 2),
        # the drop-in C entry point on page-locked host buffers (the copy is part of the call)
        _case("dropin_host", "dropin", "int", 200_000, 128, 1_000, 32),
        # the double library at the size of the reference's double demo (64 queries, k = 128)
        _case("double_host", "double", "uniform", 32_768, 128, 64, 128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_MOST = 3.1e12  # operations of the largest case


def draw(rng):
    kind = rng.choice(["small", "small_wide", "medium", "wide", "large_k", "float", "int", "serve", "resident",
                       "bf16", "fp8", "dropin", "double"])
    form, c, call, data = "exact", 0, "search", "uniform"
    if kind == "small":
        N, D, Q, k = _log(rng, 300, 16_000), _log(rng, 5, 128), _log(rng, 1, 4_096), _log(rng, 1, 100)
        data = rng.choice(["uniform", "mixture", "int"])
    elif kind == "small_wide":
        N, D, Q, k = _log(rng, 1_000, 16_000), rng.randint(129, 512), _log(rng, 1, 1_024), _log(rng, 1, 64)
    elif kind == "medium":
        N, D, Q, k = _log(rng, 16_384, 131_000), _log(rng, 16, 128), _log(rng, 1, 16_384), _log(rng, 1, 100)
        data = rng.choice(["uniform", "mixture", "int"])
    elif kind == "wide":
        N, D, Q, k = _log(rng, 16_384, 65_536), _log(rng, 129, 2_048), _log(rng, 1, 1_024), _log(rng, 1, 128)
    elif kind == "large_k":
        N, D, Q, k = _log(rng, 40_000, 200_000), _log(rng, 32, 128), _log(rng, 16, 2_048), rng.randint(129, 512)
    elif kind == "float":
        N, D, Q, k = _log(rng, 131_072, 1_500_000), _log(rng, 32, 128), _log(rng, 16, 4_096), _log(rng, 1, 100)
        data = rng.choice(["mixture", "uniform"])
    elif kind == "int":
        N, D, Q, k = _log(rng, 131_072, 1_000_000), _log(rng, 32, 128), _log(rng, 100, 10_000), _log(rng, 1, 100)
        data = "int"
    elif kind == "serve":
        N, D, Q, k = _log(rng, 500_000, 2_000_000), 128, _log(rng, 1, 512), rng.choice([1, 10, 100])
        call, data = "index", "int"
    elif kind == "resident":
        N, D, Q, k = _log(rng, 131_072, 2_000_000), _log(rng, 32, 128), _log(rng, 1, 2_048), rng.choice([1, 10, 100])
        call, data = "index", "mixture"
    elif kind == "bf16":
        N, D, Q, k = _log(rng, 500_000, 4_000_000), _log(rng, 48, 128), _log(rng, 64, 4_096), rng.choice([10, 32])
        call, data, form, c = "index", "mixture", "bf16", 4
    elif kind == "fp8":
        N, D, Q, k = _log(rng, 500_000, 2_000_000), 256, _log(rng, 64, 2_048), 32
        call, data, form, c = "index", "aniso", "fp8", 2
    elif kind == "dropin":
        N, D, Q, k = _log(rng, 20_000, 300_000), _log(rng, 32, 128), _log(rng, 16, 2_048), _log(rng, 1, 128)
        call, data = "dropin", rng.choice(["uniform", "int"])
    else:
        N, D, Q, k = _log(rng, 4_096, 65_536), _log(rng, 32, 256), _log(rng, 16, 512), _log(rng, 1, 128)
        call = "double"
    Q = max(1, min(Q, int(_MOST / (2.0 * N * D))))
    return {"call": call, "data": data, "N": N, "D": D, "Q": Q, "k": min(k, N), "form": form, "c": c}


def _rows(gen, data, n, D, dtype=torch.float32, shared=None):
    dev = gen.device
    if data == "uniform":
        return torch.rand((n, D), generator=gen, device=dev, dtype=dtype)
    if data == "int":
        x = torch.randn((n, D), generator=gen, device=dev).mul_(40.0).abs_().round_().clamp_(0, 255)
        return x.mul_(torch.rand((n, D), generator=gen, device=dev) >= 0.08)
    if data == "mixture":
        lab = torch.randint(0, shared.shape[0], (n,), generator=gen, device=dev)
        x = torch.randn((n, D), generator=gen, device=dev).mul_(0.15).add_(shared[lab])
        return x.div_(torch.linalg.vector_norm(x, dim=1, keepdim=True))
    if data == "aniso":
        s = (1.0 + torch.arange(D, device=dev, dtype=torch.float32)) ** -0.25
        return torch.randn((n, D), generator=gen, device=dev).mul_(s)
    raise ValueError(data)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 1_000_003 + 17)
    D = case["D"]
    shared = torch.randn((1024, D), generator=gen, device="cuda") if case["data"] == "mixture" else None
    dtype = torch.float64 if case["call"] == "double" else torch.float32
    return (_rows(gen, case["data"], case["N"], D, dtype, shared), _rows(gen, case["data"], case["Q"], D, dtype, shared))


def _options(case):
    if case["form"] == "bf16":
        return {"precision": cuknns.PREC_BF16, "shortlist": case["c"]}
    if case["form"] == "fp8":
        return {"precision": cuknns.PREC_FP8, "shortlist": case["c"]}
    return {}


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def prepare(case, seed):
    corpus, queries = _inputs(case, seed)
    s = {"call": case["call"], "k": case["k"], "options": _options(case)}
    if case["call"] == "dropin":
        s["corpus"], s["queries"] = _pinned(corpus), _pinned(queries)
    elif case["call"] == "double":
        s["corpus"], s["queries"] = corpus.cpu().numpy(), queries.cpu().numpy()
    else:
        s["corpus"], s["queries"] = corpus, queries
    if case["call"] == "index":
        s["index"] = cuknns.Index(corpus, tf32=case["form"] == "exact", fp8=case["form"] == "fp8")
        s["dist"] = torch.empty((case["Q"], case["k"]), dtype=torch.float32, device="cuda")
        s["idx"] = torch.empty((case["Q"], case["k"]), dtype=torch.int32, device="cuda")
    return s


def run(state):
    call, k = state["call"], state["k"]
    if call == "search":
        dist, idx = cuknns.search(state["corpus"], state["queries"], k)
    elif call == "index":
        dist, idx = state["index"].search(state["queries"], k, dist=state["dist"], idx=state["idx"], check=False,
                                          **state["options"])
    elif call == "dropin":
        dist, idx, _ = cuknns.gpuknnsBitonic(state["queries"], state["corpus"], k)
    else:
        dist, idx = cuknns.search_host_f64(state["corpus"], state["queries"], k)
    return {"dist": dist, "idx": idx}


def work(case):
    N, D, Q, k = case["N"], case["D"], case["Q"], case["k"]
    value = 8 if case["call"] == "double" else 4
    # a resident corpus is read as the copy that its keys need: 1 byte per value for E4M3 keys, 2 for
    # BF16 keys (also integer descriptors, exact in BF16)
    stored = value
    if case["call"] == "index":
        stored = 1 if case["form"] == "fp8" else 2 if case["form"] == "bf16" or case["data"] == "int" else 4
    return {"bytes": stored * N * D + value * Q * D + Q * k * (value + 4), "flops": 2 * N * Q * D}


def exact(case, seed):
    corpus, queries = _inputs(case, seed)
    c, q, k = corpus.double(), queries.double(), case["k"]
    cc = (c * c).sum(1)
    out = []
    step = max(1, min(case["Q"], (1 << 29) // case["N"]))
    for i in range(0, case["Q"], step):
        b = q[i:i + step]
        near = torch.addmm(cc[None, :], b, c.T, alpha=-2.0).topk(k, dim=1, largest=False).indices
        # the k nearest by direct difference: no cancellation in what is returned
        d = torch.cat([((c[near[j:j + 64]] - b[j:j + 64, None, :]) ** 2).sum(2) for j in range(0, b.shape[0], 64)])
        out.append(d.sort(dim=1).values)
    dist = torch.cat(out)
    if case["call"] in ("dropin", "double"):
        dist = dist.cpu().numpy()
    return {"dist": dist, "idx": None}

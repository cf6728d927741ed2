"""Workloads of the flat index that its speed is judged by.

A case is one pass of a user's program through the index's Python classes:

``search``   one call of ``search()``: queries on the device give results on the device, numpy
             queries (``host``) give numpy results.
``tokens``   four ``search_async()`` calls in flight, then their ``wait()``s: a server that answers
             independent batches.
``refill``   ``reset()``, ``add()`` of all rows, ``reconstruct_n()`` of all rows: storing vectors and
             reading them back.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges.  Inputs are synthetic
and made from the seed alone, with the distributions of this repository's benchmark and tests:
``uniform`` U[0, 1), ``normal`` N(0, 1) * 0.05, ``unit`` normal rows of length one, ``mixture`` 1,000
normal clusters of sigma 0.1 around uniform centres.
"""
import math

import torch

import faiss_metal_b200 as fm

METRIC = {"l2": fm.METRIC_L2, "ip": fm.METRIC_INNER_PRODUCT}
STORAGE = {"f32": fm.STORAGE_F32, "f16": fm.STORAGE_F16, "bf16": fm.STORAGE_BF16}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}
TOKENS = 4            # searches in flight in a "tokens" pass
CENTRES = 1000
CHUNK_BYTES = 1 << 30  # fp32 rows generated at a time

_resources = None


def _res():
    """One resources object (streams, scratch) per program, shared by its indexes."""
    global _resources
    if _resources is None:
        _resources = fm.StandardB200Resources(0)
    return _resources


def _case(name, op, metric, storage, nb, nq, d, k, dist, host=False):
    return {"name": name, "op": op, "metric": metric, "storage": storage, "nb": nb, "nq": nq, "d": d,
            "k": k, "dist": dist, "host": host}


def listed():
    return [
        # the smallest row of the usual flat-index benchmark grid: launches and latency are all of it
        _case("small_grid", "search", "l2", "f32", 10_000, 100, 32, 10, "uniform"),
        # one query at a time from host memory against a small index: an interactive lookup
        _case("single_small_host", "search", "l2", "f32", 100_000, 1, 128, 10, "uniform", host=True),
        # a retrieval server with independent requests of two dozen queries each, odd row count and width
        _case("tokens_serving", "tokens", "ip", "f16", 1_000_003, 24, 770, 100, "unit", host=True),
        # an ordinary batch against an index that fits the L2 cache
        _case("batch_100k", "search", "l2", "f32", 100_000, 1_000, 128, 10, "uniform"),
        # a large batch of unit vectors by inner product: building a k-NN graph of embeddings
        _case("batch_1m_ip", "search", "ip", "f16", 1_000_000, 10_000, 768, 100, "unit"),
        # the largest: a big embedding collection at the widest usual dimension
        _case("batch_10m_wide", "search", "l2", "bf16", 10_000_000, 4_096, 1536, 32, "normal"),
        # a thousand neighbours per query in clustered data: candidates for a second stage
        _case("candidates_1024", "search", "l2", "f32", 5_000_000, 2_048, 96, 1024, "mixture"),
        # a stream of single queries against the largest row count
        _case("single_50m_host", "search", "l2", "f16", 50_000_000, 1, 128, 10, "uniform", host=True),
        # a handful of queries, full-precision rows of an odd count and width
        _case("few_2m_f32", "search", "ip", "f32", 2_500_001, 6, 100, 32, "normal"),
        # one user's few queries with a deep list for a re-ranking model
        _case("rerank_200", "search", "l2", "bf16", 1_000_000, 4, 384, 200, "normal"),
        # very deep lists: candidate generation for offline mining
        _case("deep_2048", "search", "ip", "f16", 300_007, 50, 256, 2048, "unit"),
        # replacing the index's contents and reading them back
        _case("refill_f32", "refill", "l2", "f32", 1_000_003, 0, 384, 0, "normal"),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; half of them odd or otherwise uneven."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v if rng.random() < 0.5 else v | 1))


def draw(rng):
    """One more case of the same ranges: rows 10 k to 50 M, queries 1 to 10 k, d 32 to 1536, k 1 to 2048."""
    while True:
        op = rng.choice(["search"] * 8 + ["tokens", "refill"])
        metric = rng.choice(["l2", "ip"])
        storage = rng.choice(["f32", "f16", "bf16"])
        d = _log_int(rng, 32, 1536)
        if rng.random() < 0.5:
            d = max(32, d // 32 * 32)
        dist = rng.choice(["unit", "normal"] if metric == "ip" else ["uniform", "normal", "mixture"])
        nb = _log_int(rng, 10_000, 50_000_000)
        nq = k = 0
        host = rng.random() < 0.3
        if op == "refill":
            if nb * d * 4 > (2 << 30):
                continue
        else:
            nq = _log_int(rng, 1, 10_000)
            k = _log_int(rng, 1, 2048)
            if op == "tokens":
                host = True
                if nq > 256:
                    continue
            pairs = nq * nb
            # well inside the largest listed case, input generation included
            if 2.0 * pairs * d > 2e13 or nb * d * 4 > 26e9 or pairs > (1e9 if k > 1024 else 1e10):
                continue
        c = _case("", op, metric, storage, nb, nq, d, k, dist, host)
        del c["name"]
        return c


class _Source:
    """Rows of a case's distribution, block by block, on the device."""

    def __init__(self, case, seed):
        self.dist, self.d = case["dist"], case["d"]
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        if self.dist == "mixture":
            self.centres = torch.rand((CENTRES, self.d), generator=self.gen, device="cuda") * 2 - 1

    def rows(self, n):
        shape = (n, self.d)
        if self.dist == "uniform":
            return torch.rand(shape, generator=self.gen, device="cuda")
        x = torch.randn(shape, generator=self.gen, device="cuda")
        if self.dist == "normal":
            return x.mul_(0.05)
        if self.dist == "unit":
            return x.div_(x.norm(dim=1, keepdim=True))
        which = torch.randint(CENTRES, (n,), generator=self.gen, device="cuda")
        return x.mul_(0.1).add_(self.centres[which])


def prepare(case, seed):
    src = _Source(case, seed)
    nb, d = case["nb"], case["d"]
    index = fm.B200IndexFlat(_res(), d, METRIC[case["metric"]], STORAGE[case["storage"]])
    state = {"case": case, "index": index}
    if case["op"] == "refill":
        x = src.rows(nb)
        state["x"] = x.cpu().numpy() if case["host"] else x
        return state
    index.reserve(nb)
    step = max(1, CHUNK_BYTES // (4 * d))
    for r0 in range(0, nb, step):
        index.add(src.rows(min(step, nb - r0)))
    batches = [src.rows(case["nq"]) for _ in range(TOKENS if case["op"] == "tokens" else 1)]
    state["queries"] = [q.cpu().numpy() if case["host"] else q for q in batches]
    if case["op"] == "tokens":
        # a server's result buffers, one set per request in flight
        state["out"] = [(torch.empty((case["nq"], case["k"]), dtype=torch.float32).numpy(),
                         torch.empty((case["nq"], case["k"]), dtype=torch.int64).numpy()) for _ in batches]
    return state


def run(state):
    case, index = state["case"], state["index"]
    if case["op"] == "search":
        return index.search(state["queries"][0], case["k"])
    if case["op"] == "tokens":
        tokens = [index.search_async(q, case["k"], dist, labels)
                  for q, (dist, labels) in zip(state["queries"], state["out"])]
        for t in tokens:
            t.wait()
        return state["out"]
    x = state["x"]
    index.reset()
    index.add(x)
    if case["host"]:
        return index.reconstruct_n(0, case["nb"])
    return index.reconstruct_n(0, case["nb"], torch.empty_like(x))


def work(case):
    nb, nq, d, k, s = case["nb"], case["nq"], case["d"], case["k"], BYTES[case["storage"]]
    if case["op"] == "refill":
        # rows in, stored, read again, out; the norms' multiply-adds
        return {"bytes": nb * d * (4 + s + s + 4), "flops": 2 * nb * d}
    batches = TOKENS if case["op"] == "tokens" else 1
    return {"bytes": batches * (nb * d * s + nq * d * 4 + nq * k * 12), "flops": batches * 2 * nq * nb * d}


def tolerance(case):
    # About four times what was seen between the streaming and the tensor path (fp32 rows: rel 1.2e-5,
    # max 2.9e-5) and against float64 of the stored operands (16-bit rows: max 1.9e-6): sums in another
    # order.  Labels differ only where neighbours tie within that.
    if case["op"] == "refill":
        return "exact"
    if case["storage"] == "f32":
        return {"rel": 5e-5, "max": 1.2e-4, "differ": 0.01}
    return {"rel": 2e-6, "max": 8e-6, "differ": 0.01}

"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the public Python API of ``hnsw_gpu``: graph search
over an index opened from its file bytes, exact brute-force search, and index
construction on the device. Sizes follow the configurations of the tests and
the benchmark (10k to 1M rows, dimensions 32 to 768, M 16 and 24,
efConstruction 200, k 1 to 100, ef 16 to 512, filters of 1 % to 90 %), with
index sizes that can be built in about a second.

A case is a dict of plain values:

    kind       "graph", "brute" or "build"
    n, dim     rows of the index and their dimension
    metric     0 squared L2, 1 inner product, 2 cosine
    clusters   centers of the Gaussian mixture the rows and queries come from
               (0: independent normal components), sigma its spread
    nq, k, ef  queries of the batch, results per query, candidate list size
    ...        options of the kind, see graph_case, brute_case, build_case
"""

import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.abspath("hnsw-index_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import hnsw_gpu as H  # noqa: E402

_MIXED_K = (1, 10, 100)
_MIXED_EF = (16, 32, 64, 128, 256, 512)


def graph_case(**kw):
    """m: links per node; device: queries and results stay on the GPU
    (search_device) instead of host arrays; persistent: the work-queue mode;
    mixed: "" one k and ef for all, "batch" k of {1, 10, 100} and ef of
    {16..512} per query, "serving" k of {10, 100} and ef log-uniform 32..512;
    int8: codes walk the graph, exact re-rank; dead: share of tombstones;
    filters: number of filter bitmaps (0: none), filtered: share of the
    queries that use one, sel_lo..sel_hi: their selectivity (log-uniform)."""
    case = dict(kind="graph", metric=0, m=16, clusters=0, sigma=0.3, nq=1, k=10, ef=64, device=False, persistent=False,
                mixed="", int8=False, dead=0.0, filters=0, filtered=0.0, sel_lo=1.0, sel_hi=1.0)
    case.update(kw)
    return case


def brute_case(**kw):
    """precision: "fp32", "bf16" or "bf16x3" scoring (results are exact in
    all); sel: share of the rows that the key filter admits (1: no filter)."""
    case = dict(kind="brute", metric=0, clusters=0, sigma=0.5, nq=1, k=10, precision="fp32", sel=1.0)
    case.update(kw)
    return case


def build_case(**kw):
    """m: links per node; efc: efConstruction."""
    case = dict(kind="build", metric=0, m=16, efc=200, clusters=0, sigma=0.3)
    case.update(kw)
    return case


def listed():
    return [
        # One search at a time: what a user's `index.search(...)` costs.
        graph_case(name="graph-one", n=50_000, dim=128, clusters=50),
        # The small gaussian set: 1,000 queries from host memory.
        graph_case(name="graph-10k-gaussian", n=10_000, dim=128, nq=1_000),
        # The headline batch: clustered rows larger than L2, 10,000 queries
        # resident on the GPU, work-queue mode.
        graph_case(name="graph-500k-batch", n=500_000, dim=128, clusters=500, nq=10_000, device=True, persistent=True),
        # A wide beam with many results per query, cosine, odd sizes.
        graph_case(name="graph-cosine-wide", n=100_003, dim=100, metric=2, clusters=100, nq=2_500, k=100, ef=256),
        # The batching workload: int8 walk with exact re-rank, tombstones,
        # key filters of very different selectivity, uneven k and ef.
        graph_case(name="graph-int8-filtered", n=100_000, dim=96, metric=1, m=24, clusters=200, sigma=0.4, nq=3_000,
                   persistent=True, mixed="batch", int8=True, dead=0.05, filters=32, filtered=1.0, sel_lo=0.01,
                   sel_hi=0.9),
        # One batch of the serving workload: few requests, a third filtered;
        # its slowest request is its time.
        graph_case(name="graph-serving", n=200_000, dim=128, clusters=200, nq=256, persistent=True, mixed="serving",
                   filters=16, filtered=0.3, sel_lo=0.05, sel_hi=0.5),
        # Exact search for one query.
        brute_case(name="brute-one", n=200_000, dim=128, clusters=200),
        # The exact search of the recall measurements: 100k x 128, k = 10.
        brute_case(name="brute-100k-batch", n=100_000, dim=128, nq=1_000),
        # Exact search under a key filter, odd sizes.
        brute_case(name="brute-filtered", n=50_021, dim=100, metric=1, clusters=50, nq=100, k=20, sel=0.2),
        # Embeddings of 768 dimensions, cosine, top 100, compensated BF16
        # tensor-core scoring.
        brute_case(name="brute-768-bf16x3", n=200_000, dim=768, metric=2, clusters=800, nq=2_000, k=100,
                   precision="bf16x3"),
        # Plain BF16 scoring of a smaller batch, odd sizes.
        brute_case(name="brute-bf16", n=100_003, dim=200, clusters=400, nq=300, k=10, precision="bf16"),
        # Building an index on the GPU and writing its file.
        build_case(name="build-50k", n=50_000, dim=128, clusters=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: sizes spread over their logarithm."""
    what = rng.choice(["graph", "graph", "graph", "mixed", "brute", "brute", "tensor", "build"])
    metric = rng.choice([0, 0, 1, 2])
    clusters = rng.choice([0, 50, 200])
    if what == "graph":
        n = _log_int(rng, 2_000, 500_000)
        ef = _log_int(rng, 16, 512)
        # No more expansions in all than the headline batch has.
        nq = _log_int(rng, 1, max(2, min(10_000, 600_000 // ef)))
        return graph_case(n=n, dim=_log_int(rng, 32, 256), metric=metric, m=rng.choice([8, 16, 24]), clusters=clusters,
                          nq=nq, k=rng.randint(1, min(ef, 100)), ef=ef, device=rng.random() < 0.4,
                          persistent=rng.random() < 0.5, int8=rng.random() < 0.2)
    if what == "mixed":
        return graph_case(n=_log_int(rng, 5_000, 100_000), dim=_log_int(rng, 32, 160), metric=metric,
                          m=rng.choice([16, 24]), clusters=clusters, nq=_log_int(rng, 16, 2_000), persistent=True,
                          mixed=rng.choice(["batch", "serving"]), int8=rng.random() < 0.5,
                          dead=rng.choice([0.0, 0.05]), filters=rng.randint(1, 32), filtered=rng.uniform(0.2, 1.0),
                          sel_lo=0.02, sel_hi=0.9)
    if what == "brute":
        n = _log_int(rng, 2_000, 200_000)
        dim = _log_int(rng, 16, 768)
        nq = _log_int(rng, 1, max(2, min(2_000, 12_800_000_000 // (n * dim))))
        return brute_case(n=n, dim=dim, metric=metric, clusters=clusters, nq=nq, k=rng.randint(1, 100),
                          sel=rng.choice([1.0, 1.0, rng.uniform(0.05, 0.9)]))
    if what == "tensor":
        return brute_case(n=_log_int(rng, 20_000, 200_000), dim=_log_int(rng, 64, 768), metric=metric,
                          clusters=rng.choice([200, 800]), nq=_log_int(rng, 1, 2_000), k=rng.randint(1, 100),
                          precision=rng.choice(["bf16", "bf16x3"]))
    return build_case(n=_log_int(rng, 2_000, 50_000), dim=_log_int(rng, 32, 160), metric=metric,
                      m=rng.choice([8, 16, 24]), efc=rng.choice([100, 200]), clusters=clusters)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _data(case, seed):
    """(rows, queries) of the case's distribution, made on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + 17)
    n, nq, dim = case["n"], case.get("nq", 0), case["dim"]

    def normal(rows):
        return torch.randn(rows, dim, generator=gen, device="cuda")

    if not case["clusters"]:
        return normal(n), normal(nq)
    centers = normal(case["clusters"])

    def points(rows):
        which = torch.randint(case["clusters"], (rows,), generator=gen, device="cuda")
        return centers[which] + case["sigma"] * normal(rows)

    return points(n), points(nq)


def _bitmaps(rng, count, n, lo, hi):
    """`count` key bitmaps with selectivities log-uniform in [lo, hi]."""
    words = (n + 63) // 64
    sel = np.exp(rng.uniform(math.log(lo), math.log(hi), count))
    out = np.zeros((count, words * 8), np.uint8)
    for i in range(count):
        bits = np.packbits(rng.random(n) < sel[i], bitorder="little")
        out[i, : bits.size] = bits
    return out.view(np.uint64), words


def prepare(case, seed):
    rows, queries = _data(case, seed)
    rows_host = rows.cpu().numpy()
    if case["kind"] == "build":
        return {"case": case, "rows": rows_host, "keys": np.arange(case["n"], dtype=np.uint64)}
    queries_host = queries.cpu().numpy()
    rng = np.random.default_rng(int(seed) + 1)
    if case["kind"] == "brute":
        index = H.BruteForceIndex(case["dim"], H.Metric(case["metric"]))
        index.insert_batch(np.arange(case["n"], dtype=np.uint64), rows_host)
        kw = {}
        if case["sel"] < 1.0:
            bits, _ = _bitmaps(rng, 1, case["n"], case["sel"], case["sel"])
            kw = {"filter_bits": bits, "filter_nbits": case["n"]}
        precision = {"fp32": H.Precision.FP32, "bf16": H.Precision.BF16, "bf16x3": H.Precision.BF16X3}[case["precision"]]
        return {"case": case, "index": index, "queries": queries_host, "precision": precision, "kw": kw}

    builder = H.IndexBuilder(case["dim"], H.Metric(case["metric"]), H.HnswParams(m=case["m"], ef_construction=200, seed=7))
    builder.insert_batch_gpu(np.arange(case["n"], dtype=np.uint64), rows_host)
    if case["int8"]:
        builder.enable_quantization()
    index = H.HnswIndex.from_bytes(builder.to_bytes())
    del builder
    if case["dead"] > 0:
        index.set_tombstones((rng.random(case["n"]) < case["dead"]).astype(np.uint8))
    state = {"case": case, "index": index, "queries": queries_host}
    nq, k = case["nq"], case["k"]
    if case["device"]:
        state["d_queries"] = queries
        state["d_keys"] = torch.zeros(nq, k, dtype=torch.int64, device="cuda")
        state["d_dist"] = torch.zeros(nq, k, device="cuda")
        state["d_count"] = torch.zeros(nq, dtype=torch.int32, device="cuda")
        state["d_status"] = torch.zeros(nq, dtype=torch.int32, device="cuda")
        return state
    kw = {"quantized": case["int8"], "mode": 1 if case["persistent"] else 0}
    if case["mixed"] == "batch":
        kw["ks"] = rng.choice(np.array(_MIXED_K, np.uint32), nq)
        kw["efs"] = rng.choice(np.array(_MIXED_EF, np.uint32), nq)
    elif case["mixed"] == "serving":
        kw["ks"] = rng.choice(np.array([10, 100], np.uint32), nq)
        kw["efs"] = np.exp(rng.uniform(math.log(32), math.log(512), nq)).astype(np.uint32)
    if case["filters"]:
        bits, words = _bitmaps(rng, case["filters"], case["n"], case["sel_lo"], case["sel_hi"])
        kw["filter_bits"] = bits
        kw["filter_nbits"] = case["n"]
        kw["filter_stride"] = words
        kw["filter_ids"] = rng.integers(0, case["filters"], nq).astype(np.uint32)
        kw["filter_used"] = (rng.random(nq) < case["filtered"]).astype(np.uint8)
    state["kw"] = kw
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _found(keys, dist, count, status):
    """The results of a batch: entries past a query's count hold nothing."""
    if keys.size and int(count.min()) < keys.shape[1]:
        none = np.arange(keys.shape[1], dtype=np.uint32)[None, :] >= count[:, None]
        keys[none] = 0
        dist[none] = 0.0
    return {"keys": keys, "dist": dist, "count": count, "status": status}


def run(state):
    case = state["case"]
    if case["kind"] == "build":
        builder = H.IndexBuilder(case["dim"], H.Metric(case["metric"]),
                                 H.HnswParams(m=case["m"], ef_construction=case["efc"], seed=7))
        builder.insert_batch_gpu(state["keys"], state["rows"])
        data = builder.to_bytes()
        # Lists are stored at their own lengths: the file in a buffer of a
        # size that holds it whatever they are.
        file = np.zeros(case["n"] * (4 * case["dim"] + 16 * case["m"] + 64) + 4096, np.uint8)
        file[: len(data)] = np.frombuffer(data, np.uint8)
        return {"file": file, "bytes": len(data)}
    if case["kind"] == "brute":
        return _found(*state["index"].search_arrays(state["queries"], case["k"], state["precision"], **state["kw"]))
    if case["device"]:
        state["index"].search_device(state["d_queries"].data_ptr(), case["nq"], case["k"], case["ef"],
                                     state["d_keys"].data_ptr(), state["d_dist"].data_ptr(),
                                     state["d_count"].data_ptr(), state["d_status"].data_ptr(),
                                     stream=torch.cuda.current_stream().cuda_stream, quantized=case["int8"],
                                     mode=1 if case["persistent"] else 0)
        return {"keys": state["d_keys"], "dist": state["d_dist"], "count": state["d_count"],
                "status": state["d_status"]}
    return _found(*state["index"].search_arrays(state["queries"], case["k"], case["ef"], **state["kw"]))


# ---------------------------------------------------------------------------
# What a pass cannot do without, and its exact results
# ---------------------------------------------------------------------------
def _walk(case, ef, m):
    """Distances of one query's walk: about 11 per unit of ef at M = 16."""
    return min(case["n"], 11.0 * ef * m / 16.0)


def work(case):
    n, dim = case["n"], case["dim"]
    row = 4 * dim
    flops_per = (3 if case["metric"] == 0 else 2) * dim
    if case["kind"] == "build":
        dists = n * _walk(case, case["efc"], case["m"])
        return {"bytes": n * (2 * row + 4 * (2 * case["m"] + 1) + 16), "flops": dists * flops_per}
    nq, k = case["nq"], case["k"]
    if case["kind"] == "brute":
        scored = n * case["sel"]
        return {"bytes": scored * row + nq * (row + 12 * k), "flops": nq * scored * flops_per}
    ef = {"": case["ef"], "batch": float(np.mean(_MIXED_EF)), "serving": 173.0}[case["mixed"]]
    k = {"": k, "batch": 37.0, "serving": 55.0}[case["mixed"]]
    dists = nq * _walk(case, ef, case["m"])
    if case["filters"]:
        # A filtered walk goes on until ef admitted nodes are found.
        mean = (math.log(case["sel_hi"] / case["sel_lo"]) / (case["sel_hi"] - case["sel_lo"])
                if case["sel_hi"] > case["sel_lo"] else 1.0 / case["sel_hi"])
        per = min(n, _walk(case, ef, case["m"]) * mean)
        dists = (1.0 - case["filtered"]) * dists + case["filtered"] * nq * per
    walk_row = dim if case["int8"] else row
    lists = dists / 11.0 * 4 * (2 * case["m"])
    index_bytes = n * (walk_row + 8 * case["m"])
    return {"bytes": min(index_bytes, dists * walk_row + lists) + nq * (row + 12 * k), "flops": dists * flops_per}


def exact(case, seed):
    """Brute-force distances in 64 bits; a graph search has no such value
    (its results are those of the walk, exact distances of approximate
    neighbors), nor has a file."""
    if case["kind"] != "brute":
        return None
    rows, queries = _data(case, seed)
    rows, queries = rows.double(), queries.double()
    if case["sel"] < 1.0:
        bits, _ = _bitmaps(np.random.default_rng(int(seed) + 1), 1, case["n"], case["sel"], case["sel"])
        keep = np.unpackbits(bits.view(np.uint8).reshape(-1), bitorder="little")[: case["n"]].astype(bool)
        rows = rows[torch.from_numpy(keep).cuda()]
    if case["metric"] == 2:
        rows = rows / rows.norm(dim=1, keepdim=True)
        queries = queries / queries.norm(dim=1, keepdim=True)
    k = min(case["k"], rows.shape[0])
    dist = np.zeros((case["nq"], case["k"]))
    step = max(1, (1 << 27) // max(rows.shape[0], 1))
    for i in range(0, case["nq"], step):
        q = queries[i : i + step]
        dot = q @ rows.T
        if case["metric"] == 0:
            d = (q * q).sum(1)[:, None] + (rows * rows).sum(1)[None, :] - 2.0 * dot
        else:
            d = -dot if case["metric"] == 1 else 1.0 - dot
        dist[i : i + step, :k] = torch.topk(d, k, dim=1, largest=False, sorted=True).values.cpu().numpy()
    return {"keys": None, "dist": dist, "count": None, "status": None}

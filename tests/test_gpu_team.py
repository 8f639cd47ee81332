"""Team traversal (a block of warps per query) against the oracle: batches at
the edges of its rule (one query, two teams per SM, four per SM, one more), all
metrics and row kinds, lists of one and two 32-id chunks, walks that fill the
queue's far list, equal distances everywhere (small integers), deleted nodes,
a visited bitmap in global memory, and batches routed on the device. Keys,
distance bits, counts and statuses are equal (no tolerance)."""

import statistics
import struct
import time

import numpy as np
import pytest

import hnsw_gpu as H
import oracle as O
from conftest import build_index

pytestmark = pytest.mark.gpu


def assert_same(got, ref, what):
    np.testing.assert_array_equal(got[3], ref[3], err_msg=what)
    np.testing.assert_array_equal(got[2], ref[2], err_msg=what)
    for i in range(len(got[2])):
        c = int(got[2][i])
        np.testing.assert_array_equal(got[0][i, :c], ref[0][i, :c], err_msg=f"{what} query {i}")
        np.testing.assert_array_equal(got[1][i, :c].view(np.uint32), ref[1][i, :c].view(np.uint32), err_msg=what)


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize("dim,m,n", [(8, 4, 300), (100, 16, 4000), (40, 24, 3000), (33, 40, 2000)])
def test_team_walks(metric, dim, m, n):
    base, q = H.mixture(n, 300, dim, 20, 0.4, metric * 7 + dim)
    if dim == 8:  # ties
        base, q = np.round(base * 2), np.round(q * 2)
        base[:, 0] += 10
        q[:, 0] += 10
    if metric == 2:
        base[:, 0] += 2
        q[:, 0] += 2
    rng = np.random.default_rng(n + metric)
    deleted = rng.choice(n, n // 20, replace=False) if dim != 100 else ()
    data = build_index(base, metric=metric, m=m, ef_construction=60, quantize=True, deleted_keys=deleted)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    for nq, k, ef in ((1, 1, 1), (3, 10, 16), (296, 10, 64), (200, 100, 300)):
        what = f"nq={nq} k={k} ef={ef}"
        assert_same(gi.search_arrays(q[:nq], k, ef), oi.search(q[:nq], k, ef), what)
        assert_same(gi.search_arrays(q[:nq], k, ef, quantized=True, mode=1),
                    oi.search(q[:nq], k, ef, quantized=True), what + " int8")
        for sel in (0.01, 0.2):
            bits = H.key_bitmap(np.nonzero(rng.random(n) < sel)[0].astype(np.uint64), n)
            kw = dict(filter_bits=bits, filter_nbits=n)
            assert_same(gi.search_arrays(q[:nq], k, ef, mode=nq & 1, **kw), oi.search(q[:nq], k, ef, **kw),
                        what + f" filter {sel}")


@pytest.mark.parametrize("nq", [297, 592, 593])
def test_team_batches_around_the_rule(nq):
    base, q = H.gaussian(5000, 593, 32, 3)
    data = build_index(base, ef_construction=60)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    assert_same(gi.search_arrays(q[:nq], 10, 48), oi.search(q[:nq], 10, 48), f"nq={nq}")


@pytest.mark.parametrize("ef", [32, 200])
def test_team_retry_of_queries_that_outgrow_a_warp(ef):
    """Plain warps whose visited hash fills (2048 slots at ef = 32, 16,384 at
    200) hand the query to the teams' retry pass."""
    base, q = H.gaussian(30000, 700, 64, 9)
    b = H.IndexBuilder(64, H.Metric.L2, H.HnswParams(m=32, ef_construction=60, seed=7))
    b.insert_batch_gpu(np.arange(30000, dtype=np.uint64), base)
    data = b.to_bytes()
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    gi.set_counters(True)
    got = gi.search_arrays(q, 10, ef, mode=0)
    if ef == 32:
        assert gi.read_counters(700)[:, 0].max() > 1536
    assert_same(got, oi.search(q, 10, ef), f"ef={ef}")


@pytest.mark.parametrize("quantized", [False, True])
def test_plain_filtered_batch_that_is_mostly_redone(quantized):
    """Plain warps hand every query that outgrows the visited hash (2048 slots
    at ef = 32) to the teams' retry pass: here more than teams are resident."""
    n, nq = 30000, 900
    base, q = H.mixture(n, nq, 24, 30, 0.4, 5)
    data = build_index(base, metric=1, ef_construction=60, quantize=True)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    rng = np.random.default_rng(8)
    words = (n + 63) // 64
    bank = np.stack([H.key_bitmap(np.nonzero(rng.random(n) < p)[0].astype(np.uint64), n) for p in (0.01, 0.02, 0.9)])
    ids = rng.integers(0, 3, nq).astype(np.uint32)
    kw = dict(filter_bits=bank, filter_nbits=n, filter_stride=words, filter_ids=ids, quantized=quantized, mode=0)
    gi.set_counters(True)
    got = gi.search_arrays(q, 10, 32, **kw)
    assert (gi.read_counters(nq)[:, 0] > 2048).sum() > 400
    ref = oi.search(q, 10, 32, filter_bits=bank[ids], filter_nbits=n, filter_stride=words, quantized=quantized)
    assert_same(got, ref, f"quantized={quantized}")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("sel", [0.02, 0.9])
def test_batches_routed_on_the_device(mode, sel):
    """Few long walks among short ones, and walks of like length."""
    n, nq = 6000, 900
    base, q = H.mixture(n, nq, 24, 30, 0.4, 5)
    data = build_index(base, metric=1, ef_construction=60, quantize=True)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    rng = np.random.default_rng(8)
    bits = H.key_bitmap(np.nonzero(rng.random(n) < sel)[0].astype(np.uint64), n)
    used = (np.arange(nq) % 50 == 0).astype(np.uint8) if sel < 0.1 else np.ones(nq, np.uint8)
    ks, efs = rng.choice([1, 10, 50], nq).astype(np.uint32), rng.choice([16, 64, 128], nq).astype(np.uint32)
    kw = dict(filter_bits=bits, filter_nbits=n, filter_used=used, ks=ks, efs=efs, quantized=True)
    assert_same(gi.search_arrays(q, 10, 16, mode=mode, **kw), oi.search(q, 10, 16, **kw), f"mode={mode} sel={sel}")


def test_sparse_keys_are_routed_like_dense_ones():
    """Keys far above the node count, one query in a hundred with a filter of
    90 %: the expected work is that of the same queries on dense keys. (Read
    below the node count the bitmap is empty, those queries seem to scan the
    index, and the batch goes to teams: 1.37 times the time; 1.04 now.)"""
    n, nq, first = 20000, 12000, 1 << 20
    base, q = H.mixture(n, nq, 32, 40, 0.4, 5)
    admitted = np.nonzero(np.random.default_rng(8).random(n) < 0.9)[0].astype(np.uint64)
    used = (np.arange(nq) % 100 == 0).astype(np.uint8)
    data = [build_index(base, ef_construction=60, keys=np.arange(n, dtype=np.uint64) + off, parallel=False)
            for off in (0, first)]
    calls, times = [], [[], []]
    for d, off in zip(data, (0, first)):
        gi = H.HnswIndex.from_bytes(d)
        kw = dict(filter_bits=H.key_bitmap(admitted + np.uint64(off), n + off), filter_nbits=n + off)
        calls.append((gi, dict(kw, filter_used=used)))
        kw["filter_used"] = used[:900]
        assert_same(gi.search_arrays(q[:900], 10, 64, **kw), O.Index(d).search(q[:900], 10, 64, **kw), f"from {off}")
    for _ in range(15):
        for (gi, kw), ts in zip(calls, times):
            t = time.perf_counter()
            got = gi.search_arrays(q, 10, 64, mode=1, **kw)
            ts.append(time.perf_counter() - t)
            assert (got[3] == 0).all()
    assert statistics.median(times[1]) < 1.2 * statistics.median(times[0])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nq", [297, 640, 700, 1500])
def test_batches_of_one_filter(nq, mode):
    """One filter and one ef for the batch: teams up to about 650 queries,
    one warp per query above."""
    n = 6000
    base, q = H.mixture(n, nq, 24, 30, 0.4, 5)
    data = build_index(base, ef_construction=60, quantize=True)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    for sel in (0.01, 0.9):
        bits = H.key_bitmap(np.nonzero(np.random.default_rng(8).random(n) < sel)[0].astype(np.uint64), n)
        kw = dict(filter_bits=bits, filter_nbits=n, quantized=sel > 0.5)
        assert_same(gi.search_arrays(q, 10, 48, mode=mode, **kw), oi.search(q, 10, 48, **kw), f"nq={nq} sel={sel}")


@pytest.mark.parametrize("nq,ef", [(400, 900), (900, 1024), (900, 1100)])
def test_plain_batches_of_few_resident_warps(nq, ef):
    """At ef near 1024 a plain warp's scratch leaves four warps per SM or
    fewer, which the route compares with two teams; above it no team fits."""
    n = 5000
    base, q = H.mixture(n, nq, 24, 30, 0.4, 5)
    data = build_index(base, metric=1, ef_construction=60)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    efs = np.random.default_rng(3).integers(ef - 200, ef + 1, nq).astype(np.uint32)
    assert_same(gi.search_arrays(q, 10, 16, mode=0, efs=efs), oi.search(q, 10, 16, efs=efs), f"nq={nq} ef={ef}")


def test_team_with_its_visited_bitmap_in_global_memory():
    n = 800_000
    base, q = H.mixture(n, 160, 4, 500, 0.3, 2)
    b = H.IndexBuilder(4, H.Metric.L2, H.HnswParams(m=4, ef_construction=16, seed=7))
    b.insert_batch_gpu(np.arange(n, dtype=np.uint64), base)
    data = b.to_bytes()
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    assert_same(gi.search_arrays(q, 10, 40), oi.search(q, 10, 40), "plain")
    bits = H.key_bitmap(np.arange(0, n, 3, dtype=np.uint64), n)
    kw = dict(filter_bits=bits, filter_nbits=n)
    assert_same(gi.search_arrays(q, 10, 40, **kw), oi.search(q, 10, 40, **kw), "filtered")


@pytest.mark.parametrize("quantized", [False, True])
def test_team_ties_at_the_worst_result_across_lists(quantized):
    """A few hundred distinct distances among 20,000 nodes: neighbors shared by
    the lists of one joint expansion tie with the worst result, so the order
    of the lists decides (whichever list marked the neighbor)."""
    rng = np.random.default_rng(12)
    base = rng.integers(-8, 9, (20000, 4)).astype(np.float32)
    q = rng.integers(-8, 9, (2368, 4)).astype(np.float32)
    data = build_index(base, m=16, ef_construction=60, quantize=True)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    for ef in (20, 64):
        ref = oi.search(q, 10, ef, quantized=quantized)
        for lo in range(0, len(q), 296):
            got = gi.search_arrays(q[lo:lo + 296], 10, ef, quantized=quantized)
            assert_same(got, tuple(x[lo:lo + 296] for x in ref), f"ef={ef} from {lo}")


def test_entries_beyond_the_counts_are_zero():
    """Rows that a call fills in part (an uneven k, a filter of few rows) keep
    nothing of an earlier call's of another shape."""
    base, q = H.mixture(3000, 400, 24, 20, 0.4, 5)
    gi = H.HnswIndex.from_bytes(build_index(base, m=8, ef_construction=40))
    few = H.key_bitmap(np.arange(0, 3000, 1000, dtype=np.uint64), 3000)
    kw = dict(filter_bits=few, filter_nbits=3000)
    for nq in (400, 40):
        gi.search_arrays(q, 20, 64)
        ks = (np.arange(nq) % 10 + 1).astype(np.uint32)
        for r in (gi.search_arrays(q[:nq], 10, 64, ks=ks), gi.search_arrays(q[:nq], 10, 64, **kw)):
            beyond = np.arange(r[0].shape[1])[None, :] >= r[2][:, None]
            assert beyond.any() and not r[0][beyond].any() and not r[1][beyond].any()



@pytest.mark.parametrize("nq,k", [(40, 20), (700, 200)])
def test_rows_of_any_call_are_zero_beyond_their_counts(nq, k):
    """k above the number of points, and an invalid query, in graph and
    brute-force searches of every precision, small results (one pinned copy)
    and large ones, after a call that filled every row."""
    base, q = H.mixture(3000, nq, 24, 20, 0.4, 5)
    few = 15
    gi = H.HnswIndex.from_bytes(build_index(base, m=8, ef_construction=40, deleted_keys=range(few, 3000)))
    live = H.HnswIndex.from_bytes(build_index(base, m=8, ef_construction=40))
    bf = H.BruteForceIndex(24, H.Metric.L2)
    bf.insert_batch(np.arange(few, dtype=np.uint64), base[:few])
    full = H.BruteForceIndex(24, H.Metric.L2)
    full.insert_batch(np.arange(3000, dtype=np.uint64), base)
    bad = q.copy()
    bad[nq // 2, 3] = np.nan

    def check(r):
        filled = np.where(r[3] == 0, r[2], 0)
        beyond = np.arange(r[0].shape[1])[None, :] >= filled[:, None]
        assert beyond.any() and not r[0][beyond].any() and not r[1][beyond].any()

    gi.search_arrays(q, few, 256)
    check(gi.search_arrays(q, k, 256))
    live.search_arrays(q, k, 256)
    check(live.search_arrays(bad, k, 256, raise_on_error=False))
    for precision in (H.Precision.FP32, H.Precision.BF16, H.Precision.BF16X3):
        bf.search_arrays(q[:nq // 2], few, precision)
        check(bf.search_arrays(q, k, precision))
        full.search_arrays(q, few, precision)
        check(full.search_arrays(bad, k, precision, raise_on_error=False))


@pytest.mark.parametrize("every", [1, 4])
def test_merges_of_ties_in_a_row(every):
    """A chain of 250 levels, each two points at one distance (x and -x), the
    first listing the next level: each merge is taken one by one and the next
    expansion empties the queue, more often than its array (128) is long."""
    levels, n = 250, 501
    x = [float(levels + 1)]
    lists = [[] for _ in range(n)]
    for i in range(levels):
        lists[max(2 * i - 1, 0)] = [2 * i + 1, 2 * i + 2]
        x += [float(levels - i), -float(levels - i)]
    head = bytearray(build_index(np.zeros((1, 1), np.float32), m=8, ef_construction=40)[:56])
    struct.pack_into("<II", head, 48, n, 0)
    body = (bytes(head) + np.arange(n, dtype="<u8").tobytes() + bytes(2 * n) + np.array(x, "<f4").tobytes()
            + b"".join(struct.pack(f"<I{len(a)}I", len(a), *a) for a in lists))
    data = body + struct.pack("<I", H.crc32(body))
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    q = np.zeros((1, 1), np.float32)
    kw = {}
    if every > 1:
        bits = H.key_bitmap(np.array([i for i in range(n) if i % every < 3], np.uint64), n)
        kw = dict(filter_bits=bits, filter_nbits=n)
    for ef in (1, 5):
        ref = oi.search(q, 1, ef, **kw)
        assert ref[0][0, 0] == 499 or every > 1
        assert_same(gi.search_arrays(q, 1, ef, **kw), ref, f"ef={ef} every={every}")


@pytest.mark.parametrize("sample", [1, 700])
def test_a_tuned_index_keeps_its_teams(sample):
    """Tuning picks the schedule of the one-warp kernels: one query of a tuned
    bucket still takes a team (0.46 of one warp's time at ef = 256; the
    limit of 1.25 times the untuned call lies between the two)."""
    base, q = H.gaussian(10_000, 700, 128, 42)
    data = build_index(base, ef_construction=100)
    tuned, untuned = H.HnswIndex.from_bytes(data), H.HnswIndex.from_bytes(data)
    want = O.Index(data).search(q[:1], 10, 256)
    best, trials = tuned.autotune(q[:sample], 10, 256, reps=3)
    if sample == 1:  # the heuristic's trial takes a team, the others a warp
        assert best["heuristic"]
        assert best["ms"] < 0.8 * min(t["ms"] for t in trials if not t["heuristic"])
    times = {tuned: [], untuned: []}
    for _ in range(40):
        for ix in times:
            t = time.perf_counter()
            got = ix.search_arrays(q[:1], 10, 256, mode=H.MODE_AUTO)
            times[ix].append(time.perf_counter() - t)
            assert_same(got, want, "tuned" if ix is tuned else "untuned")
    assert statistics.median(times[tuned]) < 1.25 * statistics.median(times[untuned])

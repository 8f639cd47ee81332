"""The one-warp traversal kernels on the batches that teams of warps take when
nothing is fixed (up to two or four queries per SM): a fixed schedule keeps
every search on the one-warp kernels and their own retry passes. And the
96-register kernels of large unfiltered batches for inner product, cosine and
int8. Keys, distance bits, counts and statuses equal the oracle's (no
tolerance)."""

import numpy as np
import pytest

import hnsw_gpu as H
import oracle as O
from conftest import build_index
from test_gpu_search import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cold", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_visited_hash_and_candidate_array_overflow(mode, cold):
    """Filters that cannot fill the results: the walk outgrows the visited hash
    and the candidate array (plain: retry kernel, persistent: spill areas)."""
    base, queries = H.gaussian(5000, 48, 16, 77)
    data = build_index(base, metric=0, m=8, seed=1)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    gi.set_schedule(ef_cap=64, cand_cap=160, hash_cap=2048, warps_per_block=4, cold=cold)
    keys = np.arange(5000, dtype=np.uint64)
    for accepted, k, ef in [(keys[keys % 200 == 11], 10, 32), (keys[keys % 7 == 0], 10, 32),
                            (keys[keys % 50 == 3], 25, 64)]:
        kw = dict(filter_bits=H.key_bitmap(accepted, 5000), filter_nbits=5000)
        assert_same(gi.search_arrays(queries, k, ef, mode=mode, **kw), oi.search(queries, k, ef, **kw),
                    f"filter of {accepted.size}")
    assert_same(gi.search_arrays(queries, 10, 40, mode=mode), oi.search(queries, 10, 40), "after spill")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("quant", [False, True])
def test_distance_ties(mode, quant):
    """Points with about 40 copies each: the tie list of the single-array
    kernel overflows. Its queries go to the retry kernel under a fixed
    schedule, and in a batch above the teams' size to the teams' retry pass."""
    rng = np.random.default_rng(11)
    base = rng.integers(0, 3, size=(3000, 4)).astype(np.float32)
    queries = np.vstack([rng.integers(0, 3, size=(150, 4)), rng.integers(-1, 4, size=(50, 4))]).astype(np.float32)
    data = build_index(base, metric=0, m=8, seed=3, quantize=quant)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    for k, ef in [(1, 1), (10, 16), (10, 40), (32, 64), (50, 200)]:
        ref = oi.search(queries, k, ef, quantized=quant)
        gi.set_schedule(ef_cap=256, hash_cap=8192, warps_per_block=2)
        assert_same(gi.search_arrays(queries, k, ef, mode=mode, quantized=quant), ref, f"fixed, k={k} ef={ef}")
        gi.set_schedule()
        got = gi.search_arrays(np.tile(queries, (4, 1)), k, ef, mode=mode, quantized=quant)
        assert_same(got, tuple(np.concatenate([x] * 4) for x in ref), f"800 queries, k={k} ef={ef}")


@pytest.mark.parametrize("mode", [0, 1])
def test_cold_candidate_list_at_the_heuristics_sizes(mode):
    """Filters so selective that ef results never fill, with the geometry that
    the heuristic picks at ef = 512 (cold lists in persistent mode)."""
    base, queries = H.mixture(20000, 48, 16, 40, 0.4, 31)
    data = build_index(base, metric=0, m=8, seed=5, deleted_keys=range(0, 20000, 97))
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    rng = np.random.default_rng(32)
    words = (20000 + 63) // 64
    bank = np.stack([H.key_bitmap(np.nonzero(rng.random(20000) < p)[0].astype(np.uint64), 20000)
                     for p in (0.0003, 0.002, 0.01, 0.05, 0.3)])
    ids = rng.integers(0, len(bank), 48).astype(np.uint32)
    ks = rng.choice([1, 10, 100], 48).astype(np.uint32)
    efs = rng.choice([16, 64, 256, 512], 48).astype(np.uint32)
    kw = dict(filter_nbits=20000, filter_stride=words, ks=ks, efs=efs)
    ref = oi.search(queries, 100, 16, filter_bits=bank[ids], **kw)
    gi.set_schedule(ef_cap=512, cand_cap=1056, hash_cap=16384 if mode else 32768, warps_per_block=1, cold=mode)
    got = gi.search_arrays(queries, 100, 16, filter_bits=bank, filter_ids=ids, mode=mode, **kw)
    assert_same(got, ref, f"mode={mode}")


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("metric,quantized", [(1, False), (2, False), (0, True), (1, True)])
def test_large_batches_take_the_lean_kernels(metric, quantized, mode):
    """More than 32 queries per SM and scratch for more than 16 warps per SM:
    the 96-register kernels, for inner product, cosine and int8 rows."""
    base, q = H.mixture(4000, 5000, 24, 30, 0.5, 21)
    if metric == 2:
        base[:, 0] += 2.0
        q[:, 0] += 2.0
    data = build_index(base, metric=metric, m=8, seed=5, quantize=quantized)
    gi, oi = H.HnswIndex.from_bytes(data), O.Index(data)
    for nq, ef in ((5000, 32), (4740, 48)):
        got = gi.search_arrays(q[:nq], 10, ef, mode=mode, quantized=quantized)
        assert_same(got, oi.search(q[:nq], 10, ef, quantized=quantized), f"nq={nq} ef={ef}")

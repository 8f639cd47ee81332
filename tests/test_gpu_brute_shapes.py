"""GPU exact brute force at the edges of its tile shapes: batch sizes around
every shape's query count, row counts around its row tile, dimensions around
the 32-column steps and copy chunks, k around the 32-entry merges, the shared
lists' limit and n; keys in descending order, so that ties are broken by key
and not by row. Bit-identical to the oracle (no tolerance)."""

import numpy as np
import pytest

import hnsw_gpu as H
import oracle as O

pytestmark = pytest.mark.gpu


def _data(n, nq, dim, seed, metric):
    rng = np.random.default_rng(seed)
    # Small integers: many exact ties, broken by key.
    base = rng.integers(-2, 3, (n, dim)).astype(np.float32)
    queries = rng.integers(-2, 3, (nq, dim)).astype(np.float32)
    if metric == 2:
        base[:, 0] += 3.0
        queries[:, 0] += 3.0
    base[: n // 2] += rng.standard_normal((n // 2, dim)).astype(np.float32)
    return base, queries


@pytest.mark.parametrize("metric", [0, 1, 2])
@pytest.mark.parametrize(
    "n,nq,dim,k",
    [
        (1, 1, 1, 3), (7, 2, 31, 7), (127, 1, 32, 10), (128, 2, 33, 33), (129, 3, 40, 128),
        (300, 8, 64, 129), (65, 9, 100, 5), (1000, 16, 128, 32), (1025, 17, 129, 31),
        (2049, 32, 7, 64), (5003, 33, 260, 1), (3000, 64, 96, 300), (4000, 5, 768, 127), (20011, 1, 72, 1024),
    ],
)
def test_brute_shapes(metric, n, nq, dim, k):
    base, queries = _data(n, nq, dim, 1000 * n + dim, metric)
    keys = (np.arange(n, dtype=np.uint64) * 5 + 2)[::-1].copy()
    index = H.BruteForceIndex(dim, H.Metric(metric))
    index.insert_batch(keys, base)
    prepared = base if metric != 2 else O.normalize_rows(base)
    bits = H.key_bitmap(keys[np.random.default_rng(n).random(n) < 0.4], int(keys.max()) + 1)
    for got, ref in (
        (index.search_arrays(queries, k), O.brute(metric, prepared, queries, k, keys=keys)),
        (index.search_arrays(queries, k, filter_bits=bits, filter_nbits=int(keys.max()) + 1),
         O.brute_filtered(metric, prepared, queries, k, bits, int(keys.max()) + 1, keys=keys)),
    ):
        np.testing.assert_array_equal(got[3], ref[3])
        np.testing.assert_array_equal(got[2], ref[2])
        for i in range(nq):
            c = int(got[2][i])
            np.testing.assert_array_equal(got[0][i, :c], ref[0][i, :c])
            np.testing.assert_array_equal(got[1][i, :c].view(np.uint32), ref[1][i, :c].view(np.uint32))

"""CPU model of the team traversal's layer 0 (team_query in
hnsw-index_b200/csrc/search_team.cu) against a direct restatement of the
reference's search_layer (src/hnsw/search.rs:81-142) with its two heaps and an
admission rule.

The model keeps the kernel's structures: the candidate array C with its live
range [head, tail), the far list beyond C's capacity with its smallest entry,
the results, joint expansions of the leading candidates, and the one-by-one
merge of a batch whose equal distances reach the worst result. Distances are
few, so most of them tie. It must expand the same number of nodes and return
the same results as the sequential walk."""

import bisect
import heapq

import numpy as np

LISTS = 8


def reference_walk(adj, dist, admitted, entry, ef):
    visited = {entry}
    cand = [(dist[entry], entry)]
    res = [(-dist[entry], -entry)] if admitted[entry] else []
    expanded = 0
    while cand:
        d, c = heapq.heappop(cand)
        if len(res) >= ef and d > -res[0][0]:
            break
        expanded += 1
        for n in adj[c]:
            if n in visited:
                continue
            visited.add(n)
            if len(res) < ef or dist[n] < -res[0][0]:
                heapq.heappush(cand, (dist[n], n))
                if admitted[n]:
                    heapq.heappush(res, (-dist[n], -n))
                    if len(res) > ef:
                        heapq.heappop(res)
    return sorted((-a, -b) for a, b in res), expanded


def team_walk(adj, dist, admitted, entry, ef, cap, rng, stats):
    """None when an array is used out of its range."""
    visited = {entry}
    C, head = [(dist[entry], entry)], 0  # C[head:] is live
    far = []
    R = [C[0]] if admitted[entry] else []
    expanded = 0
    while True:
        worst = R[-1][0] if len(R) >= ef else np.inf
        live = C[head:]
        if not live:
            far = [x for x in far if x[0] <= worst]
            if not far:
                break
            far.sort()
            C, head, far = far[:cap], 0, far[cap:]
            continue
        if live[0][0] > worst:
            break
        # Leading candidates; how many have been fetched varies.
        lead = live[:int(rng.integers(1, LISTS + 1))]
        opened = [[n for n in adj[c] if n not in visited] for _, c in lead]
        j, pm, A = 0, np.inf, 0
        for i, (d, _) in enumerate(lead):
            if i:
                ok = d < pm
                if len(R) + A >= ef:
                    ok = ok and A < ef and d <= R[ef - 1 - A][0]
                if not ok:
                    break
            imp = [n for n in opened[i] if dist[n] < worst]
            pm = min([pm] + [dist[n] for n in opened[i]])
            A += sum(admitted[n] for n in imp)
            j += 1
        seq = [(dist[n], n) for o in opened[:j] for n in o if dist[n] < worst]
        visited.update(n for o in opened[:j] for n in o)
        expanded += j
        head += j
        if not seq:
            continue
        new = sorted(set(seq))
        adm = [x for x in new if admitted[x[1]]]
        fmin = min(far) if far else (np.inf, 0)
        R2 = sorted(R + adm)[:ef]
        dists = [x[0] for x in new] + [x[0] for x in R]
        ties = [x[0] for x in new if dists.count(x[0]) > 1]
        if not (ties and len(R) + len(adm) >= ef and max(ties) >= R2[ef - 1][0]):
            merged = sorted(C[head:] + [x for x in new if x <= fmin])
            far += [x for x in merged[cap:] + [x for x in new if x > fmin] if x[0] <= worst]
            C, head, R = merged[:cap], 0, R2
            continue
        stats["one_by_one"] = stats.get("one_by_one", 0) + 1
        # As in the kernel: the live range moves to the start of C first.
        C, head = C[head:], 0
        seen = set()
        for x in seq:
            if x in seen:
                continue
            seen.add(x)
            if len(R) >= ef and not x[0] < R[-1][0]:
                continue
            fm = min(far) if far else None
            if fm is not None and x > fm:
                far.append(x)
            elif len(C) >= cap:
                if len(C) <= head:
                    return None  # nothing live to move out
                last = C.pop()
                far.append(max(x, last))
                bisect.insort(C, min(x, last), lo=head)
                stats["evicted"] = stats.get("evicted", 0) + 1
            else:
                bisect.insort(C, x, lo=head)
            if admitted[x[1]]:
                bisect.insort(R, x)
                del R[ef:]
    return R, expanded


def random_case(rng):
    n = int(rng.integers(2, 250))
    m0 = int(rng.integers(1, 25))
    values = rng.integers(0, int(rng.integers(2, 40)), size=n) * 0.5
    adj = []
    for v in range(n):
        deg = int(rng.integers(0, min(m0, n - 1) + 1))
        adj.append([int(x) for x in rng.choice(np.delete(np.arange(n), v), size=deg, replace=False)])
    admitted = rng.random(n) < rng.choice([0.03, 0.2, 0.7, 1.0])
    return adj, [float(x) for x in values], admitted, int(rng.integers(0, n)), int(rng.integers(1, 24))


def test_team_walk_equals_two_heap_walk():
    rng = np.random.default_rng(31)
    stats = {}
    for _ in range(2500):
        adj, dist, admitted, entry, ef = random_case(rng)
        want = reference_walk(adj, dist, admitted, entry, ef)
        for cap in (2, 7, 64):
            got = team_walk(adj, dist, admitted, entry, ef, cap, rng, stats)
            assert got is not None, "array out of its range"
            assert got[1] == want[1], "expansions differ"
            assert got[0] == want[0], "results differ"
    assert stats["one_by_one"] > 1000 and stats["evicted"] > 100


def test_merges_of_ties_in_a_row_do_not_run_the_queue_out_of_its_array():
    """A chain of levels, each two nodes at one distance: every merge is taken
    one by one and leaves C empty after the next expansion, 250 times in a row
    with an array of 128 (tests/test_gpu_team.py runs the same chain)."""
    levels = 250
    dist = [float((levels + 1) ** 2)]
    adj = [[] for _ in range(2 * levels + 1)]
    for i in range(levels):
        adj[max(2 * i - 1, 0)] = [2 * i + 1, 2 * i + 2]
        dist += [float((levels - i) ** 2)] * 2
    for admitted in ([True] * len(dist), [i % 4 < 3 for i in range(len(dist))]):
        want = reference_walk(adj, dist, admitted, 0, 1)
        stats = {}
        assert team_walk(adj, dist, admitted, 0, 1, 128, np.random.default_rng(1), stats) == want
        assert want[1] >= levels + 1 and stats["one_by_one"] > 120

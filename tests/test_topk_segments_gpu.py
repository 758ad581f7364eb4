"""Segments of the visit tables a launch ranks: one query at a time (plain) and
a batch, tables on either side of the register path's limits (lists that one
CTA can merge, 296 segments)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(cuda_device):
    import graphwalker_b200 as gw
    with gw.Graph.rmat(18, 16, seed=4, blocksize_kb=4096) as G:
        rowptr, _ = G.export_csr()
        yield G, np.random.default_rng(4).choice(np.flatnonzero(np.diff(rowptr) > 0), 8).astype(np.uint32)


# slots: 8 a walk, rounded up to a power of two.  k = 500: 33 segments of 8192
# are merged past the registers; k = 60: 273; any k: 297 (512 segments here).
@pytest.mark.parametrize("k", [1, 60, 500, 512])
@pytest.mark.parametrize("budgets", [[300], [32_768, 32_769], [131_073, 0, 5, 262_145], [300_000] * 3])
def test_plain_and_batched_lists_are_the_same(graph, k, budgets):
    import graphwalker_b200 as gw
    G, sources = graph
    p = gw.params(gw.RULE_PPR, gw.SINK_NONE, 12, seed=6)
    b = np.array(budgets, np.uint32)
    ids, counts, _ = G.ppr(p, sources[: len(b)], b, k, batched=True)
    pids, pcounts, _ = G.ppr(p, sources[: len(b)], b, k, batched=False)
    assert np.array_equal(ids, pids) and np.array_equal(counts, pcounts)


def test_a_plain_query_is_ranked_as_fast_as_a_batch_of_one(graph):
    """300,000 walks, k = 500: twice the segments, and so twice the keys in the
    one CTA that merges them, made the plain call 12 % slower."""
    import graphwalker_b200 as gw
    G, sources = graph
    p = gw.params(gw.RULE_PPR, gw.SINK_NONE, 12, seed=6)
    b = np.full(8, 300_000, np.uint32)
    best = {}
    for _ in range(12):
        for batched in (False, True):
            t = time.perf_counter()
            for q in (slice(0, 8),) if not batched else [slice(i, i + 1) for i in range(8)]:
                G.ppr(p, sources[q], b[q], 500, batched=batched)
            best[batched] = min(best.get(batched, 1e9), time.perf_counter() - t)
    assert best[False] < 1.05 * best[True]

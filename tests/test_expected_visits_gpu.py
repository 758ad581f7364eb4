"""gw_expected_visits over rows without edges, against the FP64 power series.

Tolerances: both sides add the same non-negative FP64 terms in another order,
at most 2^17 of them a sum and L hops deep, so a value differs by less than
L * 2^17 * 2^-53 = 7.3e-10 of itself; 1e-9 is allowed."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(nv: int, at, degree: int, seed: int):
    deg = np.zeros(nv, np.int64)
    deg[at] = degree
    rp = np.zeros(nv + 1, np.uint64)
    rp[1:] = np.cumsum(deg)
    ci = np.random.default_rng(seed).choice(at, int(rp[-1])).astype(np.uint32)
    return rp, ci, np.array([0, nv], np.uint32)


@pytest.mark.parametrize("L", [4, 50], ids=["pushed", "pulled"])
@pytest.mark.parametrize("nv,at", [(1, [0]), (33, [0, 32]), (1025, [0, 31, 32, 1023, 1024]), (40_000, [5, 39_999]),
                                   (70_001, [0, 1, 33_000, 65_569, 70_000]), (40_000, list(range(0, 40_000, 997)))])
@pytest.mark.parametrize("degree", [1, 129])
def test_rows_without_edges_are_stepped_over(cuda_device, oracle, nv, at, degree, L):
    import graphwalker_b200 as gw
    rp, ci, blocks = _rows(nv, np.array(at), degree, nv)
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        for rule in (gw.RULE_PPR, gw.RULE_JUMP):
            got = G.expected_visits(gw.params(rule, gw.SINK_NONE, L), at[0])
            ref = oracle.expected_visits(rp, ci, at[0], rule, L)
            assert np.allclose(got, ref, rtol=1e-9, atol=0)


@pytest.mark.parametrize("L", [6, 50], ids=["pushed", "pulled"])
def test_a_long_gap_costs_its_logarithm(cuda_device, L):
    """150 edges at either end of four million vertices.  A warp that crosses the
    gap 32 rows at a time takes 131,072 dependent steps a hop, over 25 ms; the
    whole call, its 32 MB of results included, is allowed 60 ms."""
    import graphwalker_b200 as gw
    nv = 1 << 22
    at = np.r_[np.arange(50), np.arange(nv - 50, nv)]
    rp, ci, blocks = _rows(nv, at, 3, 1)
    p = gw.params(gw.RULE_PPR, gw.SINK_NONE, L)
    took = []
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        for _ in range(5):
            t = time.perf_counter()
            visits = G.expected_visits(p, 3)
            took.append(time.perf_counter() - t)
    assert visits[at].sum() == pytest.approx(visits.sum()) and visits[3] > 0
    assert min(took) < 0.06


@pytest.mark.parametrize("edges", ["hub", "runs", "one short"])
@pytest.mark.parametrize("rule,L", [(0, 8), (1, 9), (3, 9), (4, 8), (4, 12)])
def test_pulled_edge_runs(cuda_device, oracle, edges, rule, L):
    """Graphs just large enough to be turned around (2^17 edges) and one edge
    short of it: a hub whose row fills many runs between long empty stretches,
    rows of 127 to 129 edges, edges to every row and to a few.  As many terms a
    sum as edges and vertices, so that times 2^-53 and L bounds the error."""
    import graphwalker_b200 as gw
    nv, n = 3000, (1 << 17) - (edges == "one short")
    r = np.random.default_rng(L)
    deg = np.zeros(nv, np.int64)
    if edges == "runs":
        deg[700:2300:2] = r.choice([127, 128, 129], 800)
        deg[2900] = n - deg.sum()
    else:
        deg[[3, 700, 1500, nv - 1]] = n - 70_000, 69_000, 993, 7
    rp = np.r_[0, np.cumsum(deg)].astype(np.uint64)
    assert rp[-1] == n
    ci = r.integers(0, nv if edges == "runs" else 40, n).astype(np.uint32)
    ci[::97] = 700  # some walks come back to a vertex with edges
    with gw.Graph.from_csr(rp, ci, np.array([0, nv], np.uint32)) as G:
        for src in (700, 701):
            for _ in range(2):  # again, in the workspace the first call left
                got = G.expected_visits(gw.params(rule, gw.SINK_NONE, L), src)
            ref = oracle.expected_visits(rp, ci, src, rule, L)
            assert np.allclose(got, ref, rtol=L * (n + nv) * 2.0 ** -53, atol=0)


def test_few_hops_over_a_large_graph_are_pushed(cuda_device):
    """Seven hops from a vertex of degree 1 at R-MAT scale 24 (268 M edges) cost
    about one push more than six, not the turning around of the graph, which
    took 38 ms beside the call's 33."""
    import graphwalker_b200 as gw
    best = {}
    with gw.Graph.rmat(24, 16, seed=1, blocksize_kb=1 << 16) as G:
        G.set_edge_records(gw.EDGE_RECORDS_OFF)
        rowptr, _ = G.export_csr()
        source = int(np.flatnonzero(np.diff(rowptr) == 1)[0])
        for L in (6, 7) * 6:
            t = time.perf_counter()
            G.expected_visits(gw.params(gw.RULE_PPR, gw.SINK_NONE, L), source)
            best[L] = min(best.get(L, 1e9), time.perf_counter() - t)
    assert best[7] < 1.6 * best[6]

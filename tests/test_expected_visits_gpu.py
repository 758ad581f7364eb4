"""gw_expected_visits over rows without edges, against the FP64 power series.

Tolerances: both sides add the same non-negative FP64 terms in another order,
at most 2^17 of them a sum and L hops deep, so a value differs by less than
L * 2^17 * 2^-53 = 3e-10 of itself; 1e-9 is allowed."""
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


@pytest.mark.parametrize("L", [4, 20], ids=["pushed", "pulled"])
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


@pytest.mark.parametrize("L", [6, 24], ids=["pushed", "pulled"])
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

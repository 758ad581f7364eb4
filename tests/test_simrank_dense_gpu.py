"""SimRank's join where walks coincide: positions at which most of a tile's
walks stand on common vertices are compared pair by pair, in tiles of every
size, next to sparse positions.  Counts equal the oracle's."""
import time

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.uint32).view(np.int32)).cuda()


@pytest.mark.parametrize("R,L", [(3500, 12), (3457, 25), (4097, 9)])
@pytest.mark.parametrize("vertices", [[2], [3, 10**6, 2, 10**6], [10**6, 40, 40, 40, 40, 40, 10**6], [60, 90, 130, 200]])
def test_dense_and_sparse_positions(cuda_device, oracle, R, L, vertices):
    """Positions that turn from sparse to dense and back at any of the four
    positions a look is good for; around the share of candidates (half a tile)
    where the comparison turns; walks that have ended."""
    import graphwalker_b200 as gw
    assert R * R >= 6_000_000  # joined
    rng = np.random.default_rng(R + L)
    pa, pb = (np.stack([rng.integers(0, vertices[p % len(vertices)], R) for p in range(L)], 1).astype(np.uint32)
              for _ in range(2))
    for p in (pa, pb):
        p[np.arange(L) >= rng.integers(1, 2 * L, R)[:, None]] = 0xFFFFFFFF
    _, ref = oracle.simrank(pa, pb, R, L)
    g = load_golden("hand")
    with gw.Graph.from_csr(g["rowptr"], g["colidx"], g["blocks"]) as G:
        assert np.array_equal(G.simrank_meet(_dev(pa), _dev(pb), R, L), ref)


@pytest.mark.parametrize("nq,R,L", [(600, 100, 30), (600, 200, 30), (592, 300, 11), (13, 1000, 11), (2000, 100, 7), (64, 1000, 11),
                                     (40, 500, 140)])
@pytest.mark.parametrize("nv", [3, 24, 150])
def test_batches_on_small_graphs(cuda_device, oracle, nq, R, L, nv):
    """Tiles of 128, 256 and 512 walks, partly filled, on graphs whose walks
    meet everywhere."""
    import graphwalker_b200 as gw
    assert nq * R * R >= 6_000_000  # joined
    rng = np.random.default_rng(nv)
    rp = (np.arange(nv + 1) * 8).astype(np.uint64)
    ci = rng.integers(0, nv, nv * 8).astype(np.uint32)
    a, b = rng.integers(0, nv, (2, nq)).astype(np.uint32)
    with gw.Graph.from_csr(rp, ci, oracle.compute_blocks(rp, 1)) as G:
        _, meet = G.simrank_batch(a, b, R, L, seed=9)
    walks, refs = {}, {}
    for q in range(min(nq, 40)):
        for v in (int(a[q]), int(b[q])):
            c = np.full(R, v, np.uint32)
            if v not in walks:
                walks[v] = oracle.run_walks(rp, ci, c, ids=c, src=c, hop0=(np.arange(R) * L).astype(np.uint32), rule=3,
                                            L=L, seed=9, stride=L, counts=False)["paths"]
        key = int(a[q]), int(b[q])
        if key not in refs:
            refs[key] = oracle.simrank(walks[key[0]], walks[key[1]], R, L)[1]
        assert np.array_equal(meet[q], refs[key]), q


@pytest.mark.parametrize("shorter,R,L", [(3490, 3500, 11), (990, 1000, 135)], ids=["dense", "long"])
def test_a_few_walks_more_cost_little(cuda_device, shorter, R, L):
    """Walks on 16 vertices, just short of and just past 2^27 comparisons, from
    where on they were joined a candidate at a time: a query of 3500 walks took
    1.15 times one of 3490, one of 1000 long walks 4.7 times one of 990."""
    import graphwalker_b200 as gw
    nv = 16
    rng = np.random.default_rng(1)
    rp = (np.arange(nv + 1) * 8).astype(np.uint64)
    best = {}
    with gw.Graph.from_csr(rp, rng.integers(0, nv, nv * 8).astype(np.uint32), np.array([0, nv], np.uint32)) as G:
        pa, pb = (_dev(rng.integers(0, nv, (R, L))) for _ in range(2))
        for _ in range(30):
            for n in (shorter, R):
                t = time.perf_counter()
                G.simrank_meet(pa, pb, n, L)
                best[n] = min(best.get(n, 1e9), time.perf_counter() - t)
    assert best[R] < 1.1 * best[shorter]

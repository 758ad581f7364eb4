"""The superstep's tiles at their edges: one walk, one short of, exactly and one
past a row of 256; tiles of several rows (past 148 x 8 x 256 walks in a pool);
blocks searched in shared memory (few) and in global memory (over 2048).  The
pools and counts after a few supersteps equal the oracle's block loop, record
for record (whole numbers: no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,kb,n,L", [(10, 40, 1, 10), (10, 40, 255, 10), (10, 40, 256, 3), (10, 40, 257, 10),
                                          (12, 160, 700_003, 6), (16, 1, 4097, 8)])
@pytest.mark.parametrize("rule", [0, 3], ids=["jump", "restart"])
def test_superstep_tiles(cuda_device, oracle, scale, kb, n, L, rule):
    import graphwalker_b200 as gw
    rp, ci = oracle.rmat_csr(scale, 16, seed=7)
    blocks = oracle.compute_blocks(rp, kb)
    assert (len(blocks) - 1 > 2048) == (scale == 16)
    r = np.random.default_rng(n)
    cur = r.integers(0, len(rp) - 1, n).astype(np.uint32)
    cur = cur[np.argsort(np.searchsorted(blocks[1:], cur, side="right"), kind="stable")]
    ids = np.arange(n, dtype=np.uint32)
    for steps in (1, 4):
        ref = oracle.block_engine(rp, ci, blocks, cur, rule=rule, L=L, ids=ids, seed=11, prob=0.0, max_supersteps=steps)
        with gw.Graph.from_csr(rp, ci, blocks) as G:
            for _ in range(2):  # a second run in the pools the first one left
                G.walks_clear()
                G.add_walks_at(cur, ids=ids)
                st = G.run(gw.params(rule, gw.SINK_VERTEX_COUNT, L, seed=11, mode=gw.MODE_BLOCKED, prob=0.0,
                                     max_supersteps=steps))
                assert st.supersteps == ref["supersteps"]
                assert np.array_equal(G.read_counts(), ref["counts"])
                for b in range(G.nblocks):
                    want = ref["pools"][b]
                    assert np.array_equal(G.read_pool(b), np.stack(want, axis=1) if len(want[0])
                                          else np.zeros((0, 4), np.uint32)), f"block {b}"

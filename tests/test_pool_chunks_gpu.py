"""gw_run_pools at the sizes where its chunks turn: exactly the first chunk of
2^17 walk words and one more, and a set whose chunks reach an eighth of it;
walks with ids of their own.  Counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1 << 17, (1 << 17) + 1, 1_300_001])
def test_run_pools_chunks(cuda_device, oracle, n):
    import graphwalker_b200 as gw
    rp, ci = oracle.rmat_csr(14, 8, seed=12)
    cur = np.sort(np.random.default_rng(n).integers(0, len(rp) - 1, n))
    ids = np.arange(n, dtype=np.uint32)[::-1].copy()
    ref = oracle.run_walks(rp, ci, cur.astype(np.uint32), ids=ids, src=cur.astype(np.uint32), rule=0, L=6, seed=2)
    with gw.Graph.from_csr(rp, ci, oracle.compute_blocks(rp, 64)) as G:
        blk = np.searchsorted(G.blocks[1:], cur, side="right")
        words = gw.encode(cur, cur - G.blocks[blk].astype(np.int64), 0)
        offs = np.r_[0, np.cumsum(np.bincount(blk, minlength=G.nblocks))].astype(np.uint64)
        out = np.zeros(G.nv, np.uint32)
        for _ in range(2):
            G.run_pools(gw.params(0, gw.SINK_VERTEX_COUNT, 6, seed=2), words, offs, out, ids=ids)
            assert np.array_equal(out, ref["counts"])

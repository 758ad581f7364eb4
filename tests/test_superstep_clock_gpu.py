"""The device times of a blocked run's statistics cover what they name."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_partition_time_covers_the_whole_scatter(cuda_device):
    """16.8 M walks move from one block to the other: their scatter reads 16
    bytes of walk and 4 of destination and writes 16, 604 MB, which take 75 us
    at 8 TB/s.  It is thousands of CTAs in many waves; the first of them is done
    long before."""
    import graphwalker_b200 as gw
    per, n = 1024, 1 << 24
    rp = (np.arange(2 * per + 1) * 2).astype(np.uint64)
    ci = np.random.default_rng(1).integers(per, 2 * per, 4 * per).astype(np.uint32)
    blocks = np.array([0, per, 2 * per], np.uint32)
    cur = np.sort(np.random.default_rng(2).integers(0, per, n).astype(np.uint32))
    p = gw.params(gw.RULE_STOP, gw.SINK_VERTEX_COUNT, 6, mode=gw.MODE_BLOCKED, jump_prob=0.0, prob=0.0,
                  max_supersteps=1)
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        G.add_walks_at(cur)
        for _ in range(3):
            st = G.run(p)
            assert st.supersteps == 1 and len(G.read_pool(1)) == n
            assert st.ms_partition > 0.075
            assert st.ms_walk + st.ms_partition <= st.ms_total

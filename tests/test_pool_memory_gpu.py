"""Device memory of the block loop's walk pools: they take no more than their
walks where the rest of a run needs the room, give way to it, and grow when a
superstep moves more walks to a block than its pool holds.  Counts and pools
equal the oracle's (whole numbers: no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _inside_blocks(nblocks: int, per_block: int, degree: int, seed: int = 3):
    """A graph whose edges stay inside their block."""
    r = np.random.default_rng(seed)
    nv = nblocks * per_block
    base = np.repeat(np.arange(nblocks, dtype=np.uint32) * per_block, per_block * degree)
    ci = base + r.integers(0, per_block, nv * degree, dtype=np.uint32)
    return (np.arange(nv + 1) * degree).astype(np.uint64), ci, (np.arange(nblocks + 1) * per_block).astype(np.uint32)


def test_streamed_run_fits_beside_its_slots(cuda_device, oracle):
    """8.4 M walks (128 MB) that never leave their blocks and two 40 MB slots:
    240 MB of buffers, 290 MB of device memory.  With room for twice the walks
    taken first the slots would not fit any more."""
    import torch

    import graphwalker_b200 as gw
    p = gw.params(gw.RULE_STOP, gw.SINK_VERTEX_COUNT, 3, seed=9, mode=gw.MODE_BLOCKED)
    rp, ci, blocks = _inside_blocks(8, 64, 4)  # loads the kernels
    with gw.Graph.from_csr(rp, ci, blocks, residency=gw.STREAM_PINNED) as G:
        G.set_mapped_block_walks(0)
        G.add_walks_at(np.arange(G.nv, dtype=np.uint32))
        G.run(p)
    rp, ci, blocks = _inside_blocks(8, 4096, 2560)
    n = 8 << 20
    cur = np.sort(np.random.default_rng(1).integers(0, len(rp) - 1, n).astype(np.uint32))
    with gw.Graph.from_csr(rp, ci, blocks, residency=gw.STREAM_PINNED) as G:
        G.set_mapped_block_walks(0)
        G.add_walks_at(cur)
        torch.cuda.empty_cache()
        held = [torch.empty(max(0, torch.cuda.mem_get_info()[0] - 290 * MB), dtype=torch.uint8, device="cuda")]
        try:
            assert torch.cuda.mem_get_info()[0] <= 290 * MB
            G.run(p)
        finally:
            held.clear()
            torch.cuda.empty_cache()
        counts = G.read_counts()
    assert np.array_equal(counts, oracle.run_walks(rp, ci, cur, rule=1, L=3, seed=9)["counts"])


def test_pools_of_an_earlier_run_give_way(cuda_device, oracle):
    """The first allocation after a run fails once: the pools it left go back
    and the next run is made all the same."""
    import graphwalker_b200 as gw
    rp, ci = oracle.rmat_csr(11, 8, seed=5)
    blocks = oracle.compute_blocks(rp, 8)
    cur = np.arange(len(rp) - 1, dtype=np.uint32)
    p = gw.params(gw.RULE_JUMP, gw.SINK_VERTEX_COUNT, 10, seed=5, mode=gw.MODE_BLOCKED)
    ref = oracle.run_walks(rp, ci, cur, rule=0, L=10, seed=5)["counts"]
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        G.add_walks_at(cur)
        G.run(p)
        G.set_residency(gw.STREAM_PINNED, 3)
        G.set_mapped_block_walks(0)
        gw.inject_fault(gw.FAULT_DEVICE_ALLOC, 0)  # the first slot
        try:
            st = G.run(p)
        finally:
            gw.inject_fault(gw.FAULT_NONE)
        assert st.block_loads > 0
        assert np.array_equal(G.read_counts(), ref)
        G.run(p)
        assert np.array_equal(G.read_counts(), ref)


@pytest.mark.parametrize("nblocks", [5, 8, 33])
@pytest.mark.parametrize("budget", [0, 64 << 10])
def test_outgrown_pools(cuda_device, oracle, nblocks, budget):
    """Every walk moves to the last block, whose pool has room for an even
    share of them: after a few supersteps it holds several shares, in order."""
    import graphwalker_b200 as gw
    per, n = 64, 40_000
    nv = nblocks * per
    r = np.random.default_rng(nblocks)
    ci = r.integers(nv - per, nv, nv * 3).astype(np.uint32)
    ci[(nv - per) * 3:] = r.integers(0, nv, per * 3)
    rp = (np.arange(nv + 1) * 3).astype(np.uint64)
    blocks = (np.arange(nblocks + 1) * per).astype(np.uint32)
    cur = np.sort(r.integers(0, nv - per, n).astype(np.uint32))
    ids = np.arange(n, dtype=np.uint32)
    grown = False
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        G.set_pool_budget(budget)
        for steps in (1, 2, nblocks - 1, nblocks + 3):
            ref = oracle.block_engine(rp, ci, blocks, cur, rule=1, L=9, ids=ids, seed=11, prob=0.0,
                                      max_supersteps=steps)
            grown = grown or len(ref["pools"][-1][0]) > n // nblocks + 1024
            for _ in range(2):  # a second run in the pools the first one left
                G.walks_clear()
                G.add_walks_at(cur, ids=ids)
                st = G.run(gw.params(gw.RULE_STOP, gw.SINK_VERTEX_COUNT, 9, seed=11, mode=gw.MODE_BLOCKED, prob=0.0,
                                     max_supersteps=steps))
                assert st.supersteps == ref["supersteps"]
                assert np.array_equal(G.read_counts(), ref["counts"])
                for b in range(nblocks):
                    want = ref["pools"][b]
                    assert np.array_equal(G.read_pool(b), np.stack(want, axis=1) if len(want[0])
                                          else np.zeros((0, 4), np.uint32)), f"block {b}"
    assert grown


def test_a_call_that_runs_out_of_memory_leaves_no_error_behind(cuda_device, oracle):
    """A query batch whose tables do not fit fails with GW_E_NOMEM; the next
    call, and a graph opened after it, do not meet the allocation's error."""
    import torch

    import graphwalker_b200 as gw
    rp, ci = oracle.rmat_csr(11, 8, seed=5)
    blocks = oracle.compute_blocks(rp, 8)
    cur = np.arange(len(rp) - 1, dtype=np.uint32)
    p = gw.params(gw.RULE_JUMP, gw.SINK_VERTEX_COUNT, 10, seed=5)
    ref = oracle.run_walks(rp, ci, cur, rule=0, L=10, seed=5)["counts"]
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        torch.cuda.empty_cache()
        held = [torch.empty(max(0, torch.cuda.mem_get_info()[0] - 256 * MB), dtype=torch.uint8, device="cuda")]
        try:
            with pytest.raises(gw.GwError) as e:  # 2^26 slots of 8 bytes
                G.ppr(gw.params(gw.RULE_PPR, gw.SINK_NONE, 4), np.array([int(np.diff(rp).argmax())], np.uint32),
                      np.array([1 << 23], np.uint32))
            assert e.value.code == gw._lib.GW_E_NOMEM
        finally:
            held.clear()
            torch.cuda.empty_cache()
        for H in (G, gw.Graph.from_csr(rp, ci, blocks)):
            H.add_walks_at(cur)
            H.run(p)
            assert np.array_equal(H.read_counts(), ref)
        H.close()

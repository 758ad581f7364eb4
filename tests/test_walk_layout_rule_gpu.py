"""Which layout resident walks read is a rule on sizes (gw_walk.cu,
walks_use_records): a graph on either side of the limit gives the same walks.
GW_CSR_WALK_BYTES moves the limit, so that a small graph is walked over its
edge records (limit 0), over the plain layout, and with the two rules' limits
apart; counts, trajectories and closures equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph(oracle):
    rp, ci = oracle.rmat_csr(13, 8, seed=31)
    return rp, ci, oracle.compute_blocks(rp, 64)


@pytest.mark.parametrize("limit", ["0", "edge", "below", None], ids=["records", "at_limit", "past_limit", "default"])
@pytest.mark.parametrize("rule,L", [(0, 10), (1, 9), (2, 8), (3, 7), (4, 12)])
@pytest.mark.parametrize("rng", [0, 1])
def test_layouts_give_the_same_walks(cuda_device, oracle, graph, monkeypatch, limit, rule, L, rng):
    import graphwalker_b200 as gw
    rp, ci, blocks = graph
    size, share = len(ci) * 4 + (len(rp) - 1) * 8, 1 if rule == 0 else 2
    if limit is None:
        monkeypatch.delenv("GW_CSR_WALK_BYTES", raising=False)
    else:
        monkeypatch.setenv("GW_CSR_WALK_BYTES", {"0": "0", "edge": str(size * share), "below": str(size * share - 1)}[limit])
    r = np.random.default_rng(rule)
    cur = r.integers(0, len(rp) - 1, 3001).astype(np.uint32)
    ids = np.arange(len(cur), dtype=np.uint32)
    stride = L if rule != 2 else 256
    ref = oracle.run_walks(rp, ci, cur, ids=ids, src=cur, rule=rule, L=L, seed=4, stride=stride, rng=rng,
                           closure=True)
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        assert G.set_edge_records(gw.EDGE_RECORDS_ON)
        order = np.argsort(np.searchsorted(G.blocks[1:], cur, side="right"), kind="stable")
        for tuned in (False, True):
            G.walks_clear()
            G.add_walks_at(cur, ids=ids)
            G.run(gw.params(rule, gw.SINK_VERTEX_COUNT, L, seed=4, rng=rng))
            assert np.array_equal(G.read_counts(), ref["counts"])
            G.run(gw.params(rule, gw.SINK_PATH_RECORD, L, seed=4, rng=rng, path_stride=stride))
            paths, lens = G.read_paths(len(cur), stride)
            assert np.array_equal(lens, ref["plen"][order])
            for row, j in enumerate(order):
                assert np.array_equal(paths[row][: lens[row]], ref["paths"][j][: lens[row]]), j
            G.run(gw.params(rule, gw.SINK_CLOSURE_COUNT, L, seed=4, rng=rng))
            assert G.read_closure() == ref["closure"]
            if not tuned:  # again in a tuned launch shape
                import torch
                rec = np.stack([cur, ids, cur, np.zeros_like(cur)], 1).astype(np.uint32)
                dev = torch.from_numpy(rec.view(np.int32)).cuda()
                G.walk_autotune(gw.params(rule, gw.SINK_VERTEX_COUNT, L, seed=4, rng=rng), dev, len(cur))


@pytest.mark.parametrize("rule", [0, 1, 3], ids=["jump", "stop", "restart"])
def test_mega_hub_over_edge_records(cuda_device, oracle, monkeypatch, rule):
    """The hub whose degree escapes the packed record, on the record kernels."""
    from test_workload_sizes_gpu import _star_graph, test_mega_hub_walks_equal_oracle
    monkeypatch.setenv("GW_CSR_WALK_BYTES", "0")
    rp, ci = _star_graph()
    test_mega_hub_walks_equal_oracle((rp, ci, oracle.compute_blocks(rp, 64)), oracle, 1, rule)


@pytest.mark.parametrize("limit", ["0", str(1 << 40)], ids=["records", "csr"])
@pytest.mark.parametrize("rule,L", [(1, 5), (2, 5), (3, 20)])
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19])
def test_large_sets_on_either_side_of_the_rules(cuda_device, oracle, graph, monkeypatch, limit, rule, L, n):
    """Walk counts at which the layout (stop, uncapped: 2^19 walks) and the
    launch shape (restart: 40 MB of paths, here 2^19 walks of 20) turn."""
    import torch

    import graphwalker_b200 as gw
    monkeypatch.setenv("GW_CSR_WALK_BYTES", limit)
    rp, ci, blocks = graph
    cur = np.random.default_rng(n).integers(0, len(rp) - 1, n).astype(np.uint32)
    ids = np.arange(n, dtype=np.uint32)
    stride = L if rule != 2 else 0
    ref = oracle.run_walks(rp, ci, cur, ids=ids, src=cur, rule=rule, L=L, seed=4, stride=stride)
    rec = torch.from_numpy(np.stack([cur, ids, cur, np.zeros_like(cur)], 1).astype(np.uint32).view(np.int32)).cuda()
    with gw.Graph.from_csr(rp, ci, blocks) as G:
        counts = torch.zeros(G.nv, dtype=torch.int32, device="cuda")
        G.walk_device(gw.params(rule, gw.SINK_VERTEX_COUNT, L, seed=4), rec, n, counts=counts)
        G.sync()
        assert np.array_equal(counts.cpu().numpy().view(np.uint32), ref["counts"])
        if stride:
            paths = torch.full((n, stride), -1, dtype=torch.int32, device="cuda")
            lens = torch.zeros(n, dtype=torch.int32, device="cuda")
            G.walk_device(gw.params(rule, gw.SINK_PATH_RECORD, L, seed=4, path_stride=stride), rec, n, paths=paths,
                          plen=lens)
            G.sync()
            assert np.array_equal(lens.cpu().numpy().view(np.uint32), ref["plen"])
            assert np.array_equal(paths.cpu().numpy().view(np.uint32), ref["paths"])

"""Layout and launch shape of resident walks (gw_walk_shape): what the tuner
finds for one rule, sink and layout leaves the others as they were."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walks(n: int, nv: int, seed: int = 1):
    import torch
    cur = np.random.default_rng(seed).integers(0, nv, n).astype(np.uint32)
    rec = np.stack([cur, np.arange(n, dtype=np.uint32), cur, np.zeros_like(cur)], 1).astype(np.uint32)
    return torch.from_numpy(rec.view(np.int32)).cuda()


@pytest.mark.parametrize("limit", ["0", None], ids=["records", "by_rule"])
def test_tuning_one_rule_leaves_the_others(cuda_device, monkeypatch, limit):
    import graphwalker_b200 as gw
    if limit is not None:
        monkeypatch.setenv("GW_CSR_WALK_BYTES", limit)
    n = 1 << 20  # 12 visits each: 50 MB of paths
    params = {(rule, sink): gw.params(rule, sink, 12, path_stride=12 if sink == gw.SINK_PATH_RECORD else 0)
              for rule in (gw.RULE_JUMP, gw.RULE_STOP, gw.RULE_RESTART, gw.RULE_PPR)
              for sink in (gw.SINK_VERTEX_COUNT, gw.SINK_PATH_RECORD, gw.SINK_CLOSURE_COUNT)}
    with gw.Graph.rmat(16, 16, seed=2, blocksize_kb=1024) as G:
        assert G.set_edge_records(gw.EDGE_RECORDS_ON)
        before = {key: G.walk_shape(p, n) for key, p in params.items()}
        if limit == "0":
            assert all(records for records, _ in before.values())
            assert before[gw.RULE_JUMP, gw.SINK_VERTEX_COUNT] == (True, 5)
            often = G.walk_shape(gw.params(gw.RULE_JUMP, gw.SINK_VERTEX_COUNT, 12, jump_prob=0.5), n)
            assert often[0] and often[1] > 5
        assert before[gw.RULE_RESTART, gw.SINK_PATH_RECORD][1] == 6
        expect = dict(before)
        walks = _walks(n, G.nv)
        for key in ((gw.RULE_PPR, gw.SINK_VERTEX_COUNT), (gw.RULE_RESTART, gw.SINK_CLOSURE_COUNT),
                    (gw.RULE_JUMP, gw.SINK_VERTEX_COUNT)):
            ctas = G.walk_autotune(params[key], walks, n)
            expect[key] = (before[key][0], ctas)
            assert {k: G.walk_shape(p, n) for k, p in params.items()} == expect


def test_a_shape_is_kept_per_layout(cuda_device):
    """Stop walks: few over the records, many over the CSR of a small graph."""
    import graphwalker_b200 as gw
    p = gw.params(gw.RULE_STOP, gw.SINK_VERTEX_COUNT, 10)
    few, many = 1 << 14, 1 << 19
    with gw.Graph.rmat(16, 16, seed=2, blocksize_kb=1024) as G:
        assert G.set_edge_records(gw.EDGE_RECORDS_ON)
        shapes = G.walk_shape(p, few), G.walk_shape(p, many)
        assert [records for records, _ in shapes] == [True, False]
        ctas = G.walk_autotune(p, _walks(many, G.nv), many)
        assert G.walk_shape(p, many) == (False, ctas) and G.walk_shape(p, few) == shapes[0]
        G.set_edge_records(gw.EDGE_RECORDS_OFF)
        assert G.walk_shape(p, few)[0] is False
        G.set_residency(gw.STREAM_PINNED, 2)
        with pytest.raises(gw.GwError):
            G.walk_shape(p, few)


@pytest.mark.parametrize("scale,edges,rule,n,records",
                         [(22, 2, "jump", 1 << 22, False), (23, 2, "jump", (1 << 18) - 1, False),
                          (23, 2, "jump", 1 << 18, True), (24, 1, "jump", (1 << 16) - 1, False),
                          (24, 1, "jump", 1 << 16, True), (22, 2, "stop", 1 << 19, False),
                          (22, 2, "stop", (1 << 19) - 1, True), (23, 1, "stop", 1 << 19, True),
                          (22, 2, "prob", 1 << 19, False), (23, 1, "prob", 1 << 19, True),
                          (14, 2, "ppr", 1 << 19, True), (14, 2, "restart", 1 << 19, True)])
def test_layout_by_sizes(cuda_device, scale, edges, rule, n, records):
    """Vertices whose records leave the L2, and few walks."""
    import graphwalker_b200 as gw
    rule = {"jump": gw.RULE_JUMP, "stop": gw.RULE_STOP, "prob": gw.RULE_PROB, "ppr": gw.RULE_PPR,
            "restart": gw.RULE_RESTART}[rule]
    with gw.Graph.rmat(scale, edges, seed=2, blocksize_kb=1 << 16) as G:
        assert G.set_edge_records(gw.EDGE_RECORDS_ON)
        assert G.walk_shape(gw.params(rule, gw.SINK_VERTEX_COUNT, 10), n)[0] is records


def test_jumps_over_many_vertices_are_not_slower_with_records(cuda_device):
    """4 M jumping walks over 16.8 M vertices of two edges, a 255 MB CSR: the
    records built beside it make them a quarter faster, when they are read."""
    import torch

    import graphwalker_b200 as gw
    n, p = 1 << 22, gw.params(gw.RULE_JUMP, gw.SINK_VERTEX_COUNT, 10)
    with gw.Graph.rmat(24, 2, seed=2, blocksize_kb=1 << 16) as G:
        walks = _walks(n, G.nv)
        counts = torch.zeros(G.nv, dtype=torch.int32, device="cuda")
        ms = {}
        for mode in (gw.EDGE_RECORDS_OFF, gw.EDGE_RECORDS_ON):
            G.set_edge_records(mode)
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                G.walk_device(p, walks, n, counts=counts)
                b.record()
                b.synchronize()
                ms[mode] = min(ms.get(mode, 1e9), a.elapsed_time(b))
    assert ms[gw.EDGE_RECORDS_ON] < 0.92 * ms[gw.EDGE_RECORDS_OFF]

"""The walk tests of small graphs again, with every resident walk over the edge
records wherever they are built (GW_CSR_WALK_BYTES=0): by the layout rule most
of them would read the plain CSR in both of their layouts."""
import pytest
from test_edge_cases_gpu import (graph, test_paths_and_closure_of_short_walks,  # noqa: F401
                                 test_short_walks_equal_oracle)
from test_native_rng_gpu import small, test_native_walks_equal_oracle  # noqa: F401
from test_walk_gpu import (test_counts_match_reference_golden, test_paths_and_closure_match_reference_golden,  # noqa: F401
                           test_ppr_single_source_matches_oracle, test_rmat16_all_rules_match_oracle,
                           test_run_pools_host_call, test_run_pools_pipelined_equals_oracle,
                           test_walk_autotune_keeps_results)

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def records_wherever_built(monkeypatch):
    monkeypatch.setenv("GW_CSR_WALK_BYTES", "0")


def test_the_records_are_read(cuda_device):
    import graphwalker_b200 as gw
    with gw.Graph.rmat(12, 8, seed=3, blocksize_kb=64) as G:
        assert G.set_edge_records(gw.EDGE_RECORDS_ON)
        for rule in (gw.RULE_JUMP, gw.RULE_STOP, gw.RULE_PROB, gw.RULE_RESTART, gw.RULE_PPR):
            assert G.walk_shape(gw.params(rule, gw.SINK_VERTEX_COUNT, 5), 1 << 20)[0]

"""The bench line's critical path of a network as it is routed: the pieces of the
reaches form the graph whose longest chain is waited for."""
import numpy as np
import pytest

from test_bench_contract import _bench_module


@pytest.mark.parametrize("segments,piece", [(131_072, 1), (1_048_576, 2), (1_048_577, 0)])
def test_pieces_of_a_network(segments, piece):
    import troute_gb300 as T

    b = _bench_module()
    topo = b.workload("c0", 4)["topo"]
    p = b.routed_pieces(topo, segments)
    T.validate(p["reach_seg_start"], p["reach_seg_len"], p["reach_up_ptr"], p["reach_up_idx"], p["n_segments"])
    ln = p["reach_seg_len"]
    assert ln.sum() == topo["reach_seg_len"].sum()
    if not piece:
        assert p is topo
        return
    assert ln.max() == piece
    # one step: the longest path is the same; every further step adds a piece
    one = T.critical_path(topo, 1)
    assert T.critical_path(p, 1) == one
    if piece == 1:
        assert T.critical_path(p, 50) == one + 49
    else:
        assert one + 49 <= T.critical_path(p, 50) <= one + 2 * 49
    assert T.critical_path(topo, 50) >= one + 49 * np.max(topo["reach_seg_len"])


def test_line_states_both_chains():
    import troute_gb300 as T

    b = _bench_module()
    for name in ("c0", "ens:3:2000:w"):
        w = b.workload(name, 4)
        cp = b.critical_path_bound(T, w, 4, 6.5, 2070.0, 100.0)
        r = cp["as_routed"]
        assert r["segment_solves"] <= cp["segment_solves"] and r["lower_bound_ms"] < cp["lower_bound_ms"]
        assert abs(r["lower_bound_ms"] - r["segment_solves"] * 6.5 * cp["pass_us_min"] / 1e3) < 1e-9

"""Reaches routed as items of one, two or all of their segments (the choice goes by
the number of segments of the handle): bit-identical to the oracle over every step,
also when a run is cut into launches, the state is put back, another kernel takes
over in between or a graph is replayed, and for zeros of both signs."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O
from troute_gb300 import synth

pytestmark = pytest.mark.gpu


def network(reaches, segments, longest, seed):
    """A random forest: reaches of 0 to `longest` segments that drain into a later one."""
    rng = np.random.default_rng(seed)
    ln = rng.integers(0, longest + 1, reaches).astype(np.int32)
    while ln.sum() != segments:   # exactly `segments` of them
        i = rng.integers(reaches)
        ln[i] = np.clip(ln[i] + np.sign(segments - ln.sum()), 0, longest)
    down = np.array([rng.integers(r + 1, min(reaches, r + 40)) if r + 1 < reaches and rng.random() < 0.97 else -1
                     for r in range(reaches)])
    up = np.argsort(down, kind="stable")[np.sum(down < 0):]
    cnt = np.bincount(down[down >= 0], minlength=reaches)
    return {"n_segments": segments, "reach_seg_start": (np.cumsum(ln) - ln).astype(np.int32), "reach_seg_len": ln,
            "reach_up_ptr": np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32), "reach_up_idx": up.astype(np.int32)}


def inputs(topo, n_ts, seed):
    S, R = topo["n_segments"], len(topo["reach_seg_start"])
    rng = np.random.default_rng(seed)
    p, ql = synth.make_params(seed, S), synth.make_qlat(seed, S, n_ts)
    q0, d0, r0 = rng.uniform(0.0, 3.0, S), rng.uniform(0.0, 0.5, S), rng.uniform(0.0, 3.0, R)
    for a in (q0, d0, r0):   # no flow at all in places, with zeros of both signs
        a[rng.random(len(a)) < 0.3] = 0.0
        a[rng.random(len(a)) < 0.1] = -0.0
    ql[:, rng.random(S) < 0.3] = 0.0
    return p, ql, q0, d0, r0


def same(a, b):
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("segments,longest,n_ts", [(1, 1, 3), (900, 30, 9), (131_072, 10, 2), (131_073, 10, 2),
                                                   (1_048_576, 10, 2), (1_048_577, 10, 2)])
def test_items_around_the_sizes_of_the_rule(segments, longest, n_ts):
    topo = network(max(1, segments * 2 // (longest + 1)), segments, longest, segments)
    p, ql, q0, d0, r0 = inputs(topo, n_ts, segments)
    with O.pow_mode(1):
        o = O.route_tree(topo, p, ql, q0, d0, r0, history=True)
    g = T.route_tree(topo, p, ql, q0, d0, r0, history=True)
    for k in ("q_hist", "q", "d", "reach_last"):
        same(g[k], o[k])
    assert g["stats"]["iterations"] == o["iterations"]


@pytest.mark.parametrize("chunk", [0, 1, 3])
def test_runs_in_parts(chunk):
    torch = pytest.importorskip("torch")
    topo = network(300, 1500, 12, 5)
    n_ts = 14
    p, ql, q0, d0, r0 = inputs(topo, n_ts, 6)
    with O.pow_mode(1):
        o = O.route_tree(topo, p, ql, q0, d0, r0)
    dev = torch.from_numpy(ql).cuda()
    rows = [dev[t].data_ptr() for t in range(n_ts)]
    with T.Network(topo, p, cfg=T.make_cfg(max_chunk_steps=chunk)) as net:
        net.set_state(q0, d0, r0)
        net.run_device(rows[0], 5)
        net.sync()
        q, d, _, r = net.get_state()
        net.set_state(q, d, r)                                       # steps 0-4, put back
        net.set_cfg(T.make_cfg(mapping=2, max_chunk_steps=chunk))    # steps 5, 6 by the lane-refill kernel
        net.run_device(rows[5], 2)
        net.set_cfg(T.make_cfg(max_chunk_steps=chunk))
        saved = net.checkpoint()
        net.run_device(rows[7], 3)
        net.restore(saved)
        net.run_device(rows[7], 3)                                   # 7-9, twice
        net.graph_capture(rows[10], 4)
        net.graph_launch()                                                 # 10-13
        net.sync()
        q, d, _, r = net.get_state()
    same(q, o["q"])
    same(d, o["d"])
    same(r, o["reach_last"])

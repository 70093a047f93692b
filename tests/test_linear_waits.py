"""The linearised form's wait budget counts time without progress only: a path may
wait for another far longer than the budget while that one is being routed. A wait in
whose budget nothing is done ends the run with an error, after which the handle
routes as before."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O
from troute_gb300.api import ETIMEOUT

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def network(kind):
    """A short path that joins the end of a long one, which is the light one there."""
    if kind == "deep":   # 45 reaches of a segment, 40 reaches of 500
        ups = [[]] + [[k] for k in range(44)] + [[]] + [[45 + k] for k in range(39)] + [[44, 84]]
        ln = [1] * 45 + [500] * 40 + [1]
    else:                # a reach of a segment, one of 20,000
        ups, ln = [[], [], [0, 1]], [1, 20_000, 1]
    ln = np.array(ln, np.int32)
    return {"n_segments": int(ln.sum()), "reach_seg_start": (np.cumsum(ln) - ln).astype(np.int32), "reach_seg_len": ln,
            "reach_up_ptr": np.concatenate([[0], np.cumsum([len(u) for u in ups])]).astype(np.int32),
            "reach_up_idx": np.array([x for u in ups for x in u], np.int32)}


@pytest.mark.parametrize("kind", ["deep", "shallow"])
def test_budget_counts_time_without_progress(kind):
    topo = network(kind)
    S, n_ts = topo["n_segments"], 32
    rng = np.random.default_rng(3)
    co = [rng.uniform(0.0, 0.3, S).astype(np.float32) for _ in range(4)]
    ql = rng.uniform(0.0, 2.0, (n_ts, S)).astype(np.float32)
    q0 = rng.uniform(0.0, 9.0, S).astype(np.float32)
    want = O.linear_route(co, topo, ql, q0)
    qlat, start = torch.from_numpy(ql).cuda(), torch.from_numpy(q0).cuda()
    q = torch.empty_like(start)

    def run(wait_cycles):
        q.copy_(start)
        torch.cuda.synchronize()
        net.run_device(qlat.data_ptr(), n_ts, q.data_ptr(), wait_cycles=wait_cycles)
        np.testing.assert_array_equal(q.cpu().numpy().view(np.int32), want.view(np.int32))

    with T.LinearNetwork(topo, co) as net:
        run(0)
        run(1_000_000)   # ~0.5 ms, of a wait of several
        with pytest.raises(T.TrouteError) as e:
            run(1)
        assert e.value.code == ETIMEOUT
        run(1_000_000)

"""Reach-parallel steps of one host thread that run at the same time, on two streams
or from two captured graphs: every call routes every one of its reaches, once. The
outputs start as NaN, or are the inputs themselves; bit for bit what the same calls
give one after another, and the oracle. CPU: the shares of the blocks cover the
reaches exactly once."""
import ctypes as C

import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O
from troute_gb300 import synth

TOL = (1e-8, 1e-10, 100, 5)


class Step:
    """A call's arrays on the device; in place: discharge and depth are updated."""

    def __init__(self, torch, n, seed, in_place):
        rng = np.random.default_rng(seed)
        ln = rng.integers(1, 6, n).astype(np.int32)
        S = int(ln.sum())
        self.host = [synth.make_params(seed, S), rng.uniform(0.0, 2.0, S), (np.cumsum(ln) - ln).astype(np.int32), ln,
                     *(rng.uniform(0.0, 5.0, S) for _ in range(2)), rng.uniform(0.0, 2.0, S)]
        self.p, self.ql, self.rs, self.rl, self.qu, qd, dp = (
            torch.from_numpy(a.view(np.float64) if a.dtype.names else a).cuda() for a in self.host)
        self.start = qd, dp
        self.qd, self.dp, self.v = qd.clone(), dp.clone(), torch.empty_like(qd)
        self.q, self.d = (self.qd, self.dp) if in_place else (torch.empty_like(qd), torch.empty_like(dp))
        self.n, self.S = n, S
        self.cfg = T.make_cfg(*TOL)

    def reset(self):
        for a in (self.v, self.q, self.d):
            a.fill_(float("nan"))
        self.qd.copy_(self.start[0])
        self.dp.copy_(self.start[1])

    def call(self, stream):
        rc = T.lib().troute_mc_reach_parallel_device(
            *(a.data_ptr() for a in (self.p, self.ql, self.rs, self.rl, self.qu, self.qd, self.dp, self.q, self.v, self.d)),
            10.0, 300.0, self.n, self.S, C.byref(self.cfg), stream.cuda_stream)
        assert rc == 0, T.lib().troute_last_error()

    def result(self):
        return [a.cpu().numpy() for a in (self.q, self.v, self.d)]


def check(torch, steps, one_by_one, go):
    for _ in range(4):
        for s in steps:
            s.reset()
        torch.cuda.synchronize()
        go()
        torch.cuda.synchronize()
        for s, want in zip(steps, one_by_one):
            for a, b in zip(s.result(), want):
                np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("sizes", [(300_000, 70_000), (70_000, 200), (3000, 2431), (200, 1)])
def test_calls_side_by_side(sizes, in_place):
    torch = pytest.importorskip("torch")
    steps = [Step(torch, n, 7 + n, in_place) for n in sizes]
    streams = [torch.cuda.Stream() for _ in steps]
    one_by_one = []
    for s in steps:
        s.reset()
        torch.cuda.synchronize()
        s.call(streams[0])
        torch.cuda.synchronize()
        one_by_one.append(s.result())
    small = steps[-1]
    if small.n <= 3000:
        with O.pow_mode(1):
            want = O.cpu_mc(*small.host, uq=10.0, tol=TOL)
        for a, b in zip(one_by_one[-1], want[:3]):
            np.testing.assert_array_equal(a, b)

    def on_streams():
        for s, st in zip(steps, streams):
            s.call(st)

    check(torch, steps, one_by_one, on_streams)
    graphs = []
    for s, st in zip(steps, streams):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            s.call(st)
        graphs.append(g)

    def replayed():
        for g, st in zip(graphs, streams):
            with torch.cuda.stream(st):
                g.replay()

    check(torch, steps, one_by_one, replayed)


@pytest.mark.parametrize("nr", [1, 3, 4, 5, 607, 608, 609, 2431, 2433, 9729, 19_455, 19_456, 19_457, 20_000, 1_100_001])
def test_shares_cover_the_reaches_once(nr, sms=152, warps=4, run_of_many=16):
    """The rule of reach_parallel.cu: reach of the k-th taking of a block."""
    per_warp = -(-nr // (warps * sms))
    lanes = min(per_warp, 32)
    blocks = -(-nr // (warps * lanes)) if per_warp <= 32 else 3 * sms
    run_len = warps * lanes if per_warp <= 32 else run_of_many
    seen = np.zeros(nr, int)
    for b in range(blocks):
        k = np.arange(-(-nr // (blocks * run_len)) * run_len + 128)
        at = (k // run_len * blocks + b) * run_len + k % run_len
        assert np.all(np.diff(at) > 0)   # none below nr follows one that is not
        seen[at[at < nr]] += 1
    assert np.all(seen == 1)

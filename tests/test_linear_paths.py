"""The linearised form's path sweeps (linear.cu) at the edges of their rules:
step counts around the lanes' and blocks' shares (1 to 300 steps), paths around
the depth from which one gets a block of its own, reaches with many upstream
reaches, long reaches, -0 coefficients and inflows; bit for bit against the oracle."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O

pytestmark = pytest.mark.gpu


def topo_of(ups, seg_len):
    seg_len = np.asarray(seg_len, np.int32)
    return {"n_segments": int(seg_len.sum()), "reach_seg_start": (np.cumsum(seg_len) - seg_len).astype(np.int32),
            "reach_seg_len": seg_len,
            "reach_up_ptr": np.concatenate([[0], np.cumsum([len(u) for u in ups])]).astype(np.int32),
            "reach_up_idx": np.array([x for u in ups for x in u], np.int32)}


def comb(rng, depth, tooth):
    """A main stem of `depth` reaches; every third takes a side chain of up to
    `tooth` reaches, every seventh three short ones more."""
    ups, main = [[]], 0
    for k in range(1, depth):
        sides = [int(rng.integers(1, tooth + 1))] if k % 3 == 0 else []
        sides += [1, 2, 1] if k % 7 == 0 else []
        heads = []
        for n in sides:
            for j in range(n):
                ups.append([] if j == 0 else [len(ups) - 1])
            heads.append(len(ups) - 1)
        order = [main] + heads
        rng.shuffle(order)
        ups.append([int(u) for u in order])
        main = len(ups) - 1
    return ups


def check(ups, n_ts, seed, max_len=5):
    rng = np.random.default_rng(seed)
    topo = topo_of(ups, rng.integers(1, max_len + 1, len(ups)))
    S = topo["n_segments"]
    co = [rng.uniform(-0.2, 0.6, S).astype(np.float32) for _ in range(4)]
    ql = rng.uniform(0.0, 2.0, (n_ts, S)).astype(np.float32)
    q0 = rng.uniform(0.0, 9.0, S).astype(np.float32)
    dry = rng.random(S) < 0.2
    for c in co:
        c[dry] = np.float32(-0.0)
    ql[:, dry] = 0.0
    q0[dry] = np.float32(-0.0)
    want = O.linear_route(co, topo, ql, q0)
    got = T.linear_route(topo, co, ql, q0)
    np.testing.assert_array_equal(got.view(np.int32), want.view(np.int32))


@pytest.mark.parametrize("n_ts", [1, 2, 7, 8, 9, 32, 33, 64, 65, 128, 129, 300])
def test_step_counts(n_ts):
    check(comb(np.random.default_rng(1), 60, 20), n_ts, n_ts)


@pytest.mark.parametrize("depth", [1, 2, 30, 31, 32, 33, 200])
@pytest.mark.parametrize("n_ts", [5, 48])
def test_depths(depth, n_ts):
    check(comb(np.random.default_rng(depth), depth, max(1, depth // 2)), n_ts, depth)


def test_isolated_reaches_and_long_ones():
    check([[] for _ in range(301)], 17, 3, max_len=40)


def test_wide_confluence():
    n = 299
    check([[] for _ in range(n)] + [list(range(n))] + [[n]], 50, 4)

"""Narrow passes (up to four solves shared by a warp, narrow_pass.cuh) and the
claim rule that switches between them and full passes (route_dataflow.cu):
networks whose ready items number around the switch points, bit-identical to
the oracle over every step. Independent reaches give as many ready items as
reaches; chains of different lengths keep few solves in flight."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O
from troute_gb300 import synth

pytestmark = pytest.mark.gpu
TIGHT = (1e-8, 1e-10, 100, 5)


def _check(topo, seed, tol, n_ts, warm_depth=0.1):
    S, R = topo["n_segments"], len(topo["reach_seg_start"])
    rng = np.random.default_rng(seed)
    p, ql = synth.make_params(seed, S), synth.make_qlat(seed, S, n_ts)
    ql[:, rng.random(S) < 0.05] = 0.0
    q0, d0 = rng.uniform(0.0, 3.0, S), rng.uniform(0.0, 2 * warm_depth, S)
    d0[rng.random(S) < 0.1] = 0.0
    q0[rng.random(S) < 0.1] = 0.0
    with O.pow_mode(1):
        o = O.route_tree(topo, p, ql, q0, d0, np.full(R, 0.2), history=True, tol=tol)
    cfg = T.make_cfg(rtol=tol[0], atol=tol[1], maxiter=tol[2], attempts=tol[3])
    g = T.route_tree(topo, p, ql, q0, d0, np.full(R, 0.2), cfg=cfg, history=True)
    for k in ("q_hist", "q", "d", "reach_last"):
        np.testing.assert_array_equal(g[k], o[k])
    assert g["stats"]["iterations"] == o["iterations"]


@pytest.mark.parametrize("tol", [O.REF_TOL, TIGHT], ids=["ref_tol", "rtol_1e-8"])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 33, 607, 1215, 1217, 5000])
def test_independent_reaches(n, tol):
    ln = np.random.default_rng(n).integers(1, 5, n).astype(np.int32)
    topo = {"n_segments": int(ln.sum()), "reach_seg_start": (np.cumsum(ln) - ln).astype(np.int32), "reach_seg_len": ln,
            "reach_up_ptr": np.zeros(n + 1, np.int32), "reach_up_idx": np.zeros(0, np.int32)}
    _check(topo, 100 + n, tol, 4)


@pytest.mark.parametrize("width,length", [(1, 40), (3, 17), (6, 9)])
def test_chains_into_one_outlet(width, length):
    """`width` chains of `length` reaches meeting in one last reach."""
    n = width * length + 1
    up = [[] if i % length == 0 else [i - 1] for i in range(n - 1)] + [[length * (k + 1) - 1 for k in range(width)]]
    ln = np.random.default_rng(n).integers(0, 4, n).astype(np.int32)
    topo = {"n_segments": int(ln.sum()), "reach_seg_start": (np.cumsum(ln) - ln).astype(np.int32), "reach_seg_len": ln,
            "reach_up_ptr": np.concatenate([[0], np.cumsum([len(u) for u in up])]).astype(np.int32),
            "reach_up_idx": np.array([x for u in up for x in u], np.int32)}
    _check(topo, n, TIGHT, 12)

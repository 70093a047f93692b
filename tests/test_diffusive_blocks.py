"""The diffusive-wave kernel where its blocks, tiles and segments end and where
its short quotients do not apply: against the oracle, bit for bit."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O


def inputs(n, max_nodes, lengths, seed):
    rng = np.random.default_rng(seed)
    rp = np.zeros(n, np.dtype([("ncomp", "<i4"), ("theta", "<f4"), ("dtini", "<f4")]))
    rp["ncomp"] = np.minimum(rng.choice(lengths, n), max_nodes)
    rp["theta"] = rng.choice([0.0, 0.5, 0.55, 1.0], n)
    rp["dtini"] = rng.choice([60.0, 300.0], n)
    dx = rng.uniform(0.5, 800.0, (n, max_nodes)).astype(np.float32)
    diff = rng.uniform(0.0, 200.0, (n, max_nodes)).astype(np.float32)
    qp = rng.uniform(0.0, 60.0, (n, max_nodes)).astype(np.float32)
    return rp, dx, diff, qp


def check(rp, dx, diff, qp):
    start = np.full_like(qp, -7.0)
    with np.errstate(all="ignore"):
        want = O.diffusive_tridiag(rp, dx, diff, qp, qp_out=start)
    np.testing.assert_array_equal(T.diffusive_tridiag(rp, dx, diff, qp, qp_out=start), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 9728, 9729, 9759])
@pytest.mark.parametrize("lengths", [[1, 2, 3], [31, 32, 33], [95, 96, 97], [127, 128, 129, 140]])
def test_edges_of_blocks_and_tiles(n, lengths):
    check(*inputs(n, 140, lengths, n + lengths[0]))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 9800])
def test_values_outside_the_short_quotients(n):
    """Zeros of both signs, values near the ends of the type, infinities and NaN."""
    rp, dx, diff, qp = inputs(n, 130, [1, 5, 64, 100, 130], 9)
    rng = np.random.default_rng(10)
    odd = np.array([0.0, -0.0, 1e-45, 1e-38, 1e-30, 1e-19, 1e19, 1e30, 3e38, np.inf, -np.inf, np.nan, 1.9999999], np.float32)
    for a in (dx, diff, qp):
        at = rng.random(a.shape) < 0.01
        a[at] = rng.choice(odd, at.sum())
    qp[::5] = 0.0
    rp["theta"][::7] = rng.choice(odd, len(rp["theta"][::7]))
    check(rp, dx, diff, qp)

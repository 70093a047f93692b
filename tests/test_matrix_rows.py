"""The matrix step over every row length around its classes and batches, against
the oracle, bit for bit. With tolerance 0 row r of a chain holds r + 1 entries."""
import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O


def networks():
    for R in (1, 2, 5, 33, 64, 700):
        yield f"chain{R}", np.array([0] + list(range(R)), np.int32), np.arange(R - 1, dtype=np.int32)
    for R in (4, 9, 17, 33, 34, 129, 130, 257, 5000):   # one row of R entries, the others of one
        yield f"star{R}", np.array([0] * R + [R - 1], np.int32), np.arange(R - 1, dtype=np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("name,ptr,idx", list(networks()), ids=[n[0] for n in networks()])
@pytest.mark.parametrize("tol", [0.0, 1e-3, 10.0])
def test_row_lengths(name, ptr, idx, tol):
    R = len(ptr) - 1
    rng = np.random.default_rng(R)
    c = [rng.uniform(0.2, 0.6, R).astype(np.float32) for _ in range(4)]
    if tol < 1.0:
        c[1][::3] *= -1.0
    ql = rng.uniform(0.0, 2.0, (5, R)).astype(np.float32)
    q0 = rng.uniform(0.05, 20.0, R).astype(np.float32)
    ql[:, ::4] = 0.0
    m = O.matrix_build(ptr, idx, c, tol)
    for n_ts in (1, 4, 5):
        got = T.matrix_route(ptr, idx, c, ql[:n_ts], q0, tol)
        want = O.matrix_route(m[0], m[1], ql[:n_ts], q0)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))

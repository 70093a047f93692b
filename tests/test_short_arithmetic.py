"""The secant pass's short quotients and powers (near_rcp, near_quot, quot_doubt
in fpbits.cuh, pow23_53_near in crpow.cuh, secant_pass in mc_solve.cuh).

CPU: near_quot restated over exact rationals from any reciprocal its error
bound admits. Where it raises no doubt the result must be the correctly rounded
quotient: random operands, significands at the ends of a binade, and the
hardest quotients there are, a few units of 2^-106 from a rounding midpoint.
GPU: the device code on the same hard quotients, and solves whose parameters,
flows and depths lie outside the ranges of the short forms (they take
exact_pass) or switch between both forms, bit-identical to the oracle."""
import math
import struct
from fractions import Fraction as F

import numpy as np
import pytest

import troute_gb300 as T
from oracle import troute_oracle as O
from troute_gb300 import synth


def hi32(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0] >> 32


def near_quot(a, b, y):
    """(quotient, doubt) as fpbits.cuh forms them."""
    q0 = a * y
    r = float(F(a) - F(b) * F(q0))
    q = float(F(q0) + F(r) * F(y))
    hq, hr = hi32(q0), hi32(r) & 0x7FFFFFFF
    t = max((hi32(b) & 0x7FFFFFFF) - (1076 << 20) + (hq & 0x7FF00000), 4)
    d = hr - t
    return q, -1 <= d <= 1 or d >= int(1.49 * 1048576) or ((hq & 0xFFFFF) == 0 and hr != 0)


def reciprocals(b):
    """The doubles next to 1/b that near_rcp's bound of (1/2 + 2^-11) ulp admits."""
    y = float(F(1) / F(b))
    return [c for c in (math.nextafter(y, 0.0), y, math.nextafter(y, math.inf))
            if abs(F(c) - F(1) / F(b)) <= F(math.ulp(y)) * (F(1, 2) + F(1, 2048))]


def hard_quotients(rng, n):
    """(a, b) with a/b in (1/2, 1) within 3 units of 2^-106/b of a midpoint: for
    an odd significand B, M = -k / B mod 2^54 is the midpoint's numerator."""
    out = []
    while len(out) < n:
        B = int(rng.integers(2 ** 52, 2 ** 53)) | 1
        if rng.random() < 0.3:
            B = (2 ** 53 - 1) - 2 * int(rng.integers(0, 1000))
        for k in (-3, -2, -1, 1, 2, 3):
            M = (-k * pow(B, -1, 2 ** 54)) % 2 ** 54
            if M % 2 == 0 or M < 2 ** 53:
                continue
            A = (M * B + k) >> 54
            if 2 ** 52 <= A < B:
                out.append((float(A), float(B)))
    return out[:n]


def operands(rng):
    ones = 2.0 - 2.0 ** -52
    for a, b in hard_quotients(rng, 3000):
        yield a, b
    for _ in range(10000):
        yield math.ldexp(rng.uniform(1, 2), int(rng.integers(-150, 150))), math.ldexp(rng.uniform(1, 2), int(rng.integers(-150, 150)))
    for _ in range(2000):   # both significands near 2: the largest distance of q0
        yield ones - 2.0 ** -52 * int(rng.integers(0, 5000)), ones - 2.0 ** -52 * int(rng.integers(0, 5000))
    for _ in range(2000):   # quotients next to a power of two
        b = rng.uniform(1, 2)
        yield b + math.ulp(b) * int(rng.integers(-4, 5)), b


def test_near_quotient_is_the_ieee_quotient_unless_it_doubts():
    rng = np.random.default_rng(5)
    doubts = n = 0
    for a, b in operands(rng):
        for y in reciprocals(b):
            for s in (1.0, -1.0):
                q, doubt = near_quot(s * a, b, y)
                if not doubt:
                    assert q == s * a / b, (s * a, b, y)
        doubts += doubt
        n += 1
    assert doubts > 1000   # the hard quotients are among them
    # zero and exact quotients never doubt
    for a, b in ((0.0, 3.0), (0.0, 300.0), (6.0, 3.0), (1.0, 4.0), (450.0, 450.0)):
        q, doubt = near_quot(a, b, float(F(1) / F(b)))
        assert q == a / b and not doubt


@pytest.mark.gpu
def test_device_quotients_near_midpoints():
    rng = np.random.default_rng(6)
    ops = np.array(list(operands(rng)))
    e = rng.integers(-80, 80, (len(ops), 2))
    a, b = np.ldexp(ops[:, 0], e[:, 0]) * rng.choice([-1, 1], len(ops)), np.ldexp(ops[:, 1], e[:, 1])
    np.testing.assert_array_equal(T.debug_div(a, b), a / b)


@pytest.mark.gpu
@pytest.mark.parametrize("tol", [O.REF_TOL, (1e-8, 1e-10, 100, 5)], ids=["ref_tol", "rtol_1e-8"])
def test_solves_outside_the_short_ranges(tol):
    """Single-segment and longer reaches with flows of 1e-60, 1e-40 and negative
    lateral inflow, channels of 1e-15 and 1e15 m, a dry bed, depths of 1e-40, 1e-5,
    1e20 and 1e150 m, roughness of 1e13, twcc = 0: bit-identical to the oracle."""
    rng = np.random.default_rng(7)
    n = 1200
    p = synth.make_params(91, n)
    ql, qu, qd = (rng.uniform(0.0, 5.0, n) for _ in range(3))
    dp = rng.uniform(0.0, 2.0, n)
    for k, (name, v) in enumerate((("dx", 1e15), ("dx", 1e-15), ("n_ch", 1e13), ("bw", 1e-14), ("twcc", 0.0), ("tw", 1e14),
                                   ("s0", 1e-30), ("cs", 1e-13))):
        p[name][40 * k:40 * k + 20] = v
    for k, v in enumerate((1e-60, 1e-40, 0.0, 1e20)):
        s = slice(400 + 40 * k, 400 + 40 * k + 40)
        ql[s], qu[s], qd[s] = v, v, v
    ql[600:640] = -1e-3
    ql[640:660] = -0.0
    for k, v in enumerate((0.0, 1e-40, 1e-5, 1e20, 1e150)):
        dp[700 + 40 * k:740 + 40 * k] = v
    p["tw"][900:940] = p["bw"][900:940]
    p["tw"][940:960] = 0.5 * p["bw"][940:960]
    rl = np.tile([1, 2, 1, 5, 3], 100).astype(np.int32)[:500]
    rl = rl[np.cumsum(rl) <= n]
    rs = (np.cumsum(rl) - rl).astype(np.int32)
    m = int(rs[-1] + rl[-1])
    p, ql, qu, qd, dp = (x[:m] for x in (p, ql, qu, qd, dp))
    cfg = T.make_cfg(rtol=tol[0], atol=tol[1], maxiter=tol[2], attempts=tol[3])
    for uq in (10.0, 0.0):
        with O.pow_mode(1):
            want = O.cpu_mc(p, ql, rs, rl, qu, qd, dp, uq=uq, tol=tol)
        got = T.mc_reach_parallel(p, ql, rs, rl, qu, qd, dp, uq=uq, cfg=cfg, return_stats=True)
        for g, w in zip(got[:3], want[:3]):
            np.testing.assert_array_equal(g, w)
        assert got[3]["iterations"] == want[3]

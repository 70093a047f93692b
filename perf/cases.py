"""Performance cases: the work a user of the routing library has it do, through
its public entry points (the Python mirror and, for device arrays, the C ABI it
binds). Sizes and distributions are the benchmark's: uniform random binary
trees with about 2.45 segments per reach, dt 300 s, a flat initial state routed
a few steps ahead so that the timed steps start from a developed flow.

Kinds:
  tree      one river network, several steps, from a given state to a read-back
            state (a forecast cycle); lateral inflow from the host or the device
  basins    many independent networks routed as one batch
  ensemble  perturbed members of one network, started from the learned depth
  reach     one step over independent reaches, device arrays (kernel_mc_gpu)
  linear    the linearised form over a whole network
  matrix    the truncated propagation matrices over a reach-level network
  diffusive the diffusive-wave tridiagonal step
  fit       training the warm start's network on recorded pairs
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "noaa-gpu-kernels_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import troute_gb300 as T  # noqa: E402
from troute_gb300 import synth  # noqa: E402

DT = 300.0
TIGHT = {"rtol": 1e-8, "atol": 1e-10}   # the benchmark's depth tolerance
REF = {"rtol": 0.01, "atol": 0.01}      # the reference's constants


def listed():
    return [
        # a gauged basin of 1,000 segments over a day of 5-minute steps, host arrays, the
        # reference's tolerance: the smallest forecast, all latency
        {"name": "tree_basin", "kind": "tree", "segments": 1000, "steps": 288, "tight": False, "host": True},
        # a regional network, device inflow, tight tolerance: the dependency graph is narrow
        # next to the chip
        {"name": "tree_region", "kind": "tree", "segments": 200_000, "steps": 24, "tight": True, "host": False},
        # the national network (2.7 M segments), the largest single network
        {"name": "tree_national", "kind": "tree", "segments": 2_700_000, "steps": 24, "tight": True, "host": False},
        # a batch of independent basins of very different sizes, one launch
        {"name": "basins", "kind": "basins", "basins": 48, "segments_lo": 500, "segments_hi": 50_000, "steps": 24,
         "tight": True},
        # an ensemble forecast: 64 perturbed members with the learned warm start
        {"name": "ensemble_warm", "kind": "ensemble", "segments": 20_000, "members": 64, "steps": 16},
        # one coupling step of a small model's reaches (latency and launch)
        {"name": "reach_small", "kind": "reach", "reaches": 200, "segments": 1000, "tight": False},
        # one coupling step of all national reaches
        {"name": "reach_national", "kind": "reach", "reaches": 1_100_000, "segments": 2_700_000, "tight": True},
        # the fast approximate mode over the national network
        {"name": "linear_national", "kind": "linear", "segments": 2_700_000, "steps": 48},
        # the matrix form of a large reach-level network
        {"name": "matrix_large", "kind": "matrix", "reaches": 400_001, "steps": 48},
        # diffusive-wave steps: one model's reaches, and a continental set
        {"name": "diffusive_small", "kind": "diffusive", "reaches": 2003, "max_nodes": 500, "lo": 20, "hi": 100},
        {"name": "diffusive_large", "kind": "diffusive", "reaches": 200_000, "max_nodes": 500, "lo": 20, "hi": 100},
        # training the warm start on a network's recorded solves, one epoch
        {"name": "fit", "kind": "fit", "pairs": 1_000_000, "epochs": 1, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tree", "tree", "basins", "ensemble", "reach", "reach", "linear", "matrix", "diffusive", "fit"])
    if kind == "tree":
        s = _log_int(rng, 200, 1_000_000)
        return {"kind": kind, "segments": s, "steps": rng.randint(1, 24) if s > 20_000 else rng.randint(12, 288),
                "tight": rng.random() < 0.5, "host": rng.random() < 0.5}
    if kind == "basins":
        return {"kind": kind, "basins": rng.randint(3, 64), "segments_lo": rng.randint(50, 1000),
                "segments_hi": _log_int(rng, 2000, 50_000), "steps": rng.randint(3, 24), "tight": rng.random() < 0.7}
    if kind == "ensemble":
        return {"kind": kind, "segments": _log_int(rng, 1000, 40_000), "members": rng.randint(3, 48),
                "steps": rng.randint(4, 16)}
    if kind == "reach":
        r = _log_int(rng, 7, 1_000_000)
        return {"kind": kind, "reaches": r, "segments": r + int(r * rng.uniform(0.3, 1.45)), "tight": rng.random() < 0.5}
    if kind == "linear":
        return {"kind": kind, "segments": _log_int(rng, 500, 2_000_000), "steps": rng.randint(3, 48)}
    if kind == "matrix":
        return {"kind": kind, "reaches": 2 * _log_int(rng, 200, 150_000) - 1, "steps": rng.randint(3, 48)}
    if kind == "diffusive":
        m = rng.choice([64, 120, 257, 500])
        lo = rng.randint(1, 20)
        return {"kind": kind, "reaches": _log_int(rng, 30, 100_000), "max_nodes": m, "lo": lo,
                "hi": rng.randint(lo + 1, m + 1)}
    return {"kind": kind, "pairs": _log_int(rng, 20_000, 800_000), "epochs": rng.randint(1, 2),
            "batch": rng.choice([1024, 4096, 8192])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _tree(seed, segments):
    return synth.make_tree(seed, synth.tree_size(segments), segments, 10)


def _qlat(g, steps, n, dtype):
    """Gamma(2, 0.05) m3/s times a diurnal sine, [steps][n] on the device."""
    u = torch.rand((2, n), generator=g, device="cuda", dtype=torch.float64).clamp_min_(1e-12)
    base = -0.05 * (u[0].log() + u[1].log())
    phase = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    out = torch.empty((steps, n), dtype=dtype, device="cuda")
    for t in range(steps):
        out[t] = base * (1.0 + 0.5 * torch.sin(2 * math.pi * t * DT / 86400.0 + phase))
    return out


def _cfg(tight, **kw):
    return T.make_cfg(**(TIGHT if tight else REF), **kw)


def _spin_up(net, qlat, steps):
    """The developed state a forecast starts from: `steps` steps from the flat state."""
    S, R = net.n_segments, net.n_reaches
    net.set_state(np.full(S, 0.1), np.full(S, 0.1), np.full(R, 0.1))
    net.run_device(qlat.data_ptr(), steps)
    net.sync()
    q, d, _, r = net.get_state()
    return q, d, r


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy()


def _outs(net):
    return tuple(_pinned(n) for n in (net.n_segments, net.n_segments, net.n_segments, net.n_reaches))


def _params32(seed, n):
    return np.ascontiguousarray(synth.make_params(seed, n).view("<f8").reshape(-1, 8), np.float32)


def _diff_reaches(case, g):
    n = case["reaches"]
    rp = np.zeros(n, T.api.DIFF_REACH_DTYPE)
    rp["ncomp"] = torch.randint(case["lo"], case["hi"], (n,), generator=g, device="cuda").cpu().numpy()
    rp["theta"] = 0.6
    rp["dtini"] = 60.0
    return rp


def _pairs(g, n):
    q = torch.exp(1.5 * torch.randn((n, 4), generator=g, device="cuda"))
    u = torch.rand((n, 4), generator=g, device="cuda")
    dx, nn, bw = 500 + 4500 * u[:, 0], 0.03 + 0.05 * u[:, 2], 2 + 48 * u[:, 3]
    s0 = torch.exp(math.log(1e-5) + math.log(1e3) * u[:, 1])
    depth = 0.3 * (q[:, 1] + q[:, 3]) ** 0.6 * (nn / 0.05) ** 0.6 / (bw / 10) ** 0.5 / (s0 / 1e-3) ** 0.3
    return torch.cat([q, torch.stack([dx, s0, nn, bw, depth], 1)], 1).float().contiguous()


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind in ("tree", "basins", "ensemble"):
        steps = case["steps"]
        spin = min(24, max(8, steps))
        if kind == "tree":
            topo = _tree(seed, case["segments"])
            params = synth.make_params(seed, case["segments"])
            net = T.Network(topo, params, dt=DT, cfg=_cfg(case["tight"]))
        elif kind == "basins":
            # sizes spread evenly over the logarithm of their range
            sizes = np.geomspace(case["segments_lo"], case["segments_hi"], case["basins"])
            topos = [_tree(seed * 1000 + i, int(s)) for i, s in enumerate(sizes)]
            params = [synth.make_params(seed * 1000 + i, t["n_segments"]) for i, t in enumerate(topos)]
            topo = None
            net = T.Network(topos, params, dt=DT, cfg=_cfg(case["tight"]))
        else:
            S, M = case["segments"], case["members"]
            topo = _tree(seed, S)
            params = synth.make_params(seed, S)
            base_ql = _qlat(g, max(steps, 18), S, torch.float64)
            base = T.Network(topo, params, dt=DT, cfg=_cfg(True, record_pairs=1))
            base.set_state(np.full(S, 0.1), np.full(S, 0.1), np.full(base.n_reaches, 0.1))
            base.run_device(base_ql.data_ptr(), 18)
            base.sync()
            n = base.pairs()
            buf = torch.empty((n, 9), device="cuda")
            base.pairs(buf.data_ptr(), n)
            base.close()
            model = T.WarmModel(0)
            model.fit(buf.data_ptr(), n, epochs=3)
            qs = torch.exp(0.3 * torch.randn(M * S, generator=g, device="cuda", dtype=torch.float64)).cpu().numpy()
            ns = (0.8 + 0.4 * torch.rand(M * S, generator=g, device="cuda", dtype=torch.float64)).cpu().numpy()
            net = T.Network.ensemble(topo, params, M, n_scale=ns, qlat_scale=qs, dt=DT,
                                     cfg=_cfg(True, warm_start=1))
            net.set_warm_start(model)
        qlat = _qlat(g, max(steps, spin), net.qlat_cols, torch.float64)
        torch.cuda.synchronize()
        q, d, r = _spin_up(net, qlat, spin)
        qlat = qlat[:steps].contiguous()
        return {"kind": kind, "net": net, "topo": topo, "params": params, "q": q, "d": d, "r": r, "steps": steps,
                "qlat": qlat.cpu().numpy() if case.get("host") else qlat, "host": bool(case.get("host")),
                "out": _outs(net), "stream": torch.cuda.Stream()}
    if kind == "reach":
        R, S = case["reaches"], case["segments"]
        extra = torch.randint(0, R, (S - R,), generator=g, device="cuda")
        ln = torch.ones(R, dtype=torch.int64, device="cuda")
        ln += torch.bincount(extra, minlength=R)
        rs = torch.cumsum(ln, 0) - ln
        params = torch.from_numpy(synth.make_params(seed, S).view("<f8").reshape(-1, 8)).cuda()
        ql = _qlat(g, 1, S, torch.float64)[0].contiguous()
        f = torch.rand((3, S), generator=g, device="cuda", dtype=torch.float64)
        qu, qd, dp = 5.0 + 10.0 * f[0], 5.0 + 10.0 * f[1], 0.2 + 1.5 * f[2]
        out = torch.zeros((3, S), dtype=torch.float64, device="cuda")
        return {"kind": kind, "p": params, "ql": ql, "rs": rs.int(), "rl": ln.int(), "qu": qu.contiguous(),
                "qd": qd.contiguous(), "dp": dp.contiguous(), "out": out, "nr": R, "ns": S, "uq": 10.0,
                "cfg": _cfg(case["tight"]), "stream": torch.cuda.Stream()}
    if kind == "linear":
        topo = _tree(seed, case["segments"])
        p32 = _params32(seed, case["segments"])
        coeffs = T.linear_coeffs(p32, DT)
        ql = _qlat(g, case["steps"], case["segments"], torch.float32)
        q0 = torch.rand(case["segments"], generator=g, device="cuda") * 15.0
        return {"kind": kind, "net": T.LinearNetwork(topo, coeffs), "topo": topo, "coeffs": coeffs, "ql": ql, "q0": q0,
                "q": torch.empty_like(q0), "steps": case["steps"], "stream": torch.cuda.Stream()}
    if kind == "matrix":
        R = case["reaches"]
        topo = synth.make_tree(seed, (R + 1) // 2, int(R * 2.4545) + 1, 10)
        coeffs = T.matrix_coeffs(_params32(seed, R), DT)
        net = T.MatrixNetwork(topo["reach_up_ptr"], topo["reach_up_idx"], coeffs)
        ql = _qlat(g, case["steps"], R, torch.float32)
        q0 = 0.1 + torch.rand(R, generator=g, device="cuda") * 15.0
        return {"kind": kind, "net": net, "topo": topo, "coeffs": coeffs, "ql": ql, "q0": q0, "q": torch.empty_like(q0),
                "steps": case["steps"], "stream": torch.cuda.Stream()}
    if kind == "diffusive":
        n, m = case["reaches"], case["max_nodes"]
        rp = torch.from_numpy(_diff_reaches(case, g).view(np.uint8)).cuda()
        u = torch.rand((3, n, m), generator=g, device="cuda")
        return {"kind": kind, "rp": rp, "dx": 100 + 500 * u[0], "df": 10 + 100 * u[1], "qp": 1 + 50 * u[2],
                "out": torch.zeros((n, m), device="cuda"), "scratch": torch.empty(2 * n * m, device="cuda"),
                "n": n, "m": m, "stream": torch.cuda.Stream()}
    return {"kind": kind, "pairs": _pairs(g, case["pairs"]), "n": case["pairs"], "epochs": case["epochs"],
            "batch": case["batch"], "seed": seed}


def _ok(rc):
    if rc:
        raise RuntimeError(T.lib().troute_last_error().decode())


def run(s):
    kind = s["kind"]
    if kind in ("tree", "basins", "ensemble"):
        net = s["net"]
        net.set_state(s["q"], s["d"], s["r"])
        if s["host"]:
            net.run(s["qlat"])
        else:
            net.run_device(s["qlat"].data_ptr(), s["steps"], s["stream"].cuda_stream)
            net.sync()
        return net.get_state(s["out"])
    if kind == "reach":
        o = s["out"]
        _ok(T.lib().troute_mc_reach_parallel_device(
            s["p"].data_ptr(), s["ql"].data_ptr(), s["rs"].data_ptr(), s["rl"].data_ptr(), s["qu"].data_ptr(),
            s["qd"].data_ptr(), s["dp"].data_ptr(), o[0].data_ptr(), o[1].data_ptr(), o[2].data_ptr(), s["uq"], DT,
            s["nr"], s["ns"], C.byref(s["cfg"]), s["stream"].cuda_stream))
        return o
    if kind in ("linear", "matrix"):
        with torch.cuda.stream(s["stream"]):
            s["q"].copy_(s["q0"])
        s["net"].run_device(s["ql"].data_ptr(), s["steps"], s["q"].data_ptr(), stream=s["stream"].cuda_stream)
        return s["q"]
    if kind == "diffusive":
        _ok(T.lib().troute_diffusive_tridiag_device(
            s["rp"].data_ptr(), s["dx"].data_ptr(), s["df"].data_ptr(), None, s["qp"].data_ptr(), s["out"].data_ptr(),
            s["n"], s["m"], s["scratch"].data_ptr(), s["stream"].cuda_stream))
        return s["out"]
    model = T.WarmModel(1)
    loss = model.fit(s["pairs"].data_ptr(), s["n"], epochs=s["epochs"], batch=s["batch"], seed=s["seed"])
    state = model.get_state()
    model.close()
    return {"state": state, "loss": loss}


# ---------------------------------------------------------------------------
# work: every input read once, every output written once; floating operations
# of the solve (about 215 a pass and 4 or 8 passes by the tolerance)
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    per = 215.0 * (8 if case.get("tight", True) else 4)
    if kind in ("tree", "basins", "ensemble"):
        if kind == "tree":
            n = case["segments"]
        elif kind == "basins":
            a, b = math.log(case["segments_lo"]), math.log(case["segments_hi"])
            n = case["basins"] * (math.exp(b) - math.exp(a)) / (b - a)
        else:
            n = case["segments"] * case["members"]
        shared = case["segments"] if kind == "ensemble" else n
        scales = 16 * n if kind == "ensemble" else 0
        return {"bytes": 64 * shared + scales + 8.0 * shared * case["steps"] + 40 * n, "flops": per * n * case["steps"]}
    if kind == "reach":
        return {"bytes": 120.0 * case["segments"] + 8.0 * case["reaches"], "flops": per * case["segments"]}
    if kind == "linear":
        n, t = case["segments"], case["steps"]
        return {"bytes": 4.0 * n * t + 24.0 * n, "flops": 7.0 * n * t}
    if kind == "matrix":
        r, t = case["reaches"], case["steps"]
        return {"bytes": 4.0 * r * t + 24.0 * r, "flops": 9.0 * r * t}
    if kind == "diffusive":
        n = case["reaches"] * (case["lo"] + case["hi"] - 1) / 2.0
        return {"bytes": 16.0 * n + 12.0 * case["reaches"], "flops": 25.0 * n}
    return {"bytes": 36.0 * case["pairs"] * case["epochs"], "flops": 6.0 * 4672 * case["pairs"] * case["epochs"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _geometry(p):
    dx, bw, tw, twcc, n, ncc, cs, s0 = p.unbind(1)
    z = torch.where(cs == 0, torch.ones_like(cs), 1.0 / cs)
    bfd = torch.where(bw > tw, bw / 1e-5, torch.where(bw == tw, bw / (2 * z), (tw - bw) / (2 * z)))
    return torch.stack([dx, bw, twcc, n, ncc, s0, z, bfd])


def _at_depth(h, g):
    dx, bw, twcc, n, ncc, s0, z, bfd = g
    twl = bw + 2 * z * h
    above = (h - bfd).clamp_min(0)
    below = torch.minimum(h, bfd)
    dry = (above > 0) & (twcc <= 0)
    above, below = torch.where(dry, torch.zeros_like(h), above), torch.where(dry, h, below)
    sq = torch.sqrt(1 + z * z)
    wp = bw + 2 * below * sq
    wpc = torch.where(above > 0, twcc + 2 * above, torch.zeros_like(h))
    a = (bw + below * z) * below + twcc * above
    p = wp + wpc
    R = torch.where(p > 0, a / p, torch.zeros_like(h))
    r23, r53 = R ** (2.0 / 3.0), R ** (5.0 / 3.0)
    ck = torch.sqrt(s0) / n * (5.0 / 3.0 * r23 - 2.0 / 3.0 * r53 * (2 * sq / (bw + 2 * z * h)))
    ck = torch.where(h > 0, ck.clamp_min(0), torch.zeros_like(h))
    km = torch.where(ck > 0, (dx / ck).clamp_min(DT), torch.full_like(h, DT))
    tw = torch.where((h > bfd) & (twcc > 0), twcc, twl)
    qmn = torch.where(p > 0, 1.0 / ((wp * n + wpc * ncc) / p) * a * r23 * torch.sqrt(s0), torch.zeros_like(h))
    return ck, km, tw, qmn


def _coeffs(e, q, lo, g, fl):
    ck, km, tw, _ = e
    den = tw * g[5] * ck * g[0]
    X = torch.where((ck > 0) & (den > 0), (0.5 * (1 - q / (2 * den))).clamp(lo, 0.5), torch.full_like(q, 0.5))
    D = km * (1 - X) + DT / 2
    D = torch.where(D == 0, torch.ones_like(D), D)
    return (km * X + DT / 2) / D, (DT / 2 - km * X) / D, (km * (1 - X) - DT / 2) / D, fl[3] * DT / D


def _solve64(qup, quc, qdp, ql, g, depth, rtol, atol):
    """Discharge, velocity and depth of one segment step (the secant on depth)."""
    out = torch.zeros((3, qup.numel()), dtype=torch.float64, device=qup.device)
    ok = (g[3] > 0) & (g[5] > 0) & (g[6] > 0) & (g[1] > 0) & ~((ql <= 0) & (qup <= 0) & (quc <= 0) & (qdp <= 0))
    at = torch.nonzero(ok).flatten()
    fl = torch.stack([qup, quc, qdp, ql])[:, at]
    g = g[:, at]
    d = depth[at].clamp_min(0)
    z = torch.zeros_like(d)
    # rows: h, h_0, Qj_0, iter, maxiter, attempt
    st = torch.stack([d * 1.33 + 0.01, d * 0.67, z, z, z + 100, z])
    while at.numel():
        h, h0 = st[0], st[1]
        e0 = _at_depth(h0, g)
        c = _coeffs(e0, st[2], 0.0, g, fl)
        qm = c[0] * fl[0] + c[1] * fl[1] + c[2] * fl[2] + c[3]
        qj0 = qm - e0[3]
        e1 = _at_depth(h, g)
        k = list(_coeffs(e1, qm, 0.25, g, fl))
        s3 = k[0] * fl[0] + k[1] * fl[1] + k[2] * fl[2]
        k[3] = torch.where((k[3] < 0) & (k[3].abs() > s3), -s3, k[3])
        q = s3 + k[3]
        qj = q - e1[3]
        dq = qj0 - qj
        h1 = torch.where(dq != 0, h - qj * (h0 - h) / torch.where(dq != 0, dq, torch.ones_like(dq)), h)
        h1 = torch.where(h1 < 0, h, h1)
        pos = h > 0
        aerr = torch.where(pos, (h1 - h).abs(), torch.full_like(h, 0.9))
        rerr = torch.where(pos, ((h1 - h) / torch.where(pos, h, torch.ones_like(h))).abs(), torch.zeros_like(h))
        it, mx, att = st[3] + 1, st[4], st[5]
        h0, h = h.clamp_min(0), h1.clamp_min(0)
        stop = (h < 0.01) | ~((rerr > rtol) & (aerr >= atol) & (it <= mx))
        widen = stop & (it >= mx)
        h, h0 = torch.where(widen, h * 1.33, h), torch.where(widen, h0 * 0.67, h0)
        mx, att = mx + 25 * widen, att + widen
        again = widen & (att < 5)
        it = torch.where(again, torch.zeros_like(it), it)
        done = stop & ~again
        neg = torch.where((k[3] < 0) & (k[3].abs() > s3), torch.zeros_like(q),
                          torch.maximum(k[0] * fl[0] + k[1] * fl[1] + k[3], k[0] * fl[0] + k[2] * fl[2] + k[3]))
        q = torch.where(q < 0, neg, q)
        bw, twl = g[1], g[1] + 2 * g[6] * h
        R = (h * (bw + twl) / 2) / (bw + 2 * torch.sqrt(((twl - bw) / 2) ** 2 + h * h))
        v = R.clamp_min(0) ** (2.0 / 3.0) / g[3] * torch.sqrt(g[5])
        out[:, at[done]] = torch.stack([q, v, h])[:, done]
        go = ~done
        st = torch.stack([h, h0, qj0, it, mx, att])[:, go]
        g, fl, at = g[:, go], fl[:, go], at[go]
    return out


def _levels(up_ptr, up_idx):
    R = len(up_ptr) - 1
    left = np.diff(up_ptr).astype(np.int64)
    down = np.full(R, -1, np.int64)
    down[up_idx] = np.repeat(np.arange(R), left)
    level, front, k = np.zeros(R, np.int64), np.nonzero(left == 0)[0], 0
    while len(front):
        level[front] = k
        d = down[front]
        d, n = np.unique(d[d >= 0], return_counts=True)
        left[d] -= n
        front, k = d[left[d] == 0], k + 1
    return level


def _route64(topo, steps, out0, device, segment):
    """Routes `steps` steps wave by wave (wave = step + level): segment(s, t, qup,
    quc) advances the segments s at steps t and returns (old, new) discharge."""
    up_ptr = topo["reach_up_ptr"].astype(np.int64)
    up_idx = np.asarray(topo["reach_up_idx"], np.int64)
    R = len(up_ptr) - 1
    level = _levels(up_ptr, up_idx)
    order = np.argsort(level, kind="stable")
    first = np.searchsorted(level[order], np.arange(level.max() + 2))
    n_up = np.diff(up_ptr)
    width = int(n_up.max()) if R else 0
    ups = np.full((R, width), R, np.int64)
    for j in range(width):
        has = n_up > j
        ups[has, j] = up_idx[up_ptr[:-1][has] + j]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)  # noqa: E731
    ups, start, ln, level_t, order_t = dev(ups), dev(topo["reach_seg_start"].astype(np.int64)), dev(
        topo["reach_seg_len"].astype(np.int64)), dev(level), dev(order)
    hist = torch.zeros((steps + 1, R + 1), dtype=torch.float64, device=device)
    hist[0, :R] = out0
    for w in range(steps + int(level.max())):
        a, b = first[max(0, w - steps + 1)], first[min(int(level.max()), w) + 1]
        r = order_t[a:b]
        if not r.numel():
            continue
        t = w - level_t[r]
        qup = hist[t[:, None], ups[r]].sum(1)
        quc = hist[t[:, None] + 1, ups[r]].sum(1)
        i = 0
        while r.numel():
            s = start[r] + i
            qup, quc = segment(s, t, qup, quc)
            i += 1
            last = ln[r] == i
            hist[t[last] + 1, r[last]] = quc[last]
            if bool(last.all()):
                break
            more = ~last
            r, t, qup, quc = r[more], t[more], qup[more], quc[more]
    return hist


def _mix(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _hash(seed, stream, ctr):
    m = (1 << 64) - 1
    return _mix((_mix(seed ^ _mix((stream * 0xD1B54A32D192ED03) & m)) + ctr) & m)


def _fit64(case, seed):
    """The training run in 64 bits: initial weights, shuffles and AdamW as documented."""
    pairs = prepare(case, seed)["pairs"]
    n, batch = case["pairs"], case["batch"] // 64 * 64
    raw = pairs.double()
    raw[:, :4] = (pairs[:, :4] + 1e-3).double()
    lg = raw.log()
    stat = lg[:: max(1, n // 4_000_000 if n > 4_000_000 else 1)]
    mu, sd = stat.mean(0), stat.std(0, unbiased=False)
    x = (lg - mu.float().double()) / sd.float().double()
    sizes = [512, 64, 4096, 64, 64, 1]
    scale = [math.sqrt(6 / 8), 0.0, math.sqrt(6 / 64), 0.0, math.sqrt(6 / 64), 0.0]
    w, i = [], 0
    for k, m in enumerate(sizes):
        u = [((_hash(1, 777, i + j) >> 11) + 0.5) / 2.0 ** 53 * 2 - 1 for j in range(m)] if scale[k] else [0.0] * m
        w.append(torch.tensor(u, dtype=torch.float64, device="cuda").mul_(scale[k] * 0.5).float().double())
        i += m
    w[0], w[2] = w[0].view(64, 8), w[2].view(64, 64)
    w = [p.requires_grad_(True) for p in w]
    m1, m2 = [torch.zeros_like(p) for p in w], [torch.zeros_like(p) for p in w]
    per = -(-n // batch)
    total, step, losses = per * case["epochs"], 0, []
    for ep in range(case["epochs"]):
        a = (_hash(seed, 31, ep) | 1) % n or 1
        while math.gcd(a, n) != 1:
            a = (a + 1) % n or 1
        b = _hash(seed, 37, ep) % n
        # (a i + b) mod n in 64 unsigned bits wraps only past 2^64: a, i < n <= 2^31
        perm = (a * torch.arange(n, device="cuda") + b) % n
        loss_sum = torch.zeros((), dtype=torch.float64, device="cuda")
        for k in range(per):
            d = x[perm[k * batch:(k + 1) * batch]]
            z = torch.nn.functional.silu(torch.nn.functional.silu(d[:, :8] @ w[0].T + w[1]) @ w[2].T + w[3]) @ w[4] + w[5]
            s = 0.5 * (z - d[:, 8]).square().sum()
            loss_sum += s.detach()
            grad = torch.autograd.grad(s / d.shape[0], w)
            lr = 2e-3 * 0.5 * (1 + math.cos(math.pi * step / max(1, total - 1)))
            step += 1
            with torch.no_grad():
                for j, (p, gr) in enumerate(zip(w, grad)):
                    m1[j].mul_(0.9).add_(gr, alpha=0.1)
                    m2[j].mul_(0.999).addcmul_(gr, gr, value=0.001)
                    if scale[j]:
                        p.mul_(1 - lr * 1e-4)
                    p -= lr * (m1[j] / (1 - 0.9 ** step)) / ((m2[j] / (1 - 0.999 ** step)).sqrt() + 1e-8)
        losses.append(loss_sum / n)
    flat = torch.cat([p.detach().reshape(-1) for p in w] + [mu[:8], sd[:8], mu[8:], sd[8:]])
    return {"state": flat, "loss": torch.stack(losses)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("basins", "ensemble") or (kind == "tree" and (case["tight"] or case["segments"] * case["steps"] > 400_000)):
        return None   # at 1e-8 the stopping depth of a long run depends on every rounding; longer runs take minutes
    s = prepare(case, seed)
    if kind == "tree":
        dev = "cpu"
        g = _geometry(torch.from_numpy(np.ascontiguousarray(s["params"]).view("<f8").reshape(-1, 8).copy()))
        q, d = torch.from_numpy(s["q"].copy()), torch.from_numpy(s["d"].copy())
        v = torch.zeros_like(q)
        qlat = torch.as_tensor(s["qlat"]).cpu()

        def segment(i, t, qup, quc):
            old = q[i]
            r = _solve64(qup, quc, old, qlat[t, i], g[:, i], d[i], REF["rtol"], REF["atol"])
            q[i], v[i], d[i] = r[0], r[1], r[2]
            return old, r[0]

        hist = _route64(s["topo"], case["steps"], torch.from_numpy(s["r"].copy()), dev, segment)
        return q, d, v, hist[-1, :-1]
    if kind == "reach":
        g = _geometry(s["p"])
        tol = TIGHT if case["tight"] else REF
        out = torch.zeros_like(s["out"])
        r = torch.arange(s["nr"], device="cuda")
        quc = torch.full((s["nr"],), s["uq"], dtype=torch.float64, device="cuda")
        i = 0
        while r.numel():
            at = (s["rs"][r] + i).long()
            x = _solve64(s["qu"][at], quc, s["qd"][at], s["ql"][at], g[:, at], s["dp"][at], tol["rtol"], tol["atol"])
            out[:, at] = x
            i += 1
            more = s["rl"][r] > i
            r, quc = r[more], x[0][more]
        return out
    if kind in ("linear", "matrix"):
        topo = s["topo"]
        if kind == "matrix":   # one routing unit per reach
            R = case["reaches"]
            topo = dict(topo, reach_seg_start=np.arange(R), reach_seg_len=np.ones(R, np.int64))
        c = [torch.from_numpy(np.asarray(x, np.float64)).cuda() for x in s["coeffs"]]
        q, ql = s["q0"].double(), s["ql"]

        def segment(i, t, qup, quc):
            old = q[i]
            new = c[0][i] * quc + c[1][i] * qup + c[2][i] * old + c[3][i] * ql[t, i].double()
            q[i] = new
            return old, new

        last = torch.from_numpy(np.asarray(topo["reach_seg_start"]).astype(np.int64) + topo["reach_seg_len"] - 1).cuda()
        _route64(topo, case["steps"], q[last].clone(), "cuda", segment)
        return q
    if kind == "diffusive":
        rp = _diff_reaches(case, _gen(seed))
        n, m = case["reaches"], case["max_nodes"]
        nc = torch.from_numpy(rp["ncomp"].astype(np.int64)).cuda()
        th, dt = float(np.float32(0.6)), 60.0
        dx, df, qp = s["dx"].double().clamp_min(1.0), s["df"].double().clamp_min(0.01), s["qp"].double()
        top = int(nc.max())
        E = torch.zeros((top, n), dtype=torch.float64, device="cuda")
        F = torch.zeros_like(E)
        E[0] = 1.0
        for i in range(1, top):
            h2 = dx[:, i - 1] ** 2
            p = -th * df[:, i] * dt / h2
            nxt = torch.where(i < nc - 1, qp[:, min(i + 1, m - 1)], qp[:, i])
            rhs = qp[:, i] + dt * df[:, i] * (1 - th) * (qp[:, i - 1] - 2 * qp[:, i] + nxt) / h2
            den = p * E[i - 1] + 1 - 2 * p
            E[i], F[i] = -p / den, (rhs - p * F[i - 1]) / den
        out = torch.zeros((n, m), dtype=torch.float64, device="cuda")
        cur = qp.gather(1, (nc - 1)[:, None])[:, 0]   # the ghost node's value
        for i in range(top - 1, -1, -1):
            inside = i < nc
            cur = torch.where(inside, E[i] * cur + F[i], cur)
            out[:, i] = torch.where(inside, cur, out[:, i])
        return out
    return _fit64(case, seed)

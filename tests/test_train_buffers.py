"""The training launches' device buffers over calls of different shapes on one
model. CPU: the sizing code itself (train_buffers.h) with cudaMalloc and cudaFree
that only keep count, against what the kernels index. GPU: a model fitted twice
with different batches and asked for a gradient equals a fresh one bit for bit."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

PROG = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
static std::map<void*, size_t> live;
static long allocs = 0, fail_at = -1;
#include "train_buffers.h"
extern "C" cudaError_t cudaMalloc(void** p, size_t bytes)
{
    if (allocs++ == fail_at) return cudaErrorMemoryAllocation;
    live[*p = std::malloc(1)] = bytes;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFree(void* p)
{
    if (!live.erase(p)) std::abort();
    std::free(p);
    return cudaSuccess;
}
int main(int argc, char** argv)   // [allocation that fails] then "f pairs batch" or "g pairs" lines
{
    if (argc > 1) fail_at = std::atol(argv[1]);
    {
        tr::TrainBuffers b;
        char what;
        long long n;
        while (std::scanf(" %c %lld", &what, &n) == 2) {
            int batch = (int)n, steps = 1;
            if (what == 'f') {
                if (std::scanf("%d", &batch) != 1) return 1;
                batch = batch / tr::kTrainRows * tr::kTrainRows;
                steps = tr::train_steps_kept((n + batch - 1) / batch, batch / tr::kTrainRows);
            }
            const int tiles = (batch + tr::kTrainRows - 1) / tr::kTrainRows;
            const int rc = b.reserve(tiles, steps);
            auto bytes = [](void* p) { return p ? live.at(p) : 0; };
            std::printf("%d %d %d %zu %zu %zu %zu\n", rc, tiles, steps, bytes(b.part.p), bytes(b.err.p), bytes(b.loss.p),
                        bytes(b.step.p));
        }
    }
    return live.empty() ? 0 : 2;
}
"""

CALLS = {
    "batch_8192_then_1024": ["f 1000000 8192", "f 800000 1024"],
    "batch_8192_then_64": ["f 1000000 8192", "f 500000 64"],
    "many_small_batches_then_gradient": ["f 4300000 64", "g 4300000"],
    "gradient_then_many_steps": ["g 4300000", "f 4000000 64", "f 1000000 8192"],
    "one_tile": ["f 2 64", "g 1", "f 65 64", "g 65", "f 2 128"],
}


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    d = tmp_path_factory.mktemp("train_buffers")
    src, exe = str(d / "t.cpp"), str(d / "t")
    open(src, "w").write(PROG)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "noaa-gpu-kernels_gb300", "csrc"), "-I",
                    os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), src, "-o", exe], check=True)

    def run(calls, *args):
        r = subprocess.run([exe, *args], input="\n".join(calls), capture_output=True, text=True, check=True)   # 2: a leak
        return [[int(x) for x in line.split()] for line in r.stdout.splitlines()]

    return run


def rows_of(calls):
    rng = np.random.default_rng(3)
    if calls != "random":
        return CALLS[calls]
    pairs = lambda: int(2 ** rng.uniform(1, 22))
    return [f"g {pairs()}" if rng.random() < 0.3 else f"f {pairs()} {int(2 ** rng.uniform(6, 16))}" for _ in range(200)]


def check(row):
    rc, tiles, steps, part, err, loss, step = row
    assert rc == 0
    assert part >= tiles * 4804 * 4           # a row of gradients a tile
    assert err >= steps * tiles * 64 * 4      # a float a sample of every tile of every step
    assert loss >= (steps * tiles + steps) * 8
    assert step >= steps * 12


@pytest.mark.parametrize("calls", [*CALLS, "random"])
def test_every_call_has_room(sizes, calls):
    rows = sizes(rows_of(calls))
    assert len(rows) == len(rows_of(calls))
    for row in rows:
        check(row)


@pytest.mark.parametrize("fails", range(8))
def test_a_failed_allocation_leaves_no_size_behind(sizes, fails):
    calls = ["f 1000000 8192", "f 4000000 64", "g 100000", "g 100000", "f 4000000 64", "f 1000000 8192"]
    rows = sizes(calls, str(fails))
    assert [r[0] != 0 for r in rows].count(True) <= 1
    for row in rows:
        if row[0] == 0:
            check(row)


@pytest.mark.gpu
@pytest.mark.parametrize("first,second", [((100_000, 8192), (80_000, 1024)), ((100_000, 8192), (50_000, 64)),
                                          ((70_000, 64), (70_000, 8192))])
def test_a_reused_model_equals_a_fresh_one(first, second):
    torch = pytest.importorskip("torch")
    import troute_gb300 as T

    g = torch.Generator(device="cuda").manual_seed(1)
    n = 100_000
    q = torch.exp(torch.randn((n, 4), generator=g, device="cuda"))
    u = torch.rand((n, 4), generator=g, device="cuda")
    pairs = torch.cat([q, torch.stack([500 + 4500 * u[:, 0], 1e-5 + 1e-2 * u[:, 1], 0.03 + 0.05 * u[:, 2], 2 + 48 * u[:, 3],
                                       0.3 * q[:, 1] ** 0.6 + 0.1], 1)], 1).float().contiguous()
    host = pairs.cpu().numpy()
    used = T.WarmModel(3)
    used.fit(pairs.data_ptr(), first[0], epochs=1, batch=first[1], seed=5)
    for k in (n, 65, n):   # a gradient of many pairs, of few, then fits and gradients again
        fresh = T.WarmModel(4)
        fresh.set_state(used.get_state())
        a, b = used.grad(host[:k]), fresh.grad(host[:k])
        np.testing.assert_array_equal(a[0], b[0])
        assert a[1] == b[1]
        losses = [m.fit(pairs.data_ptr(), second[0], epochs=2, batch=second[1], seed=7) for m in (used, fresh)]
        np.testing.assert_array_equal(losses[0], losses[1])
        np.testing.assert_array_equal(used.get_state(), fresh.get_state())

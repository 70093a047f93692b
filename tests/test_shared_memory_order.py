"""Shared memory that one lane writes and another reads has a barrier or fence in
between. A converged warp does not show its absence, so the source is read."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "noaa-gpu-kernels_gb300", "csrc")


def function(file, name):
    """Text of a function's body, without comments."""
    src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, file)).read(), flags=re.S)
    at = src.index("{", re.search(rf"\b{name}\s*\([^;{{]*\)\s*\{{", src).start())
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i]


def test_narrow_passes_read_other_lanes_buffers_between_barriers():
    body = function("narrow_pass.cuh", "narrow_passes")
    reads = [m.start() for m in re.finditer(r"warp_seg|staged_seg\(rec\)|\*c[12]\b", body)]
    # the last access is the owner's own buffer, after everybody's reads
    own = body.index("staged_seg(warp_seg + lane")
    reads = [r for r in reads if r < own]
    barriers = [m.start() for m in re.finditer(r"__syncwarp\(\);", body)]
    assert len(reads) >= 4
    assert any(b < min(reads) for b in barriers), "no barrier before the first read of another lane's buffer"
    assert any(max(reads) < b < body.index("return") for b in barriers), "no barrier between the reads and the return"


def test_deep_paths_ring_is_handed_over_behind_fences():
    """Both flags of the ring: a fence between the accesses and the raising of the
    flag, and one between the seen flag and the accesses."""
    wait = function("linear.cu", "wait_smem")
    assert re.search(r"while.*\}\s*\}\s*__threadfence_block\(\);\s*return __all_sync", wait, re.S)
    body = function("linear.cu", "lin_deep_kernel")
    for flag in (r"R\.rounds = i;", r"R\.full\[b %"):
        assert re.search(r"__syncwarp\(\);\s*__threadfence_block\(\);\s*if \(c == 0\) " + flag, body), flag

"""Kernels that are launched while their predecessor still runs (grid_begin, csrc/common.cuh) take no const __restrict__
parameters (CPU, on the sources): the compiler may read those through the read-only path, which asks for data that nothing
writes while the kernel is resident, and the predecessor may write them until grid_begin returns."""
import glob
import os
import re

import __graft_entry__ as entry

KERNEL = re.compile(r"__global__ void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\s*\(([^)]*)\)\s*\{")


def _kernels():
    for path in sorted(glob.glob(os.path.join(entry.PKG_DIR, "csrc", "*.cu*"))):
        src = open(path).read()
        for m in KERNEL.finditer(src):
            end, depth = m.end(), 1
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            yield m.group(1), m.group(2), src[m.end():end]


def test_early_launched_kernels_take_no_read_only_parameters():
    early = [(name, params) for name, params, body in _kernels() if "grid_begin();" in body]
    assert len(early) >= 12  # the chain of a try, the per-call kernels, the read-back
    for name, params in early:
        assert not re.search(r"const [\w ]+\* *__restrict__", params), name

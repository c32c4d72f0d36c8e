"""Every kernel that the launch helper `chained` may start before the one in
front of it has finished opens with `chain_wait()`: without it the kernel
would read what is still being written, and the kernels after it too."""
from __future__ import annotations

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2dfmm_gb300", "csrc")
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*"
                    r"\((?:[^()]|\([^()]*\))*\)\s*\{\s*(\w+)")


def test_chained_kernels_wait_first():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            src = f.read()
        first = dict(KERNEL.findall(src))
        direct = set(re.findall(r"chained\((k_\w+)", src))
        # launches through a variable: any kernel of the file may be behind it
        if re.search(r"chained\((?!k_)\w+", src):
            direct |= set(first)
        for name in direct:
            assert first.get(name) == "chain_wait", f"{os.path.basename(path)}: {name}"
        seen += len(direct)
        assert len(first) == src.count("__global__ void"), path  # every kernel was parsed
    assert seen > 50

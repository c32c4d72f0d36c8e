"""Device memory per form: only plain solves that sum in fixed point hold the
coefficients a second time."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import ROOT

CHILD = """
import importlib, sys
import torch
sys.path.insert(0, {root!r})
P = importlib.import_module("2dfmm_gb300")
P.load()
n = 400_000
g = torch.Generator(device="cuda")
g.manual_seed(1)
xy = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
cir = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
cor, uv = torch.full_like(cir, 1e-3), torch.empty_like(xy)
P.set_mode({mode})
P.set_mixed_leaf(4)

def held(nterms):
    P.set_params(nterms, 5, {theta})
    P.solve_device(xy.data_ptr(), cir.data_ptr(), cor.data_ptr(), uv.data_ptr(), n)
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free

small = held(2)
print((held(32) - small) / (30 * 16 * P.stats()["n_cells"]))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("mode,theta,arrays", [("P.MODE_PLAIN", 0.5, 2), ("P.MODE_PLAIN", 0.9, 1), ("P.MODE_MIXED", 0.5, 1),
                                               ("P.MODE_LEARNED", 0.5, 1)])
def test_arrays_of_coefficients(gpu_lib, mode, theta, arrays):
    """Memory that 30 more coefficients per cell take, in arrays of them: one
    (two with the fixed-point ones), an arena's spare eighth, and what the
    allocator rounds up."""
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, mode=mode, theta=theta)], capture_output=True,
                       text=True, env=dict(os.environ), timeout=300)
    assert p.returncode == 0, p.stderr
    grown = float(p.stdout.split()[-1])
    assert arrays * 0.9 <= grown <= arrays * 1.125 * 32 / 30 + 0.1, grown

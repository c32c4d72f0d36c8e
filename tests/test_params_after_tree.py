"""The parameters a tree was built with go with it: queries answer by the last
make_tree, whatever is set between the two (the reference reads its parameters
in make_tree only, ver-c/src/quadtree.c:12-27)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import oracle, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["plain", "mixed"])
@pytest.mark.parametrize("built", [(5, 33, 0.5), (13, 17, 0.9)])
def test_queries_use_the_parameters_of_the_tree(gpu_lib, mode, built):
    """Points off the blobs after other parameters are set (more and fewer
    terms, other angles and leaf sizes), by batches and one by one, first and
    later queries: bit for bit the answers without the change."""
    P = gpu_lib
    b = workloads().uniform(3000, seed=21)
    rng = np.random.default_rng(3)
    pts = np.concatenate([rng.uniform(-0.2, 1.2, (1500, 2)), [[30.0, 4.0], [-200.0, 7.0]]])
    P.set_mode(P.MODE_PLAIN if mode == "plain" else P.MODE_MIXED)
    try:
        P.set_params(*built)
        P.make_tree(b.xy, b.cir, b.cor)
        uv = P.biot_tree_batch(pts)
        for other in [(32, 500, 0.3), (2, 5, 0.7), (32, 17, 1.5), (0, 65536, 0.5)]:
            P.set_params(*built)
            P.make_tree(b.xy, b.cir, b.cor)
            P.set_params(*other)
            assert np.array_equal(P.biot_tree_batch(pts).view(np.uint64), uv.view(np.uint64)), other
            assert P.biot_tree(*pts[7]) == tuple(uv[7]), other
            P.set_params(*built)
            assert np.array_equal(P.biot_tree_batch(pts[:900]), uv[:900]), other
    finally:
        P.clear_params()
        P.set_mode(P.MODE_PLAIN)


@pytest.mark.gpu
def test_opening_angle_of_minus_one(gpu_lib):
    """An angle below zero opens every cell (region > theta r always): the
    direct sum over the blobs."""
    P = gpu_lib
    b = workloads().uniform(1500, seed=22)
    P.set_params(9, 33, -1.0)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(b.xy, b.cir, b.cor)
        uv = P.biot_tree_batch(b.xy)
    finally:
        P.clear_params()
    ref = oracle().direct(b.xy, b.xy, b.cir, b.cor)
    assert np.abs(uv - ref).max() <= 1e-12 * np.abs(ref).max()

"""Mixed trees whose leaves are larger than a stage buffer of the near field."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import oracle, workloads


@pytest.mark.gpu
@pytest.mark.parametrize("cores", ["one", "several"])
@pytest.mark.parametrize("leaf,n", [(128, 8192), (129, 8192), (300, 4097), (300, 70_000), (1000, 12_345)])
def test_variants_around_the_stage_buffer(gpu_lib, leaf, n, cores):
    """Every near-field variant gives the same bits for leaves up to, just
    beyond and far beyond 128 blobs, with one core radius and with several,
    and they are within 1e-6 of the direct sum."""
    P = gpu_lib
    b = workloads().lamb_oseen(n, seed=leaf)
    rng = np.random.default_rng(leaf)
    cor = b.cor if cores == "one" else b.cor * rng.uniform(0.5, 1.0, n)
    P.set_params(13, 65, 0.5)
    P.set_mode(P.MODE_MIXED)
    P.set_mixed_params()
    P.set_mixed_leaf(leaf)
    uv = []
    try:
        for v in range(5):
            P.set_tuning(False, v)
            P.make_tree(b.xy, b.cir, cor)
            uv.append(P.biot_tree_batch(b.xy))
            assert P.stats()["eval_variant"] == v
    finally:
        P.set_tuning()
        P.set_mixed_leaf()
        P.clear_params()
        P.set_mode(P.MODE_PLAIN)
    for v in range(1, 5):
        assert np.array_equal(uv[v].view(np.uint64), uv[0].view(np.uint64)), v
    idx = rng.choice(n, 300, replace=False)
    ref = oracle().direct(b.xy[idx], b.xy, b.cir, cor)
    assert np.linalg.norm(uv[4][idx] - ref) <= 1e-6 * np.linalg.norm(ref)

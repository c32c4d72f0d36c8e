"""The tables of the blobs by position: the hash of csrc/position_hash.h (the
same code compiled for the host) spreads positions along the diagonals and in
symmetric pairs as well as any others, and the device table finds such blobs."""
from __future__ import annotations

import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

from conftest import oracle

HERE = os.path.dirname(os.path.abspath(__file__))
U = ctypes.POINTER(ctypes.c_uint64)


@pytest.fixture(scope="module")
def hashes(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("position_hash") / "position_hash.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "position_hash_shim.cpp")], check=True)
    fn = ctypes.CDLL(so).position_hashes

    def of(xy):
        xy = np.ascontiguousarray(xy, np.float64)
        out = np.empty(len(xy), np.uint64)
        fn(len(xy), xy.view(np.uint64).ctypes.data_as(U), out.ctypes.data_as(U))
        return out
    return of


def positions(kind, n):
    rng = np.random.default_rng(6)
    t = rng.uniform(-1, 1, n)
    if kind == "diagonal":
        return np.stack([t, t], axis=1)
    if kind == "antidiagonal":
        return np.stack([t, -t], axis=1)
    if kind == "mirrored":
        p = rng.uniform(-1, 1, (n // 2, 2))
        return np.concatenate([p, p[:, ::-1]])
    if kind == "lattice":
        k = np.arange(math.isqrt(n)) / 8.0
        return np.stack(np.meshgrid(k, k), axis=-1).reshape(-1, 2)
    if kind == "row":
        return np.stack([np.arange(n) * 1e-3, np.full(n, 0.5)], axis=1)
    return rng.uniform(-1, 1, (n, 2))


@pytest.mark.parametrize("kind", ["diagonal", "antidiagonal", "mirrored", "lattice", "row", "random"])
def test_positions_spread_over_the_slots(hashes, kind):
    """n positions in a table of 2n to 4n slots: as many slots are hit first as
    by independent draws (a deviation of 6 standard deviations, at most
    sqrt(n) / 2, would be chance once in 10^8)."""
    p = positions(kind, 20_000)
    n = len(p)
    cap = 1 << (2 * n - 1).bit_length()
    h = hashes(p)
    assert len(np.unique(h)) == n
    hit = len(np.unique(h & np.uint64(cap - 1)))
    expected = cap * -math.expm1(n * math.log1p(-1.0 / cap))
    assert abs(hit - expected) <= 3.0 * math.sqrt(n), (kind, hit, expected)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["diagonal", "mirrored"])
def test_blobs_on_the_diagonal_are_found(gpu_lib, kind):
    """Permuted queries at the blobs answer with the blobs' own velocities, bit
    for bit, and points beside them are evaluated."""
    P = gpu_lib
    n = 4096
    xy = positions(kind, n)
    rng = np.random.default_rng(7)
    cir, cor = rng.standard_normal(n) / n, np.full(n, 0.01)
    P.set_params(11, 33, 0.5)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(xy, cir, cor)
        own = P.biot_tree_batch(xy)
        order = rng.permutation(n)
        beside = xy[:100] + [0.0, 1e-3]
        uv = P.biot_tree_batch(np.concatenate([xy[order], beside]))
    finally:
        P.clear_params()
    assert np.array_equal(uv[:n].view(np.uint64), own[order].view(np.uint64))
    o = oracle().Oracle(11, 33, 0.5)
    o.make_tree(xy, cir, cor)
    ref = o.biot(beside)
    assert np.abs(uv[n:] - ref).max() <= 1e-12 * np.abs(ref).max()

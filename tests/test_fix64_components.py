"""Each component of the regularised pair and of its sums keeps the accuracy of
its own terms, however small beside the other: blobs nearly in a row along an
axis (csrc/fix64.cuh; fmm.c:121-142 forms the two products apart)."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_direct_gpu import run_direct
from test_fix64 import U, dp, tables  # noqa: F401  (the fixture)

L = np.longdouble
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def pair_sum(tmp_path_factory, tables):  # noqa: F811
    so = str(tmp_path_factory.mktemp("fix64c") / "fix64c.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "fix64_components_shim.cpp")], check=True, cwd=ROOT)
    fn = ctypes.CDLL(so).pair_sum

    def of(dx, dy, g, ic):
        a = [np.ascontiguousarray(v, np.float64) for v in (dx, dy, g, ic)]
        out = np.empty(2)
        fn(len(a[0]), *[dp(v) for v in a], tables[0].ctypes.data_as(U), tables[1].ctypes.data_as(U), dp(out))
        return out
    return of


def terms(dx, dy, g, ic):
    """The exact terms (-dy, dx) G (1 - exp(-r^2 ic)) / r^2 and their point-vortex values."""
    r2 = L(1) * dx * dx + L(1) * dy * dy
    e = -np.expm1(-r2 * ic)
    f = g / r2
    d = np.stack([-L(1) * dy, L(1) * dx], axis=1)
    return (f * e)[:, None] * d, f[:, None] * d


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("ratio", [1.0, 1e-2, 1.3e-3, 1.3e-5, 1.3e-7, 1.3e-9, 1.3e-12, 1.3e-18, 1e-30, 1e-150, 1e-300, 5e-324, 0.0])
def test_component_of_one_pair(pair_sum, ratio, swap):
    """Within 2^-52 of each component, besides 2^-55 in the bracket."""
    rng = np.random.default_rng(17)
    for i in range(300):
        big = rng.uniform(0.5, 1.0) * rng.choice([-1, 1])
        small = ratio * rng.uniform(0.5, 1.0) * rng.choice([-1, 1])
        dx, dy = (small, big) if swap else (big, small)
        a = [np.array([v]) for v in (dx, dy, rng.standard_normal(), np.exp(rng.uniform(-8, 8)))]
        t, v = terms(*a)
        err = np.abs(pair_sum(*a) - t[0])
        assert (err <= np.abs(t[0]) * 2.0**-52 + np.abs(v[0]) * 2.0**-55 + L(2.0**-1074)).all(), (dx, dy)


@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("width", [0.3, 1e-3, 1e-6, 1e-9, 1e-12, 1e-18, 1e-40])
def test_component_of_a_row(pair_sum, width, swap):
    """The sum over 700 blobs within `width` of an axis, strengths over 20
    binades: within 2^-52 of each component's terms' magnitudes."""
    rng = np.random.default_rng(int(-np.log10(width)))
    n = 700
    dx, dy = rng.uniform(-1, 1, n), width * rng.standard_normal(n)
    g = rng.standard_normal(n) * np.exp2(rng.uniform(-20, 0, n))
    ic = np.full(n, 1.0 / 0.01**2)
    if swap:
        dx, dy = dy, dx
    t, v = terms(dx, dy, g, ic)
    bound = np.abs(t).sum(axis=0) * 2.0**-52 + np.abs(v).sum(axis=0) * 2.0**-55
    assert (np.abs(pair_sum(dx, dy, g, ic) - t.sum(axis=0)) <= bound).all()


def sheet(n, width, vertical):
    rng = np.random.default_rng(n)
    x, y = np.sort(rng.uniform(0, 1, n)), 0.375 + width * rng.standard_normal(n)
    xy = np.stack([x, y] if not vertical else [y, x], axis=1)
    return xy, rng.standard_normal(n) / n, np.full(n, 0.01)


@pytest.mark.gpu
@pytest.mark.parametrize("vertical", [False, True])
@pytest.mark.parametrize("width", [1e-3, 1e-7, 1e-11, 1e-15, 0.0])
def test_sheet_along_an_axis(gpu_lib, width, vertical):
    """Direct sum, allocating and static solve (opening every cell) of a sheet,
    each component against long double: within its own terms' roundings, 2^-52
    for the pair, 2^-49 for 1/sigma^2 in e^-x and 2^-51 for the partial sums."""
    torch = pytest.importorskip("torch")
    P = gpu_lib
    n = 1500
    xy, cir, cor = sheet(n, width, vertical)
    P.set_params(11, 33, -1.0)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(xy, cir, cor)
        uv = {"direct": run_direct(P, torch, xy, xy, cir, cor), "tree": P.biot_tree_batch(xy)}
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xy, cir, cor)]
        out = torch.empty_like(d[0])
        assert P.solve_device_static(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), n) == P.OK
        torch.cuda.synchronize()
        uv["static"] = out.cpu().numpy()
    finally:
        P.clear_params()
    r = xy[:, None, :] - xy  # the kernels' FP64 differences
    r2 = (L(1) * r * r).sum(axis=2)
    with np.errstate(all="ignore"):
        f = np.where(r2 > 1e-20, cir / r2, 0)
    e = -np.expm1(-r2 / (L(1) * cor * cor))
    for k, c in ((0, -r[:, :, 1]), (1, r[:, :, 0])):
        t = f * e * c
        bound = np.abs(t).sum(axis=1) * (2.0**-52 + 2.0**-49 + 2.0**-51) + np.abs(f * c).sum(axis=1) * 2.0**-53
        for name, v in uv.items():
            assert (np.abs(v[:, k] - t.sum(axis=1) / (2 * L(np.pi))) <= bound / (2 * np.pi)).all(), (name, k)

"""The plain kernel's fixed-point terms (2dfmm_gb300/csrc/fix64.cuh, the same
code compiled for the host) against exact arithmetic: the regularised pair
(fmm.c:121-142), the multipole sum (fmm.c:60-67) and the running sum."""
from __future__ import annotations

import ctypes
import math
import os
import subprocess
import zlib
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))
D = ctypes.POINTER(ctypes.c_double)
U = ctypes.POINTER(ctypes.c_uint64)


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fix64") / "fix64.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "fix64_shim.cpp")], check=True)
    return ctypes.CDLL(so)


def dp(a):
    return a.ctypes.data_as(D)


def exp_fixed(x: Fraction) -> int:
    """e^-x in units of 2^-62, to nearest, by the Taylor series."""
    t, s, k = Fraction(1), Fraction(0), 0
    while abs(t) > Fraction(1, 1 << 80):
        s += t
        k += 1
        t = t * -x / k
    return int(s * (1 << 62) + Fraction(1, 2))


@pytest.fixture(scope="module")
def tables():
    e1 = Fraction(exp_fixed(Fraction(1)), 1 << 62)  # only to check the range of the tables
    assert abs(float(e1) - math.exp(-1)) < 1e-15
    ints = np.array([exp_fixed(Fraction(n)) for n in range(40)], np.uint64)
    fracs = np.array([exp_fixed(Fraction(j, 2048)) for j in range(2048)], np.uint64)
    return ints, fracs


# r/sigma from blobs almost on top of each other to where e^-x is nothing
@pytest.mark.parametrize("lo,hi", [(1e-9, 1e-6), (1e-4, 1e-2), (0.03, 0.3), (0.3, 3.0), (3.0, 6.2), (6.2, 6.4), (6.4, 1e9)])
@pytest.mark.parametrize("scale", [1e-8, 1.0, 1e9])
def test_pair_against_long_double(shim, tables, lo, hi, scale):
    """G (1 - e^-x)/r^2 (-dy, dx): within 2^-52 of each component, besides an
    absolute 2^-55 in the bracket (the tables' and the polynomial's units)."""
    rng = np.random.default_rng(int(1000 * hi) % 99991)
    n = 20_000
    sigma = scale * np.exp(rng.uniform(-1, 1, n))
    r = sigma * np.exp(rng.uniform(math.log(lo), math.log(hi), n))
    a = rng.uniform(-math.pi, math.pi, n)
    dx, dy = r * np.cos(a), r * np.sin(a)
    dx[:40] = 0.0                     # on an axis
    dy[40:80] *= 1e-30                # one component far below the other
    dx[80:200] = np.exp2(np.round(np.log2(np.abs(dx[80:200]))))  # powers of two
    dy[80:140] = 0.0
    far = dx * dx + dy * dy > 1e-20   # the kernel's own cut
    g = rng.standard_normal(n) * np.exp(rng.uniform(-30, 30, n))
    g[200:220] = 0.0
    ic = 1.0 / (sigma * sigma)
    out = np.empty((n, 2))
    shim.pair_terms(n, dp(dx), dp(dy), dp(g), dp(ic), tables[0].ctypes.data_as(U), tables[1].ctypes.data_as(U), dp(out))
    L = np.longdouble
    r2 = L(1) * dx * dx + L(1) * dy * dy
    with np.errstate(all="ignore"):
        f = g / r2
        e = -np.expm1(-r2 * ic)
    for k, d in ((0, -dy), (1, dx)):
        exact = f * e * d
        bound = np.abs(exact) * 2.0**-52 + np.abs(f * d) * 2.0**-55
        bad = far & ~(np.abs(out[:, k] - exact) <= bound)
        # one component at most 2^-54 of the other is below the common unit
        bad &= ~(np.abs(out[:, k] - exact) <= np.abs(f * e) * np.hypot(dx, dy) * 2.0**-53)
        assert not bad.any(), (k, np.flatnonzero(bad)[:5], dx[bad][:3], dy[bad][:3])


def test_pair_point_vortex_and_infinite_core(shim, tables):
    """1/sigma^2 = inf (core radius 0) gives the point vortex, 0 (infinite core) nothing."""
    dx, dy = np.array([1e-3, 0.5, 3e-10]), np.array([2e-3, 0.0, 0.0])
    g, out = np.array([2.0, -1.0, 1.0]), np.empty((3, 2))
    for ic in (np.inf, 0.0):
        c = np.full(3, ic)
        shim.pair_terms(3, dp(dx), dp(dy), dp(g), dp(c), tables[0].ctypes.data_as(U), tables[1].ctypes.data_as(U), dp(out))
        f = g / (dx * dx + dy * dy) * (1.0 if ic else 0.0)
        assert np.allclose(out, np.stack([-f * dy, f * dx], axis=1), rtol=1e-15, atol=0)


def blobs_in(rng, kind, R):
    if kind == "corner":
        p, g = np.array([[0.5, 0.5]]), np.array([1.0])
    elif kind == "centre":
        p, g = np.array([[0.0, 0.0]]), np.array([-3.0])
    elif kind == "dipole":
        p, g = np.array([[0.1, 0.2], [-0.1, -0.2]]), np.array([1.0, -1.0])
    elif kind == "zero":
        p, g = np.array([[0.3, 0.1]]), np.array([0.0])
    else:
        m = int(kind)
        p, g = rng.uniform(-0.5, 0.5, (m, 2)), rng.standard_normal(m)
    return p * R, g


@pytest.mark.parametrize("kind", ["corner", "centre", "dipole", "zero", "2", "40"])
@pytest.mark.parametrize("theta", [0.05, 0.35, np.nextafter(0.35, 1), 0.4, 0.5, 0.6, 0.61, 0.7])
def test_cell_against_long_double(shim, kind, theta):
    """sum_k a_k w^(k+1) at accepted offsets (R <= theta |d|), from the
    boundary outwards: within 2^-50 of the sum of the terms' magnitudes (an
    FP64 Horner scheme's own bound is about 2K 2^-53 of it), for every K at
    and around the FP32 pairs' first term."""
    rng = np.random.default_rng(zlib.crc32(f"{kind} {float(theta)}".encode()))
    L = np.longdouble
    for R in (1.0, 3.7e-9, 8.1e7):
        p, g = blobs_in(rng, kind, R)
        z = p[:, 0] + 1j * p[:, 1]
        for K in (1, 2, 4, 5, 6, 7, 8, 11, 12, 13, 20, 31):
            a = np.array([(g * z**k).sum() for k in range(K)])
            n = 400
            d = R / theta * np.exp(np.concatenate([rng.uniform(0, 1e-6, n // 4), rng.uniform(0, 1.5, n // 2),
                                                   rng.uniform(0, 25, n - n // 4 - n // 2)]))
            d *= 1 + 1e-14
            t = rng.uniform(-math.pi, math.pi, n)
            t[:8] = np.arange(8) * math.pi / 4
            dx, dy = d * np.cos(t), d * np.sin(t)
            ab, out = np.ascontiguousarray(np.stack([a.real, a.imag], axis=1)), np.empty((n, 2))
            shim.cell_terms(K, dp(ab), ctypes.c_double(R), ctypes.c_double(theta), n, dp(dx), dp(dy), dp(out))
            w = (L(1) * dx - 1j * (L(1) * dy)) / (L(1) * dx * dx + L(1) * dy * dy)
            s, mag, pw = np.zeros(n, np.clongdouble), np.zeros(n), w
            for k in range(K):
                s = s + (L(1) * a[k].real + 1j * (L(1) * a[k].imag)) * pw
                mag += np.abs(a[k]) * np.abs(pw).astype(float)
                pw = pw * w
            err = np.abs((out[:, 0] + 1j * out[:, 1]) - s).astype(float)
            left = np.isnan(err)  # far targets are left to FP64, none within 2R/theta + 2R
            assert theta < 0.2 or not left[d <= 2 * R / theta + 2 * R].any()
            err[left] = 0.0
            assert (err <= 2.0**-50 * mag + 1e-300).all(), (R, K, float((err / np.maximum(mag, 1e-300)).max()))


def cancelling(kind, R):
    """Blobs whose first moments are exactly zero (dyadic offsets), or zero but
    for what one more blob adds."""
    if kind.startswith("line"):  # moments 0 to 2 vanish: third difference
        p = np.array([[-0.375, 0.0], [-0.125, 0.0], [0.125, 0.0], [0.375, 0.0]])
        g = np.array([-1.0, 3.0, -3.0, 1.0])
    else:  # the 4 x 4 tensor product of + - - +
        c = np.array([-0.375, -0.125, 0.125, 0.375])
        s = np.array([1.0, -1.0, -1.0, 1.0])
        p = np.stack(np.meshgrid(c, c), axis=-1).reshape(-1, 2)
        g = np.outer(s, s).ravel()
    if "+" in kind:
        p, g = np.concatenate([p, [[0.25, -0.1875]]]), np.append(g, float(kind.split("+")[1]))
    return p * R, g


@pytest.mark.parametrize("kind", ["line", "square", "line+1e-12", "square+1e-30", "line+1e-200", "square+1e-280"])
@pytest.mark.parametrize("theta", [0.3, 0.5, 0.7])
def test_cell_whose_first_moments_cancel(shim, kind, theta):
    """As test_cell_against_long_double, for cells whose first coefficients
    vanish or are far below the later ones, over circulation scales and sides:
    left to FP64, or within the a-priori bound of the FP64 Horner scheme, K
    complex multiply-adds of 3 2^-53 each (sqrt(5) for the product, 1 for the
    sum)."""
    rng = np.random.default_rng(zlib.crc32(f"{kind} {theta}".encode()))
    L = np.longdouble
    for R in (1.0, 0.25, 2.0**-20, 3.0):
        for scale in (1.0, 10.0, 1e-6, 1e20):
            p, g = cancelling(kind, R)
            g = g * scale
            z = p[:, 0] + 1j * p[:, 1]
            for K in (4, 5, 8, 10, 12, 20, 31):
                a = np.zeros(K, complex)
                pw = np.ones(len(z), complex)
                for k in range(K):
                    a[k] = complex(math.fsum((g * pw).real), math.fsum((g * pw).imag))
                    pw = pw * z
                n = 200
                d = R / theta * np.exp(np.concatenate([rng.uniform(0, 1e-6, 50), rng.uniform(0, 1.1, n - 50)])) * (1 + 1e-14)
                t = rng.uniform(-math.pi, math.pi, n)
                dx, dy = d * np.cos(t), d * np.sin(t)
                ab, out = np.ascontiguousarray(np.stack([a.real, a.imag], axis=1)), np.empty((n, 2))
                shim.cell_terms(K, dp(ab), ctypes.c_double(R), ctypes.c_double(theta), n, dp(dx), dp(dy), dp(out))
                w = (L(1) * dx - 1j * (L(1) * dy)) / (L(1) * dx * dx + L(1) * dy * dy)
                s, mag, pw = np.zeros(n, np.clongdouble), np.zeros(n), w
                for k in range(K):
                    s = s + (L(1) * a[k].real + 1j * (L(1) * a[k].imag)) * pw
                    mag += np.abs(a[k]) * np.abs(pw).astype(float)
                    pw = pw * w
                err = np.abs((out[:, 0] + 1j * out[:, 1]) - s).astype(float)
                err[np.isnan(err)] = 0.0  # left to FP64
                assert (err <= 3 * K * 2.0**-53 * mag + 1e-300).all(), (R, scale, K, float((err / np.maximum(mag, 1e-300)).max()))


@pytest.mark.parametrize("scale", [1e-290, 1e-300, 1e-306, 1e-315, 1e290, 1e300, 1e306])
@pytest.mark.parametrize("R", [1e-3, 1.0, 1e3, 1e30])
@pytest.mark.parametrize("theta", [0.35, 0.5, 0.7])
def test_cell_near_the_ends_of_the_range(shim, scale, R, theta):
    """Circulations and sides whose higher moments leave FP64's normal range:
    such a cell is left to FP64, never summed without those moments."""
    rng = np.random.default_rng(11)
    p, g = rng.uniform(-0.5, 0.5, (5, 2)), rng.uniform(0.5, 1.0, 5)
    z = (p[:, 0] + 1j * p[:, 1]) * R
    K, n = 12, 50
    with np.errstate(all="ignore"):
        a = np.array([((g * scale) * z**k).sum() for k in range(K)])
    d = R / theta * np.exp(rng.uniform(0, 1, n)) * (1 + 1e-14)
    t = rng.uniform(-math.pi, math.pi, n)
    dx, dy = d * np.cos(t), d * np.sin(t)
    ab, out = np.ascontiguousarray(np.stack([a.real, a.imag], axis=1)), np.empty((n, 2))
    shim.cell_terms(K, dp(ab), ctypes.c_double(R), ctypes.c_double(theta), n, dp(dx), dp(dy), dp(out))
    size = np.abs(ab[ab != 0])
    if not np.isfinite(ab).all() or (size < np.finfo(float).tiny).any():
        assert np.isnan(out).all()
        return
    # the exact sum at unit scale: sum_j g_j / (z - z_j) up to order K
    L = np.clongdouble
    w = 1 / (L(dx) + 1j * L(dy))
    s, pw = np.zeros(n, L), w
    for k in range(K):
        s, pw = s + (L(g) * L(z / R) ** k).sum() * pw * np.longdouble(R) ** k, pw * w
    s = s * np.longdouble(scale)
    # coefficients rounded in FP64 (k + 1 products) and the sum's own 2^-50; results
    # beyond the largest number are infinite, those below the smallest normal
    # one to its unit
    for got, exact in ((out[:, 0], s.real), (out[:, 1], s.imag)):
        large = np.abs(exact) >= np.finfo(float).max
        assert np.isinf(got[large]).all()
        err = np.abs(got[~large] - exact[~large])
        assert (err <= 2.0**-47 * np.abs(s[~large]) + np.longdouble(2.0**-1074)).all()


@pytest.mark.parametrize("span", [0, 6, 40, 200])
def test_running_sum_is_exact_to_its_unit(shim, span):
    """Terms of exponents spread over `span` bits, in growing, falling and
    random order: within 2^-31 units of the largest term per term."""
    rng = np.random.default_rng(span)
    for order in ("up", "down", "random"):
        n = 3000
        e = rng.integers(-span // 2 - 1, span // 2 + 1, n).astype(np.int32)
        e = np.sort(e) if order == "up" else np.sort(e)[::-1].copy() if order == "down" else e
        m = rng.integers(-(2**62) + 1, 2**62, (2, n), dtype=np.int64)
        m[:, ::97] = 2**62 - 1  # the same sign in a row, too
        m[:, -500:] = np.abs(m[:, -500:])
        out = np.empty(2)
        q = [np.ascontiguousarray(v) for v in m]
        ll, ip = ctypes.POINTER(ctypes.c_longlong), ctypes.POINTER(ctypes.c_int)
        shim.sum_terms(n, q[0].ctypes.data_as(ll), q[1].ctypes.data_as(ll), e.ctypes.data_as(ip), dp(out))
        for k in range(2):
            exact = sum(Fraction(int(v)) * Fraction(2) ** int(x) for v, x in zip(m[k], e))
            # unit of the sum's low word: 2^-32 of 2^(at most the sum's growth) units 2^8 above the largest term's
            unit = Fraction(2) ** (int(e.max()) + 13 + 4 - 31)
            assert abs(Fraction(float(out[k])) - exact) <= n * unit + abs(exact) * Fraction(2) ** -53


@pytest.mark.gpu
@pytest.mark.parametrize("theta,nterms", [(0.3, 6), (0.3, 7), (0.5, 2), (0.5, 8), (0.5, 9), (0.5, 32), (0.6, 12), (0.7, 21),
                                          (np.nextafter(0.7, 1), 21), (1.2, 13)])
@pytest.mark.parametrize("n,num_p", [(61, 2), (3001, 5), (2500, 131)])
def test_velocity_around_the_forms_limits(gpu_lib, theta, nterms, n, num_p):
    """GPU velocities against the oracle on both sides of every rule that picks
    an arithmetic (opening angle, first FP32 pair term), with leaves of one
    blob and leaves longer than one 128-blob stretch, at blobs, between them
    and far outside."""
    from conftest import oracle, workloads
    from test_plain_parity import assert_parity, ext_for
    P = gpu_lib
    b = workloads().uniform(n, seed=n + nterms)
    rng = np.random.default_rng(5)
    pts = np.concatenate([rng.uniform(-0.3, 1.3, (40, 2)), [[3.0, -2.0], [40.0, 9.0], [-1e4, 2e4]]])
    P.set_params(nterms, num_p, theta)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(b.xy, b.cir, b.cor)
        uv = P.biot_tree_batch(np.concatenate([b.xy, pts]))
    finally:
        P.clear_params()
    o = oracle().SparseOracle(nterms, num_p, float(theta))
    o.make_tree(b.xy, b.cir, b.cor)
    t = np.concatenate([b.xy, pts])
    ref = o.biot(t)
    o.close()
    assert_parity(uv, ref, t, ext_for(b.xy, b.cir, b.cor, nterms, num_p, float(theta)), label=f"{theta} {nterms} {n}")


@pytest.mark.gpu
@pytest.mark.parametrize("theta", [0.3, 0.5, 0.7])
def test_velocity_of_cancelling_clusters(gpu_lib, theta):
    """A field of clusters whose first three moments vanish, so that every
    cell's leading coefficients are rounding residues: blobs and far points
    against the oracle, and the static solve (whose converted coefficients
    take the place of the FP64 ones) bit for bit with the allocating one."""
    torch = pytest.importorskip("torch")
    from conftest import oracle
    P = gpu_lib
    rng = np.random.default_rng(9)
    q, g = cancelling("line", 2.0**-8)
    at = rng.permutation(64 * 64)[:500]
    xy = (np.stack([at % 64, at // 64], axis=1)[:, None, :] / 64.0 + q).reshape(-1, 2)
    cir = np.tile(g, 500)
    cor = np.full(len(xy), 2e-3)
    P.set_params(12, 33, theta)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(xy, cir, cor)
        pts = np.concatenate([xy, rng.uniform(-0.2, 1.2, (200, 2))])
        uv = P.biot_tree_batch(pts)
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xy, cir, cor)]
        out = torch.empty_like(d[0])
        assert P.solve_device_static(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), len(xy)) == P.OK
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint64), uv[: len(xy)].copy().view(np.uint64))
    finally:
        P.clear_params()
    o = oracle().SparseOracle(12, 33, float(theta))
    o.make_tree(xy, cir, cor)
    ref = o.biot(pts)
    o.close()
    # What cancels leaves the roundings of the moments, 8 (k + 1) levels 2^-53
    # of sum |G| (1.5 R)^k each (test_coefficients_are_the_cells_moments): at
    # R <= 0.7 |d| and 6 levels some 2^-41 of the point vortices' speeds
    r = np.hypot(pts[:, None, 0] - xy[:, 0], pts[:, None, 1] - xy[:, 1])
    with np.errstate(divide="ignore"):
        speed = np.where(r > 0, np.abs(cir) / r, 0.0).sum(axis=1) / (2 * math.pi)
    assert (np.abs(uv - ref) <= 2.0**-41 * speed[:, None]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("size,strength", [(0.05, 3001e-290), (1.0, 1e290), (1e30, 1e-100)])
def test_velocity_near_the_ends_of_the_range(gpu_lib, size, strength):
    """Sets whose smaller cells' higher moments are subnormal (to 2^-35 of
    themselves at least), or whose larger ones' are near the top of the range,
    against the oracle; the static solve bit for bit with the allocating one."""
    torch = pytest.importorskip("torch")
    from conftest import oracle, workloads
    P = gpu_lib
    b = workloads().uniform(3001, seed=13)
    xy, cir, cor = b.xy * size, b.cir * strength, b.cor * size
    P.set_params(11, 33, 0.5)
    P.set_mode(P.MODE_PLAIN)
    try:
        P.make_tree(xy, cir, cor)
        uv = P.biot_tree_batch(xy)
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (xy, cir, cor)]
        out = torch.empty_like(d[0])
        assert P.solve_device_static(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), len(xy)) == P.OK
        torch.cuda.synchronize()
    finally:
        P.clear_params()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), uv.view(np.uint64))
    o = oracle().SparseOracle(11, 33, 0.5)
    o.make_tree(xy, cir, cor)
    ref = o.biot(xy)
    o.close()
    assert np.isfinite(uv).all()
    assert np.abs(uv - ref).max() <= 1e-12 * np.abs(ref).max()

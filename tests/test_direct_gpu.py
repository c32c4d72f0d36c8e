"""FP64 direct-sum kernel (the accuracy yardstick) against the oracle's direct sum."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import oracle


@pytest.mark.gpu
def test_direct_kernel_matches_oracle(gpu_lib):
    torch = pytest.importorskip("torch")
    P = gpu_lib
    rng = np.random.default_rng(3)
    sxy = rng.random((5000, 2))
    cir = rng.standard_normal(5000) / 5000
    cor = np.full(5000, 0.01)
    txy = np.concatenate([sxy[:100], rng.random((300, 2))])
    ref = oracle().direct(txy, sxy, cir, cor)
    dev = torch.device("cuda:0")
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    out = torch.empty((len(txy), 2), dtype=torch.float64, device=dev)
    tt, ss, cc, rr = t(txy), t(sxy), t(cir), t(cor)
    P.direct_device(tt.data_ptr(), len(txy), ss.data_ptr(), cc.data_ptr(), rr.data_ptr(), len(cir), out.data_ptr())
    torch.cuda.synchronize()
    uv = out.cpu().numpy()
    assert np.abs(uv - ref).max() <= 1e-12 * np.abs(ref).max()


def run_direct(P, torch, txy, sxy, cir, cor):
    dev = torch.device("cuda:0")
    t = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (txy, sxy, cir, cor)]
    out = torch.empty((len(txy), 2), dtype=torch.float64, device=dev)
    P.direct_device(t[0].data_ptr(), len(txy), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), len(cir), out.data_ptr())
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("ntgt,nsrc", [(1, 1), (31, 2), (255, 257), (256, 256), (257, 1023), (700, 4097)])
def test_direct_kernel_within_its_roundings(gpu_lib, ntgt, nsrc):
    """Against long double: each pair within 2^-52 of itself and 2^-55 of its
    point-vortex value (fix64.cuh), the block sums added in FP64 (at most 8
    chunks here).  Core radii from 0 (point vortex) over ordinary ones to
    infinity (no velocity), zero circulations and coincident points."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(ntgt)
    sxy = rng.random((nsrc, 2))
    cir = rng.standard_normal(nsrc)
    cor = np.exp(rng.uniform(-9, 0, nsrc))
    cor[::5], cor[1::7], cir[2::9] = 0.0, np.inf, 0.0
    txy = np.concatenate([sxy[: ntgt // 2], rng.random((ntgt - ntgt // 2, 2))])
    uv = run_direct(gpu_lib, torch, txy, sxy, cir, cor)
    L = np.longdouble
    rx, ry = L(1) * txy[:, None, 0] - sxy[:, 0], L(1) * txy[:, None, 1] - sxy[:, 1]
    r2 = rx * rx + ry * ry
    with np.errstate(all="ignore"):
        f = np.where(r2 > 1e-20, cir / r2, 0)
        e = np.where(cor > 0, -np.expm1(-r2 / (L(1) * cor * cor)), 1)
    for k, d in ((0, -ry), (1, rx)):
        exact = (f * e * d).sum(axis=1) / (2 * L(np.pi))
        # 1/sigma^2 is formed in FP64: 2 roundings, at most 0.37 2^-52 in e^-x
        bound = (np.abs(f * e * d) * 2.0**-52 + np.abs(f * d) * 2.0**-53).sum(axis=1) + np.abs(f * e * d).sum(axis=1) * 2.0**-49
        assert (np.abs(uv[:, k] - exact) <= bound / (2 * np.pi) + 1e-300).all()


@pytest.mark.gpu
def test_direct_kernel_passes_on_what_is_not_finite(gpu_lib):
    """A NaN position takes part in nothing (r > 1e-10 is false); a NaN core
    radius or a non-finite circulation reaches every target it acts on; an
    infinite target position gives NaN: as the FP64 formula has it."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1)
    sxy, cir, cor = rng.random((300, 2)), rng.standard_normal(300), np.full(300, 0.05)
    txy = rng.random((64, 2))
    ok = run_direct(gpu_lib, torch, txy, sxy, cir, cor)
    s2, c2, r2, t2 = sxy.copy(), cir.copy(), cor.copy(), txy.copy()
    s2[7, 0] = np.nan
    c3 = cir.copy()
    c3[7] = 0.0
    assert np.array_equal(run_direct(gpu_lib, torch, txy, s2, cir, cor), run_direct(gpu_lib, torch, txy, sxy, c3, cor))
    for bad in (np.nan, np.inf):
        c2[9] = bad
        assert not np.isfinite(run_direct(gpu_lib, torch, txy, sxy, c2, cor)).any()
    r2[9] = np.nan
    assert np.isnan(run_direct(gpu_lib, torch, txy, sxy, cir, r2)).all()
    t2[3, 0], t2[5, 1], t2[6, 0] = np.nan, np.inf, -np.inf
    uv = run_direct(gpu_lib, torch, t2, sxy, cir, cor)
    assert np.array_equal(uv[3], [0.0, 0.0]) and np.isnan(uv[[5, 6]]).all()
    keep = np.setdiff1d(np.arange(64), [3, 5, 6])
    assert np.array_equal(uv[keep], ok[keep])

"""Legendre stages at the edges of their tiles, against the FP64 oracle.

Field counts cross every tile width of the FP64 path (1 and 2 on the FP64 pipes; 4, 8 and 16
fields a synthesis warp; 8 and 16 fields an analysis warp, 16, 32 and 64 a CTA) and of the mixed
path's one- and two-field kernels; degrees and latitude pairs cross the steps of 8 (chains,
quarters), 32 (segments, lanes) and 64 (tiles, chunks). Bounds: the paths' own 1e-12 and 1e-6.
"""
import numpy as np
import pytest
import torch

import shtb200 as sht
from oracle import sht_oracle as so

from _util import rand_alm, rel_l2

pytestmark = pytest.mark.gpu

GRIDS = [
    dict(lmax=0, nlat=1, nlon=2),
    dict(lmax=6, nlat=7, nlon=14),                      # below one chain
    dict(lmax=31, nlat=63, nlon=64),                    # 32 degrees, 32 pairs with an equator row
    dict(lmax=32, nlat=66, nlon=70),                    # one more of each
    dict(lmax=65, nlat=130, nlon=132, mmax=9),          # tiles of 64 degrees plus two, 65 pairs
    dict(lmax=47, nlat=50, nlon=96, mres=3, mmax=45),
]
IDS = ["l0", "l6", "l31", "l32", "l65", "l47-mres3"]


def check(cfg, ocfg, nf, lcap, precision, tol):
    a = rand_alm(cfg.lmax, cfg.mmax, nf, seed=nf, mres=cfg.mres)
    g = np.random.default_rng(nf).standard_normal((cfg.nlat, cfg.nlon, nf))
    if precision == "mixed":
        a, g = a.astype(np.complex64), g.astype(np.float32)
    f = sht.to_host(sht.synthesis_batch(cfg, a, lcap=lcap, precision=precision))
    b = sht.to_host(sht.analysis_batch(cfg, g, lcap=lcap, precision=precision))
    for k in sorted({0, nf // 2, nf - 1}):
        af = a[:, :, k].astype(complex)
        assert rel_l2(f[:, :, k], so.synthesis(ocfg, af, ltr=lcap)) <= tol, (nf, k)
        assert rel_l2(b[:, :, k], so.analysis(ocfg, g[:, :, k].astype(float), ltr=lcap)) <= tol, (nf, k)


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_fp64_tiles(grid):
    c = dict(grid)
    lmax, nlat = c.pop("lmax"), c.pop("nlat")
    cfg, ocfg = sht.create_gauss_config(lmax, nlat, **c), so.create_gauss_config(lmax, nlat, **c)
    for nf in (1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 65):
        check(cfg, ocfg, nf, None, "fp64", 1e-12)
    for nf in (1, 2, 3, 17):
        check(cfg, ocfg, nf, max(0, lmax - 5), "fp64", 1e-12)


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_mixed_one_and_two_fields(grid):
    c = dict(grid)
    lmax, nlat = c.pop("lmax"), c.pop("nlat")
    cfg, ocfg = sht.create_gauss_config(lmax, nlat, **c), so.create_gauss_config(lmax, nlat, **c)
    for nf in (1, 2, 3):
        check(cfg, ocfg, nf, None, "mixed", 1e-6)
        check(cfg, ocfg, nf, max(0, lmax - 5), "mixed", 1e-6)


def test_late_starts_and_two_row_tiles():
    """Orders high enough that the pairs near the poles start late (extended-range seeds), with
    enough CTAs for two row tiles per warp: batches of 3 and 5 fields against single fields."""
    cfg = sht.create_gauss_config(700, 702, mmax=640, nlon=1500)
    a = rand_alm(700, 640, 5, seed=3)
    g = np.random.default_rng(4).standard_normal((702, 1500, 5))
    one = [sht.to_host(sht.synthesis(cfg, a[:, :, k])) for k in range(5)]
    ana = [sht.to_host(sht.analysis(cfg, g[:, :, k])) for k in range(5)]
    for nf in (2, 3, 5):
        f, b = sht.to_host(sht.synthesis_batch(cfg, a[:, :, :nf])), sht.to_host(sht.analysis_batch(cfg, g[:, :, :nf]))
        for k in range(nf):
            assert rel_l2(f[:, :, k], one[k]) <= 1e-12 and rel_l2(b[:, :, k], ana[k]) <= 1e-12
    assert rel_l2(sht.to_host(sht.analysis(cfg, one[0])), a[:, :, 0]) <= 1e-12


@pytest.mark.parametrize("lmax", [1799, 2047, 2999, 3599], ids=["step16", "step32", "step64", "step128"])
def test_sparse_checkpoints(lmax):
    """Sizes at which the checkpoint table exceeds its budget (2 GiB) at 8 degrees, so that chains
    are rolled forward from checkpoints 16, 32, 64 and 128 degrees apart: analyses of three or more
    fields (every tile width), of two fields (segments of 16 degrees) from 32 on and of one field
    (32 degrees) from 64 on. Roundtrip error grows with the number of degrees (7e-14 at 1023)."""
    step = 8
    while step < 128 and sum((lmax + 1 - m + step) // step for m in range(lmax + 1)) * ((lmax + 2) // 2) * 16 > 2 ** 31:
        step *= 2
    assert step == {1799: 16, 2047: 32, 2999: 64, 3599: 128}[lmax]
    cfg = sht.create_gauss_config(lmax, lmax + 1, nlon=2 * lmax + 2)
    g = torch.Generator(device="cuda").manual_seed(5)
    l = torch.arange(lmax + 1, device="cuda")
    keep = (l[:, None] >= l[None, :]) / (l[:, None] + 1.0)
    for nf in (1, 2, 3, 9, 17, 33):
        a = sht.julia_empty((lmax + 1, lmax + 1, nf), torch.complex128, "cuda")
        for k in range(nf):
            z = torch.randn((lmax + 1, lmax + 1, 2), dtype=torch.float64, device="cuda", generator=g)
            z[:, 0, 1] = 0
            a[:, :, k] = torch.view_as_complex(z) * keep
        back = sht.analysis_batch(cfg, sht.synthesis_batch(cfg, a))
        for k in range(nf):
            assert float((back[:, :, k] - a[:, :, k]).norm() / a[:, :, k].norm()) <= 1e-12, (nf, k)
        del a, back, z
    cfg.clear_plans()

"""Longitude FFTs whose length has prime factors above 13 (passes of their own radix between
two row buffers): every edge of that path against the FP64 oracle.

Bounds: the FP64 path's 1e-12 relative L2 (a prime pass sums (r + 1) / 2 products per output,
about sqrt(r) 1.1e-16 relative), the mixed path's 1e-6, complex grids 1e-12.
"""
import numpy as np
import pytest
import torch

import shtb200 as sht
from oracle import sht_oracle as so

from _util import rand_alm, rel_l2

pytestmark = pytest.mark.gpu

# one prime factor (smallest, odd, large), alone, squared, two different ones, after each radix kind
NLONS = [17, 34, 289, 646, 127, 16 * 19, 8 * 3 * 5 * 23, 2 * 509, 1021]


@pytest.mark.parametrize("nlon", NLONS)
@pytest.mark.parametrize("nlat,nf", [(9, 1), (34, 3)])
def test_prime_radix_passes(nlon, nlat, nf):
    lmax = min(nlat - 1, (nlon - 1) // 2, 20)
    cfg, ocfg = sht.create_gauss_config(lmax, nlat, nlon=nlon), so.create_gauss_config(lmax, nlat, nlon=nlon)
    a = rand_alm(lmax, lmax, nf, seed=nlon)
    ref = so.synthesis_batch(ocfg, a)
    g = np.random.default_rng(nlon).standard_normal((nlat, nlon, nf))
    aref = so.analysis_batch(ocfg, g)
    assert rel_l2(sht.to_host(sht.synthesis_batch(cfg, a)), ref) <= 1e-12
    assert rel_l2(sht.to_host(sht.analysis_batch(cfg, g)), aref) <= 1e-12
    f32 = sht.synthesis_batch(cfg, a.astype(np.complex64), precision="mixed")
    assert rel_l2(sht.to_host(f32), so.synthesis_batch(ocfg, a.astype(np.complex64).astype(complex))) <= 1e-6
    b32 = sht.analysis_batch(cfg, g.astype(np.float32), precision="mixed")
    assert rel_l2(sht.to_host(b32), so.analysis_batch(ocfg, g.astype(np.float32).astype(float))) <= 1e-6
    z = g[:, :, 0] + 1j * g[::-1, :, 0]
    zref = so.analysis(ocfg, z)
    assert rel_l2(sht.to_host(sht.analysis(cfg, z)), zref) <= 1e-12
    fz = sht.synthesis(cfg, a[:, :, 0], real_output=False)
    torch.cuda.synchronize()
    assert rel_l2(sht.to_host(fz), so.synthesis(ocfg, a[:, :, 0], real_output=False)) <= 1e-12

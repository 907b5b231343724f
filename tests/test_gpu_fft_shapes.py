"""Launch shapes of the general longitude FFT: both sides of each line that the choice of latitude
pairs and threads per CTA draws, against the FP64 oracle.

Row lengths below, at and above 2048 points in FP32 (where the runs may shrink to 16 bytes) and at
the lengths where the most pairs that fit change from 16 to 8, 4 and 2; one field (split until the
last CTA fits) and a batch that is not split. An odd nlat keeps power-of-two rows in this kernel.
"""
import numpy as np
import pytest

import shtb200 as sht
from oracle import sht_oracle as so

from _util import rand_alm, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nlon", [("mixed", n) for n in (690, 720, 1350, 1440, 1500, 2046, 2048, 2880, 3000)]
                         + [("fp64", n) for n in (640, 720, 1350, 1440, 2700, 3000)])
@pytest.mark.parametrize("nlat,nf", [(33, 1), (33, 3), (301, 13), (301, 24)])
def test_launch_shapes(precision, nlon, nlat, nf):
    lmax, tol = 20, 1e-12 if precision == "fp64" else 1e-6
    cfg, ocfg = sht.create_gauss_config(lmax, nlat, nlon=nlon), so.create_gauss_config(lmax, nlat, nlon=nlon)
    a = rand_alm(lmax, lmax, nf, seed=nlon)
    g = np.random.default_rng(nlon).standard_normal((nlat, nlon, nf))
    if precision == "mixed":
        a, g = a.astype(np.complex64), g.astype(np.float32)
    f = sht.to_host(sht.synthesis_batch(cfg, a, precision=precision))
    b = sht.to_host(sht.analysis_batch(cfg, g, precision=precision))
    for k in sorted({0, nf // 2, nf - 1}):
        assert rel_l2(f[:, :, k], so.synthesis(ocfg, a[:, :, k].astype(complex))) <= tol
        assert rel_l2(b[:, :, k], so.analysis(ocfg, g[:, :, k].astype(float))) <= tol

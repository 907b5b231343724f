"""Lazily conjugated and negated tensors: views whose memory holds other values than they show.
Every entry point must read, or write, the values that torch shows."""
import pytest
import torch

import shtb200 as sht
from shtb200 import transforms as T

from _util import rand_alm


def test_to_device_materializes_lazy_views(monkeypatch):
    monkeypatch.setattr(T, "_cuda_device", lambda index: torch.device("cpu"))
    a = T.julia_empty((3, 4), torch.complex128, "cpu")
    a.copy_(torch.randn(3, 4, dtype=torch.complex128))
    plain = T.to_device(a, torch.complex128, 0)
    assert plain.data_ptr() == a.data_ptr()                     # ordinary tensors are not copied
    for lazy in (a.conj(), torch._neg_view(a), torch._neg_view(a.real.clone(memory_format=torch.preserve_format))):
        d = T.to_device(lazy, lazy.dtype, 0)
        assert not d.is_conj() and not d.is_neg() and T.is_julia_dense(d)
        assert torch.equal(d, lazy.resolve_conj().resolve_neg())


def _pair(lmax, nlat, nf=2):
    cfg = sht.create_gauss_config(lmax, nlat)
    a = sht.to_device(rand_alm(lmax, lmax, nf, seed=1), torch.complex128, 0)
    b = sht.to_device(rand_alm(lmax, lmax, nf, seed=2, lmin=1), torch.complex128, 0)
    return cfg, a, b


@pytest.mark.gpu
def test_inputs():
    cfg, a, b = _pair(15, 18)
    ac, bc = a.conj(), b.conj()
    am, bm = ac.resolve_conj(), bc.resolve_conj()
    assert ac.is_conj() and not am.is_conj()
    vt, vp = sht.synthesis_sphtor_batch(cfg, a, b)
    neg, pos = torch._neg_view(vt), (-vt)
    cases = [
        (sht.synthesis_batch, (ac,), (am,)), (sht.synthesis_sphtor_batch, (ac, bc), (am, bm)),
        (sht.synthesis_divvort_batch, (ac, bc), (am, bm)), (sht.divergence_from_spheroidal, (ac,), (am,)),
        (sht.analysis_batch, (neg,), (pos,)), (sht.analysis_sphtor_batch, (neg, vp), (pos, vp)),
        (sht.analysis_divvort_batch, (neg, vp), (pos, vp)),
        (lambda c, q: sht.synthesis_packed(c, q), (sht.pack_lm(cfg, a[:, :, 0]).conj(),), (sht.pack_lm(cfg, am[:, :, 0]),)),
        (lambda c, z: sht.synthesis(c, z, real_output=False), (ac[:, :, 0],), (am[:, :, 0],)),
    ]
    for fn, lazy, plain in cases:
        x, y = fn(cfg, *lazy), fn(cfg, *plain)
        for u, v in zip(x if isinstance(x, tuple) else (x,), y if isinstance(y, tuple) else (y,)):
            assert torch.equal(u, v)


@pytest.mark.gpu
def test_outputs():
    cfg, a, b = _pair(15, 18)
    f = sht.synthesis_batch(cfg, a)
    out = torch._neg_view(sht.julia_empty(tuple(f.shape), f.dtype, f.device))
    assert sht.synthesis_into(cfg, out, a) is out and torch.equal(out, f)
    d = sht.divergence_from_spheroidal(cfg, a)
    oc = sht.julia_empty(tuple(a.shape), a.dtype, a.device).conj()
    assert sht.divergence_from_spheroidal_into(cfg, oc, a) is oc and torch.equal(oc, d)
    # in place on a conjugate view: the scaling is real
    c = a.clone().conj()
    assert sht.gpu_apply_laplacian(cfg, c) is c and c.is_conj() and torch.equal(c, d.conj())
    ao = sht.julia_empty(tuple(a.shape), a.dtype, a.device).conj()
    sht.analysis_into(cfg, ao, f)
    assert torch.equal(ao, sht.analysis_batch(cfg, f))


@pytest.mark.gpu
def test_conjugated_gradient():
    """backward() hands the analysis' gradient over with the conjugate bit set."""
    cfg, a, b = _pair(15, 18)
    g = sht.synthesis_batch(cfg, a)
    grads = []
    for lazy in (b.conj(), b.conj().resolve_conj()):
        x = g.clone().requires_grad_(True)
        sht.analysis_batch(cfg, x).backward(lazy)
        grads.append(x.grad)
    assert torch.equal(grads[0], grads[1])

"""The work that users of this library have it do, as measurable cases.

Every case goes through the public Python entry points (``shtb200``), on the
Gauss-Legendre grids and coefficient layouts that a program passes. Kinds:

  scalar    synthesis_batch then analysis_batch of the result, FP64 or mixed precision
  vector    the same for scalar fields plus one spheroidal/toroidal vector field (FP64)
  divvort   divergence/vorticity spectra to winds and back, one field per level (FP64)
  grad      gradient of a least-squares misfit through synthesis and its vector form (FP64)
  packed    transforms on packed LM coefficients with degree truncation
  uneven    many one-field mixed-precision roundtrips of different sizes in one graph launch

``exact`` restates each kind in plain torch float64 (nodes in 80-bit floats).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "shtnskit.jl_b200"))

import shtb200 as sht  # noqa: E402
from shtb200.group import UnevenBatch  # noqa: E402


def _smooth(n):
    """Smallest 2^a 3^b 5^c >= n."""
    while True:
        k = n
        for p in (2, 3, 5):
            while k % p == 0:
                k //= p
        if k == 1:
            return n
        n += 1


def _max_prime(n):
    p, big = 2, 1
    while n > 1:
        while n % p == 0:
            n //= p
            big = p
        p += 1
    return big


def _case(kind, lmax, nlat, nlon, nf, **kw):
    c = dict(kind=kind, lmax=lmax, nlat=nlat, nlon=nlon, nf=nf, mmax=lmax, norm="orthonormal", precision="fp64",
             ltr=lmax, members=0, sizes=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest ordinary call: one field of a test or teaching grid, where launches and
        # host work are the time
        _case("scalar", 63, 64, 128, 1, name="f64_l63_nf1"),
        # a single global field at the highest resolution (one variable of an analysis, a
        # gravity or magnetic model)
        _case("scalar", 1023, 1024, 2048, 1, name="f64_l1023_nf1"),
        # a grid nobody tuned: odd nlat, the default nlon of create_gauss_config (402 = 2 3 67),
        # Schmidt normalization, a handful of fields
        _case("scalar", 200, 203, 402, 3, norm="schmidt", name="f64_l200_ragged_nf3"),
        # a model state: 16 scalar fields and one wind field at lmax 511
        _case("vector", 511, 512, 1024, 16, name="f64_l511_nf16_wind"),
        # the largest FP64 batch
        _case("scalar", 1023, 1024, 2048, 64, name="f64_l1023_nf64"),
        # the headline: the same batch in mixed precision
        _case("scalar", 1023, 1024, 2048, 64, precision="mixed", name="mixed_l1023_nf64"),
        # one field in mixed precision (inference on one variable)
        _case("scalar", 511, 512, 1024, 1, precision="mixed", name="mixed_l511_nf1"),
        # a dealiased grid (3/2 rule) with an odd field count, mixed precision
        _case("scalar", 341, 512, 1080, 13, precision="mixed", name="mixed_l341_dealiased_nf13"),
        # differentiation: gradient of a misfit on 32 fields and one vector field
        _case("grad", 255, 256, 512, 32, name="grad_l255_nf32"),
        # one step of a spectral dynamical core: div/vort to winds and back on a dealiased grid
        _case("divvort", 170, 256, 512, 8, name="divvort_l170_nf8"),
        # packed LM coefficients (SHTns files) with truncation, a few fields, mixed precision
        _case("packed", 127, 160, 320, 4, precision="mixed", ltr=106, name="packed_l127_nf4"),
        # a training batch of mixed resolutions, one field each
        _case("uneven", 511, 512, 1024, 1, precision="mixed", members=32, sizes=7, name="uneven_32"),
    ]


# Drawn cases stay below this cost (FP64 flops of the largest listed case; mixed-precision
# flops count an eighth).
def _cost(c):
    f = work(c)["flops"] * (0.125 if c["precision"] == "mixed" else 1.0)
    if _max_prime(c["nlon"]) > 13:   # dense DFTs along longitude
        f += 8.0 * c["nlon"] ** 2 * c["nlat"] * c["nf"]
    return f


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    cap = _cost(_case("scalar", 1023, 1024, 2048, 64))
    while True:
        kind = rng.choice(["scalar", "scalar", "scalar", "vector", "divvort", "grad", "packed", "uneven"])
        precision = "fp64"
        if kind in ("scalar", "packed"):
            precision = rng.choice(["fp64", "mixed"])
        if kind == "uneven":
            precision = "mixed"
            return _case(kind, 511, 512, 1024, 1, precision="mixed", members=rng.randint(8, 32),
                         sizes=rng.randint(1, 10 ** 6))
        top = {"scalar": 1023, "vector": 511, "divvort": 340, "grad": 340, "packed": 511}[kind]
        nftop = {"scalar": 64, "vector": 16, "divvort": 32, "grad": 32, "packed": 16}[kind]
        lmax = _log_int(rng, 15, top)
        nf = _log_int(rng, 1, nftop)
        grid = rng.choice(["plain", "default", "odd", "dealiased"])
        nlat, nlon = lmax + 1, _smooth(2 * lmax + 2)
        if grid == "default":            # create_gauss_config's nlon, whatever its factors
            nlon = 2 * lmax + 2
            if _max_prime(nlon) > 13 and (lmax > 300 or nf > 8):
                continue
        elif grid == "odd":
            nlat = lmax + 1 + rng.randint(0, 9)
            nlon = _smooth(2 * lmax + 1 + rng.randint(0, 9))
        elif grid == "dealiased":
            nlat = (3 * lmax + 2) // 2
            nlon = _smooth(3 * lmax + 1)
        c = _case(kind, lmax, nlat, nlon, nf, precision=precision)
        if kind == "packed":
            c["ltr"] = lmax - rng.randint(0, lmax // 3)
        if kind == "scalar" and rng.random() < 0.25:
            c["mmax"] = max(1, (2 * lmax) // 3)
        if kind == "scalar" and lmax < 256 and rng.random() < 0.25:
            c["norm"] = rng.choice(["schmidt", "fourpi"])
        if _cost(c) <= cap:
            return c


def _member_sizes(case):
    r = np.random.default_rng(case["sizes"])
    return [int(v) for v in r.integers(31, case["lmax"] + 1, case["members"])]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _coeffs(lmax, mmax, nf, seed, power, lmin, dtype):
    """Complex coefficients ~ N(0,1)/(l+1)^power, zero for l < max(m, lmin), real at m = 0;
    shape (lmax+1, mmax+1, nf), l fastest in memory."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    z = torch.randn((nf, mmax + 1, lmax + 1, 2), dtype=torch.float64, device=dev, generator=g)
    l = torch.arange(lmax + 1, device=dev)
    m = torch.arange(mmax + 1, device=dev).view(-1, 1)
    keep = ((l >= m) & (l >= lmin)).to(torch.float64) / (l + 1.0) ** power
    z = z * keep[None, :, :, None]
    z[:, 0, :, 1] = 0
    return torch.view_as_complex(z).to(dtype).permute(2, 1, 0)


def _noise(nlat, nlon, nf, seed):
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    return torch.randn((nf, nlon, nlat), dtype=torch.float64, device=dev, generator=g).permute(2, 1, 0)


def _ctype(case):
    return torch.complex64 if case["precision"] == "mixed" else torch.complex128


def _inputs(case, seed):
    k, L, M, nf = case["kind"], case["lmax"], case["mmax"], case["nf"]
    s = 64 * seed
    if k == "scalar":
        return [_coeffs(L, M, nf, s, 1.0, 0, _ctype(case))]
    if k == "vector":
        return [_coeffs(L, M, nf, s, 1.0, 0, torch.complex128),
                _coeffs(L, M, 1, s + 1, 1.5, 1, torch.complex128)[:, :, 0],
                _coeffs(L, M, 1, s + 2, 1.5, 1, torch.complex128)[:, :, 0]]
    if k == "divvort":
        return [_coeffs(L, M, nf, s + i, 0.5, 1, torch.complex128) for i in range(2)]
    if k == "grad":
        return [_coeffs(L, M, nf, s, 1.0, 0, torch.complex128), _noise(case["nlat"], case["nlon"], nf, s + 1),
                _coeffs(L, M, 1, s + 2, 1.5, 1, torch.complex128), _coeffs(L, M, 1, s + 3, 1.5, 1, torch.complex128),
                _noise(case["nlat"], case["nlon"], 1, s + 4), _noise(case["nlat"], case["nlon"], 1, s + 5)]
    if k == "packed":
        a = _coeffs(L, M, nf, s, 1.0, 0, _ctype(case))
        q = torch.cat([a[m:, m, :] for m in range(M + 1)], dim=0)       # (nlm, nf)
        return [q.t().contiguous().t()]
    return [_coeffs(l, l, 1, s + i, 1.0, 0, torch.complex64) for i, l in enumerate(_member_sizes(case))]


def prepare(case, seed):
    ins = _inputs(case, seed)
    if case["kind"] == "uneven":
        cfgs = [sht.create_gauss_config(l, l + 1, nlon=_smooth(2 * l + 2)) for l in _member_sizes(case)]
        batch = UnevenBatch(cfgs, 1)
        for dst, src in zip(batch.alm_in, ins):
            dst.copy_(src)
        batch.autotune()
        return dict(case=case, batch=batch)
    cfg = sht.create_gauss_config(case["lmax"], case["nlat"], mmax=case["mmax"], nlon=case["nlon"], norm=case["norm"])
    if torch.cuda.is_available():
        cfg.plan(torch.cuda.current_device())
    return dict(case=case, cfg=cfg, ins=ins)


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "uneven":
        batch = state["batch"]
        batch.roundtrip()
        return list(batch.grid) + list(batch.alm_out)
    cfg, ins = state["cfg"], state["ins"]
    if k == "scalar":
        p = case["precision"]
        if case["nf"] == 1:
            f = sht.synthesis(cfg, ins[0][:, :, 0], precision=p)
            return f, sht.analysis(cfg, f, precision=p)
        f = sht.synthesis_batch(cfg, ins[0], precision=p)
        return f, sht.analysis_batch(cfg, f, precision=p)
    if k == "vector":
        f = sht.synthesis_batch(cfg, ins[0])
        a = sht.analysis_batch(cfg, f)
        vt, vp = sht.synthesis_sphtor(cfg, ins[1], ins[2])
        s, t = sht.analysis_sphtor(cfg, vt, vp)
        return f, a, vt, vp, s, t
    if k == "divvort":
        vt, vp = sht.synthesis_divvort_batch(cfg, ins[0], ins[1])
        d, z = sht.analysis_divvort_batch(cfg, vt, vp)
        return vt, vp, d, z
    if k == "grad":
        a, s, t = (ins[i].detach().requires_grad_(True) for i in (0, 2, 3))
        r = sht.synthesis_batch(cfg, a) - ins[1]
        vt, vp = sht.synthesis_sphtor_batch(cfg, s, t)
        rt, rp = vt - ins[4], vp - ins[5]
        loss = (r * r).sum() + (rt * rt).sum() + (rp * rp).sum()
        loss.backward()
        return loss.detach(), a.grad, s.grad, t.grad
    f = sht.synthesis_packed_batch(cfg, ins[0], lcap=case["ltr"], precision=case["precision"])
    return f, sht.analysis_packed_batch(cfg, f, lcap=case["ltr"], precision=case["precision"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _dims(case):
    if case["kind"] == "uneven":
        return [(l, l, l + 1, _smooth(2 * l + 2), 1) for l in _member_sizes(case)]
    return [(case["lmax"], case["mmax"], case["nlat"], case["nlon"], case["nf"])]


def work(case):
    """Legendre sums folded about the equator, 4 (nlat/2) nlm flops a field and direction, and
    real FFTs, 2.5 nlat nlon log2 nlon; coefficients and grids moved once per call."""
    k = case["kind"]
    r = 4 if case["precision"] == "mixed" else 8
    nbytes = flops = 0.0
    for lmax, mmax, nlat, nlon, nf in _dims(case):
        nlm = sum(lmax - m + 1 for m in range(mmax + 1))
        coef, grid = 2.0 * r * nlm, float(r) * nlat * nlon
        fld = 2.0 * nlat * nlm + 2.5 * nlat * nlon * math.log2(nlon)
        if k == "vector":
            n = nf + 2
        elif k == "divvort":
            n = 2 * nf
        elif k == "grad":
            n = nf + 2
        else:
            n = nf
        flops += 2 * n * fld
        nbytes += 2 * n * (coef + grid)
        if k == "grad":                  # the target grid, read once; residuals written and summed
            nbytes += n * grid
            flops += 3.0 * n * nlat * nlon
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # mixed: fp16x3 products and FP32 sums, 1e-7 to 3e-7 measured against 64 bits
    if case["precision"] == "mixed":
        return {"rel": 1.2e-6}
    # FP64: sums over up to 1024 degrees of recurrences whose rounding grows with the degree,
    # 1e-15 to 2.2e-13 measured (the vector gradients carry l(l+1)-weighted sums)
    return {"rel": 9e-13}


# ---------------------------------------------------------------------------
# the same outputs in plain torch float64
# ---------------------------------------------------------------------------

class _Exact:
    """Dense transforms on one grid: P[m, l, i] for l <= lmax + 1, orthonormal with the
    Condon-Shortley phase."""

    def __init__(self, lmax, mmax, nlat, nlon):
        self.lmax, self.mmax, self.nlat, self.nlon = lmax, mmax, nlat, nlon
        dev = self.dev = _device()
        # Gauss nodes, north first: Newton on P_n in 80-bit floats
        n = nlat
        i = np.arange(1, n + 1).astype(np.longdouble)
        x = np.cos(np.longdouble(math.pi) * (i - 0.25) / (n + 0.5))
        for _ in range(8):
            p0, p1 = np.ones_like(x), x.copy()
            for l in range(2, n + 1):
                p0, p1 = p1, ((2 * l - 1) * x * p1 - (l - 1) * p0) / l
            if n == 1:
                p0, p1 = np.ones_like(x), x
            dp = n * (x * p1 - p0) / (x * x - 1)
            x = x - p1 / dp
        s = np.sqrt((1 - x) * (1 + x))
        self.w = torch.tensor((2 / ((1 - x * x) * dp * dp)).astype(np.float64), device=dev)
        self.sint = torch.tensor(s.astype(np.float64), device=dev)
        xs = torch.tensor(x.astype(np.float64), device=dev)
        # sectoral seeds as mantissa and power of two, so that no order underflows at the poles
        mm = np.arange(mmax + 1)
        half = np.zeros(mmax + 1, dtype=np.longdouble)
        half[1:] = np.cumsum(np.log2((2 * mm[1:] + 1) / (2 * mm[1:].astype(np.longdouble))) / 2)
        lg = half[:, None] + mm[:, None] * np.log2(s)[None, :] - np.log2(4 * np.longdouble(np.pi)) / 2
        e = np.floor(lg)
        sgn = np.where(mm % 2, -1.0, 1.0)[:, None]
        cur = torch.tensor((sgn * np.exp2(lg - e)).astype(np.float64), device=dev)      # (m, lat)
        ex = torch.tensor(e.astype(np.int64), device=dev)
        prev = torch.zeros_like(cur)
        L1 = lmax + 1
        self.P = torch.zeros((mmax + 1, L1 + 1, nlat), dtype=torch.float64, device=dev)
        ms = torch.arange(mmax + 1, device=dev, dtype=torch.float64)
        val = torch.zeros_like(cur)
        up = torch.zeros_like(prev)
        exc = torch.zeros_like(ex)
        for l in range(L1 + 1):
            # orders m < l step the recurrence, order m = l starts from its seed
            k = min(l, mmax + 1)
            if k > 0:
                d2 = (l * l - ms[:k] ** 2)
                a = torch.sqrt((4.0 * l * l - 1) / d2)
                b = torch.sqrt(torch.clamp((2.0 * l + 1) * ((l - 1.0) ** 2 - ms[:k] ** 2) / ((2.0 * l - 3) * d2), min=0.0))
                new = a[:, None] * xs[None, :] * val[:k] - b[:, None] * up[:k]
                big = new.abs() > 2.0 ** 200
                up[:k] = torch.where(big, val[:k] * 2.0 ** -200, val[:k])
                val[:k] = torch.where(big, new * 2.0 ** -200, new)
                exc[:k] += torch.where(big, 200, 0)
            if l <= mmax:
                val[l], up[l], exc[l] = cur[l], 0.0, ex[l]
                k += 1
            ec = torch.clamp(exc[:k], min=-1200, max=1000)
            h = torch.div(ec, 2, rounding_mode="floor")
            two = torch.tensor(2.0, dtype=torch.float64, device=dev)
            self.P[:k, l] = val[:k] * torch.pow(two, h.double()) * torch.pow(two, (ec - h).double())
        # l-direction factors d(l, m) of sin(theta) dP/dtheta
        ll = torch.arange(L1 + 2, device=dev, dtype=torch.float64)
        self.d = torch.sqrt(torch.clamp((ll[None, :] ** 2 - ms[:, None] ** 2) / (4 * ll[None, :] ** 2 - 1), min=0.0))
        self.ms = ms

    def dp(self):
        """sin(theta) dP/dtheta for l <= lmax (m, l, lat)."""
        L = self.lmax
        l = torch.arange(L + 1, device=self.dev, dtype=torch.float64)
        out = (l * self.d[:, 1:L + 2])[:, :, None] * self.P[:, 1:L + 2]
        out[:, 1:] -= ((l[1:] + 1) * self.d[:, 1:L + 1])[:, :, None] * self.P[:, 0:L]
        return out

    @staticmethod
    def _mul(A, z):
        return torch.complex(torch.matmul(A, z.real.contiguous()), torch.matmul(A, z.imag.contiguous()))

    def bins(self, A, a):
        """sum_l A[m, l, i] a[l, m, k] -> (m, i, k)."""
        return self._mul(A.transpose(1, 2), a.permute(1, 0, 2).to(torch.complex128).contiguous())

    def grid(self, F):
        """Fourier bins (m, i, k) to the real grid (i, j, k)."""
        F = F.clone()
        F[0].imag.zero_()
        full = torch.zeros((self.nlon // 2 + 1,) + tuple(F.shape[1:]), dtype=torch.complex128, device=self.dev)
        full[: self.mmax + 1] = F
        return torch.fft.irfft(full, n=self.nlon, dim=0, norm="forward").permute(1, 0, 2)

    def fourier(self, f):
        return torch.fft.rfft(f.to(torch.float64).permute(1, 0, 2), dim=0)[: self.mmax + 1]

    def coef(self, A, F):
        """sum_i A[m, l, i] F[m, i, k] -> (l, m, k)."""
        return self._mul(A, F).permute(1, 0, 2)

    def scalar(self):
        return self.P[:, : self.lmax + 1]

    def synthesis(self, a):
        return self.grid(self.bins(self.scalar(), a))

    def analysis(self, f):
        F = self.fourier(f) * (2 * math.pi / self.nlon * self.w)[None, :, None]
        return self.coef(self.scalar(), F)

    def sphtor(self, S, T):
        D, Q = self.dp(), self.scalar()
        im = (1j * self.ms)[:, None, None]
        g = (1.0 / self.sint)[None, :, None]
        Ft = self.bins(D, S) - im * self.bins(Q, T)
        Fp = im * self.bins(Q, S) + self.bins(D, T)
        return self.grid(Ft * g), self.grid(Fp * g)

    def _adj(self, Ft, Fp):
        D, Q = self.dp(), self.scalar()
        im = (1j * self.ms)[None, :, None]
        s = self.coef(D, Ft) - im * self.coef(Q, Fp)
        t = im * self.coef(Q, Ft) + self.coef(D, Fp)
        return s, t

    def analysis_sphtor(self, vt, vp, inv_ll=True):
        g = (2 * math.pi / self.nlon * self.w / self.sint)[None, :, None]
        s, t = self._adj(self.fourier(vt) * g, self.fourier(vp) * g)
        l = torch.arange(self.lmax + 1, device=self.dev, dtype=torch.float64)
        q = torch.where(l > 0, 1.0 / torch.clamp(l * (l + 1), min=1.0) if inv_ll else torch.ones_like(l),
                        torch.zeros_like(l))
        return s * q[:, None, None], t * q[:, None, None]

    def order_weight(self):
        return torch.where(self.ms > 0, 2.0, 1.0)[None, :, None]


def exact(case, seed):
    ins = _inputs(case, seed)
    k, L, M = case["kind"], case["lmax"], case["mmax"]
    if k == "uneven":
        fs, As = [], []
        for a, l in zip(ins, _member_sizes(case)):
            ex = _Exact(l, l, l + 1, _smooth(2 * l + 2))
            f = ex.synthesis(a)
            fs.append(f)
            As.append(ex.analysis(f))
        return fs + As
    ex = _Exact(L, M, case["nlat"], case["nlon"])
    if k == "scalar":
        l = torch.arange(L + 1, device=ex.dev, dtype=torch.float64)[:, None, None]
        sc = {"orthonormal": torch.ones_like(l), "fourpi": torch.full_like(l, math.sqrt(4 * math.pi)),
              "schmidt": torch.sqrt(4 * math.pi / (2 * l + 1))}[case["norm"]]
        f = ex.synthesis(ins[0] * sc)
        a = ex.analysis(f) / sc
        return (f[:, :, 0], a[:, :, 0]) if case["nf"] == 1 else (f, a)
    if k == "vector":
        f = ex.synthesis(ins[0])
        vt, vp = ex.sphtor(ins[1][:, :, None], ins[2][:, :, None])
        s, t = ex.analysis_sphtor(vt, vp)
        return f, ex.analysis(f), vt[:, :, 0], vp[:, :, 0], s[:, :, 0], t[:, :, 0]
    if k == "divvort":
        l = torch.arange(L + 1, device=ex.dev, dtype=torch.float64)
        q = -1.0 / torch.clamp(l * (l + 1), min=1.0)[:, None, None]
        vt, vp = ex.sphtor(ins[0] * q, ins[1] * q)
        d, z = ex.analysis_sphtor(vt, vp, inv_ll=False)
        return vt, vp, -d, -z
    if k == "grad":
        r = ex.synthesis(ins[0]) - ins[1]
        vt, vp = ex.sphtor(ins[2], ins[3])
        rt, rp = vt - ins[4], vp - ins[5]
        loss = (r * r).sum() + (rt * rt).sum() + (rp * rp).sum()
        wm = ex.order_weight()
        ga = ex.coef(ex.scalar(), ex.fourier(2 * r)) * wm
        g = (1.0 / ex.sint)[None, :, None]
        gs, gt = ex._adj(ex.fourier(2 * rt) * g, ex.fourier(2 * rp) * g)
        return loss, ga, gs * wm, gt * wm
    # packed, truncated at ltr
    nf, ltr = case["nf"], case["ltr"]
    a = torch.zeros((L + 1, M + 1, nf), dtype=torch.complex128, device=ex.dev)
    o = 0
    for m in range(M + 1):
        a[m:, m, :] = ins[0][o:o + L - m + 1]
        o += L - m + 1
    a[ltr + 1:] = 0
    f = ex.synthesis(a)
    b = ex.analysis(f)
    b[ltr + 1:] = 0
    q = torch.cat([b[m:, m, :] for m in range(M + 1)], dim=0)
    return f.permute(2, 1, 0).reshape(nf, -1).permute(1, 0), q

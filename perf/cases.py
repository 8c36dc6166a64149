"""The transforms a user of this package runs, as cases that can be timed and checked.

A case is a dict of plain values with a ``kind``:

  sht      analysis of a batch of maps (``SHTCUDA``)
  isht     synthesis of a batch of coefficients (``iSHTCUDA``)
  round    analysis, then synthesis of its result
  layer    a spectral layer y = iSHT(w_l SHT(x)) with its backward pass
           (gradients with respect to x and w)
  vec      spin-1 analysis, then synthesis (``VectorSHTCUDA``, ``VectoriSHTCUDA``)
  regrid   HEALPix -> equiangular grid with its backward pass (``Regridding``)
  ragged   analysis and synthesis of several resolutions in one call
           (``RaggedSHT``, ``RaggedISHT``)
  remap    pixel reordering of a batch of maps (``nest2ring`` and the others)

``listed()`` gives the named ones, ``draw(rng)`` others of the same ranges:
nside 16 to 1024 (powers of two with ring weights, and others with uniform
weights), 1 to 64 maps, odd and even band limits, float32, float64 and the
fp16-split tensor-core precision.  ``exact`` restates the transforms in
float64 with torch alone.
"""

import math
import os

import numpy as np
import torch

import cuhpx_b200 as hpx

_WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(hpx.__file__)), "data", "ring_weights.npz")


# ----------------------------------------------------------------------- cases
def listed():
    return [
        # one map of a coarse grid through a module with its default band limit:
        # what an interactive user, or a model that looks at a map at a time, calls
        {"name": "sht_f32_n32_b1", "kind": "sht", "nside": 32, "lmax": 127, "mmax": 65, "batch": 1, "prec": "fp32",
         "weights": "ring", "refine": 0},
        # synthesis of a few channels on an odd grid size without ring weights
        {"name": "isht_f32_n96_b5", "kind": "isht", "nside": 96, "lmax": 191, "mmax": 177, "batch": 5, "prec": "fp32",
         "weights": "none", "refine": 0},
        # a spectral layer of a neural operator in training: 16 channels, forward and backward
        {"name": "layer_f32_n64_b16", "kind": "layer", "nside": 64, "lmax": 128, "mmax": 128, "batch": 16,
         "prec": "fp32", "weights": "ring", "refine": 0},
        # filtering a handful of fields at a common weather / climate resolution
        {"name": "round_f32_n256_b8", "kind": "round", "nside": 256, "lmax": 511, "mmax": 511, "batch": 8,
         "prec": "fp32", "weights": "ring", "refine": 0},
        # one sky map at full resolution in the default precision
        {"name": "round_f32_n1024_b1", "kind": "round", "nside": 1024, "lmax": 2047, "mmax": 2047, "batch": 1,
         "prec": "fp32", "weights": "ring", "refine": 0},
        # a bulk run in the default precision
        {"name": "round_f32_n512_b64", "kind": "round", "nside": 512, "lmax": 1023, "mmax": 1023, "batch": 64,
         "prec": "fp32", "weights": "ring", "refine": 0},
        # double precision with the default band limit (4 nside - 1, 2 nside + 1)
        {"name": "round_f64_n128_b4", "kind": "round", "nside": 128, "lmax": 511, "mmax": 257, "batch": 4,
         "prec": "fp64", "weights": "ring", "refine": 0},
        # the benchmark's headline step: 64 maps at nside 1024 on the tensor cores
        {"name": "round_f16x3_n1024_b64", "kind": "round", "nside": 1024, "lmax": 2047, "mmax": 2047, "batch": 64,
         "prec": "f16x3", "weights": "ring", "refine": 0},
        # analysis with one Jacobi iteration, a medium batch on the tensor cores
        {"name": "sht_f16x3_n256_b12_k1", "kind": "sht", "nside": 256, "lmax": 513, "mmax": 511, "batch": 12,
         "prec": "f16x3", "weights": "ring", "refine": 1},
        # winds: tangent fields to spheroidal / toroidal coefficients and back
        {"name": "vec_f32_n128_b4", "kind": "vec", "nside": 128, "lmax": 255, "mmax": 255, "batch": 4,
         "prec": "fp32"},
        # regridding inside a training step (forward and backward)
        {"name": "regrid_f32_n128_b8", "kind": "regrid", "nside": 128, "nlat": 256, "nlon": 512, "lmax": 255,
         "mmax": 255, "batch": 8, "prec": "fp32"},
        # a NEST archive's maps brought into RING order before a transform
        {"name": "remap_f32_n512_b16", "kind": "remap", "nside": 512, "batch": 16, "dtype": "float32",
         "src": "nest", "dst": "ring"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sht", "isht", "round", "round", "layer", "vec", "regrid", "ragged", "remap"])
    top = {"layer": 256, "vec": 256, "regrid": 256, "ragged": 512}.get(kind, 1024)
    if rng.random() < 0.7 or kind in ("layer", "vec", "regrid", "ragged", "remap"):
        nside, weights = 1 << rng.randint(4, int(math.log2(top))), "ring"
    else:
        nside, weights = _log_int(rng, 16, top), "none"
    batch = _log_int(rng, 1, 64)
    if kind == "remap":
        src, dst = rng.sample(["ring", "nest", "flat"], 2)
        return {"kind": kind, "nside": nside, "batch": batch, "dtype": rng.choice(["float32", "float64", "float16"]),
                "src": src, "dst": dst}
    if kind == "ragged":
        nsides = sorted(rng.sample([32, 64, 128, 256, 512], 3))
        return {"kind": kind, "nsides": ",".join(map(str, nsides)), "prec": rng.choice(["fp32", "f16x3"]),
                "batches": ",".join(str(_log_int(rng, 1, 16)) for _ in nsides)}
    lmax = rng.choice([2 * nside - 1, 2 * nside, int(rng.uniform(nside, 3 * nside if nside <= 512 else 2 * nside)) | 1])
    mmax = min(rng.choice([lmax, 2 * nside + 1, int(rng.uniform(0.5 * lmax, lmax)) | 1]), 2 * nside + 1)
    if kind == "regrid":
        return {"kind": kind, "nside": nside, "nlat": 2 * nside, "nlon": 4 * nside, "lmax": min(lmax, 2 * nside),
                "mmax": min(mmax, lmax, 2 * nside), "batch": min(batch, 16), "prec": rng.choice(["fp32", "fp32", "f16x3"])}
    if kind == "vec":
        return {"kind": kind, "nside": nside, "lmax": min(lmax, 2 * nside), "mmax": min(mmax, lmax, 2 * nside),
                "batch": min(batch, 16), "prec": rng.choice(["fp32", "fp32", "fp64"])}
    prec = rng.choice(["fp32", "fp32", "fp64", "f16x3"])
    case = {"kind": kind, "nside": nside, "lmax": lmax, "mmax": mmax, "batch": batch, "prec": prec,
            "weights": weights, "refine": rng.choice([0, 0, 1]) if kind == "sht" else 0}
    # no more work than the largest listed case of the precision would take
    limit = {"fp32": 512 ** 3 * 64, "fp64": 256 ** 3 * 16, "f16x3": 1024 ** 3 * 64}[prec] * 4.0
    while 1.0 * lmax * mmax * nside * case["batch"] > limit and case["batch"] > 1:
        case["batch"] = (case["batch"] + 1) // 2
    while 1.0 * case["lmax"] * case["mmax"] * case["nside"] > limit:
        case.update(nside=case["nside"] // 2, lmax=case["lmax"] // 2, mmax=case["mmax"] // 2)
    return case


# ---------------------------------------------------------------------- inputs
def _real(case):
    return torch.float64 if case["prec"] == "fp64" else torch.float32


def _fields(g, xyz, batch, dtype):
    """Smooth structure on many scales (plane waves through the sphere) plus noise."""
    n = xyz.shape[1]
    out = torch.empty(batch, n, dtype=dtype, device=xyz.device)
    for b in range(batch):
        k = torch.randn(12, 3, generator=g, device=xyz.device, dtype=torch.float64)
        k *= 2.0 ** torch.arange(12, device=xyz.device, dtype=torch.float64)[:, None] * 0.25
        ph = 6.28 * torch.rand(12, generator=g, device=xyz.device, dtype=torch.float64)
        f = 0.03 * torch.randn(n, generator=g, device=xyz.device, dtype=dtype)
        for i in range(12):
            wave = (k[i] @ xyz + ph[i]).to(torch.float32)
            f += (torch.cos(wave) / (i + 1.0)).to(dtype)
        out[b] = f
    return out


def _alm(g, batch, L, M, dtype, device):
    """Gaussian coefficients with C_l ~ (l+1)^-2, zero for m > l, real for m = 0."""
    a = torch.randn(batch, L, M, 2, generator=g, device=device, dtype=dtype)
    l = torch.arange(L, device=device)
    a /= (l + 1.0).to(dtype)[:, None, None]
    a *= (torch.arange(M, device=device)[None, :] <= l[:, None]).to(dtype)[..., None]
    a[:, :, 0, 1] = 0
    return torch.view_as_complex(a)


_last = None


def _inputs(case, seed, device):
    """Inputs alone (shared by prepare and exact)."""
    g = torch.Generator(device=device).manual_seed(1_000_003 * int(seed) + 17)
    kind = case["kind"]
    if kind == "remap":
        shape = (case["batch"], 12 * case["nside"] ** 2)
        return {"x": torch.randn(shape, generator=g, device=device).to(getattr(torch, case["dtype"]))}
    if kind == "ragged":
        return {"x": [_fields(g, _Sphere.healpix(n, "ring", device).xyz(), b, torch.float32)
                      for n, b in zip(_ints(case["nsides"]), _ints(case["batches"]))]}
    dt, B, L, M = _real(case), case["batch"], case["lmax"], case["mmax"]
    sp = _Sphere.healpix(case["nside"], case.get("weights", "ring"), device)
    if kind == "isht":
        return {"a": _alm(g, B, L, M, dt, device)}
    if kind == "vec":
        return {"x": _fields(g, sp.xyz(), 2 * B, dt).reshape(B, 2, -1)}
    s = {"x": _fields(g, sp.xyz(), B, dt)}
    if kind == "layer":
        s["w"] = 1.0 + 0.3 * torch.randn(L, 1, generator=g, device=device, dtype=dt)
        s["gy"] = torch.randn(s["x"].shape, generator=g, device=device, dtype=dt)
    if kind == "regrid":
        s["gy"] = torch.randn(B, case["nlat"], case["nlon"], generator=g, device=device, dtype=dt)
    return s


def _ints(text):
    return [int(t) for t in str(text).split(",")]


def prepare(case, seed):
    """Inputs on the GPU and the modules a program keeps (they share one cached plan per size)."""
    global _last
    key = repr(sorted(case.items()))
    if key != _last:
        hpx.clear_plan_cache()  # one case's plans at a time
        _last = key
    s = _inputs(case, seed, torch.device("cuda", torch.cuda.current_device()))
    s["case"], kind = case, case["kind"]
    if kind in ("sht", "isht", "round", "layer"):
        kw = dict(lmax=case["lmax"], mmax=case["mmax"], quad_weights=case["weights"])
        if case["prec"] != "fp64":
            kw["precision"] = case["prec"]
        s["sht"] = hpx.SHTCUDA(case["nside"], refine_iters=case["refine"], **kw)
        s["isht"] = hpx.iSHTCUDA(case["nside"], **kw)
        if kind == "layer":
            s["x"].requires_grad_(True)
            s["w"].requires_grad_(True)
    elif kind == "vec":
        s["sht"] = hpx.VectorSHTCUDA(case["nside"], case["lmax"], case["mmax"])
        s["isht"] = hpx.VectoriSHTCUDA(case["nside"], case["lmax"], case["mmax"])
    elif kind == "regrid":
        s["regrid"] = hpx.Regridding(hpx.Grid("healpix", case["nside"]),
                                     hpx.Grid("equiangular", (case["nlat"], case["nlon"])), lmax=case["lmax"],
                                     mmax=case["mmax"], precision=case["prec"])
        s["x"].requires_grad_(True)
    elif kind == "ragged":
        s["sht"] = hpx.RaggedSHT(_ints(case["nsides"]), precision=case["prec"])
        s["isht"] = hpx.RaggedISHT(_ints(case["nsides"]), precision=case["prec"])
    return s


# ------------------------------------------------------------------------- run
def _remap(x, nside, src, dst):
    flat = ("S", True)
    if src == "ring":
        return hpx.ring2nest(x, nside) if dst == "nest" else hpx.ring2flat(x, *flat, nside)
    if src == "nest":
        return hpx.nest2ring(x, nside) if dst == "ring" else hpx.nest2flat(x, *flat, nside)
    return hpx.flat2ring(x, *flat, nside) if dst == "ring" else hpx.flat2nest(x, *flat, nside)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "remap":
        return _remap(s["x"], case["nside"], case["src"], case["dst"])
    if kind == "sht":
        return s["sht"](s["x"])
    if kind == "isht":
        return s["isht"](s["a"])
    if kind in ("round", "vec", "ragged"):
        a = s["sht"](s["x"])
        return {"alm": a, "map": s["isht"](a)}
    if kind == "layer":
        y = s["isht"](s["w"] * s["sht"](s["x"]))
        gx, gw = torch.autograd.grad(y, (s["x"], s["w"]), s["gy"])
        return {"y": y.detach(), "gx": gx, "gw": gw}
    y = s["regrid"](s["x"])
    (gx,) = torch.autograd.grad(y, (s["x"],), s["gy"])
    return {"y": y.detach(), "gx": gx}


# ------------------------------------------------------------------------ work
def _ring_sizes(nside):
    """Pixels of the north rings and the equator."""
    return np.minimum(4 * (np.arange(2 * nside) + 1), 4 * nside)


def _legendre_flops(sizes, L, M):
    """4 flops per (ring pair, order, degree) of one real map: the mirrored rings share one sum."""
    mt = np.minimum(np.minimum(M, L), sizes // 2 + 1).astype(np.float64)
    return float(np.sum(4.0 * (mt * L - mt * (mt - 1) / 2)))


def _fft_flops(sizes):
    return float(np.sum(2 * 2.5 * sizes * np.log2(np.maximum(sizes, 2))))


def work(case):
    kind = case["kind"]
    if kind == "remap":
        el = {"float16": 2, "float32": 4, "float64": 8}[case["dtype"]]
        return {"bytes": 2.0 * el * case["batch"] * 12 * case["nside"] ** 2, "flops": 0.0}
    if kind == "ragged":
        out = {"bytes": 0.0, "flops": 0.0}
        for n, b in zip(_ints(case["nsides"]), _ints(case["batches"])):
            w = work({"kind": "round", "nside": n, "lmax": 2 * n - 1, "mmax": 2 * n - 1, "batch": b, "prec": "fp32"})
            out = {k: out[k] + w[k] for k in out}
        return out
    el = 8.0 if case["prec"] == "fp64" else 4.0
    N, L, M, B = case["nside"], case["lmax"], case["mmax"], case["batch"]
    sizes = _ring_sizes(N)
    one = _legendre_flops(sizes, L, M) + _fft_flops(sizes)
    maps, alm = el * B * 12 * N * N, 2 * el * B * L * M
    if kind in ("sht", "isht"):
        return {"bytes": maps + alm, "flops": B * one * (1 + 2 * case.get("refine", 0))}
    if kind == "round":
        return {"bytes": 2 * maps + alm, "flops": 2 * B * one}
    if kind == "layer":
        return {"bytes": 4 * maps, "flops": 4 * B * one}
    if kind == "vec":  # two components, two products each
        return {"bytes": 4 * maps + 2 * alm,
                "flops": 2 * B * (4 * _legendre_flops(sizes, L, M) + 2 * _fft_flops(sizes))}
    grid = np.full((case["nlat"] + 1) // 2, case["nlon"])
    return {"bytes": 2 * maps + 2 * el * B * case["nlat"] * case["nlon"],
            "flops": 2 * B * (one + _legendre_flops(grid, L, M) + _fft_flops(grid))}


# ----------------------------------------------------------------------- exact
class _Sphere:
    """Iso-latitude rings: pixels, first pixel, phase of the first pixel, cos and
    sin^2 of the colatitude and quadrature weight of each, north to south."""

    def __init__(self, nphi, phi0, z, s2, w, device):
        self.nphi, self.phi0, self.device = np.asarray(nphi), np.asarray(phi0, np.float64), device
        self.start = np.concatenate([[0], np.cumsum(self.nphi)])
        self.npix = int(self.start[-1])
        t = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=device)  # noqa: E731
        self.z, self.s2, self.w = t(z), t(s2), t(w)

    @classmethod
    def healpix(cls, nside, weights, device):
        t = np.arange(4 * nside - 1)
        i = np.minimum(t + 1, 4 * nside - 1 - t)  # ring counted from the nearer pole
        cap = i < nside
        nphi = 4 * np.minimum(i, nside)
        zn = np.where(cap, 1 - i ** 2 / (3.0 * nside ** 2), 4 / 3.0 - 2 * i / (3.0 * nside))
        u = i ** 2 / (3.0 * nside ** 2)
        s2 = np.where(cap, u * (2 - u), (1 - zn) * (1 + zn))
        phi0 = np.where(cap | ((t + 1 - nside) % 2 == 0), np.pi / nphi, 0.0)
        w = np.full(t.shape, 4 * np.pi / (12.0 * nside ** 2))
        if weights == "ring":
            with np.load(_WEIGHTS) as d:
                w = w * (1.0 + d["n%d" % nside][i - 1])
        return cls(nphi, phi0, np.where(t < 2 * nside, zn, -zn), s2, w, device)

    @classmethod
    def equiangular(cls, nlat, nlon, device):
        th = np.pi * np.arange(nlat) / (nlat - 1)
        z, s2 = np.cos(th), np.sin(th) ** 2
        s2[[0, -1]] = 0.0
        return cls(np.full(nlat, nlon), np.zeros(nlat), z, s2, np.zeros(nlat), device)

    def xyz(self):
        """Unit vectors of the pixels, [3, npix]."""
        ring = torch.repeat_interleave(torch.arange(len(self.nphi), device=self.device),
                                       torch.as_tensor(self.nphi, device=self.device), output_size=self.npix)
        n = torch.as_tensor(self.nphi, device=self.device)[ring].to(torch.float64)
        j = (torch.arange(self.npix, device=self.device) - torch.as_tensor(self.start[:-1], device=self.device)[ring])
        phi = torch.as_tensor(self.phi0, device=self.device)[ring] + 2 * np.pi * j.to(torch.float64) / n
        s = torch.sqrt(self.s2)[ring]
        return torch.stack([s * torch.cos(phi), s * torch.sin(phi), self.z[ring]])

    def _groups(self):
        """Runs of rings of equal size: (first ring, count, size)."""
        cut = np.flatnonzero(np.diff(self.nphi)) + 1
        lo = np.concatenate([[0], cut])
        hi = np.concatenate([cut, [len(self.nphi)]])
        return [(int(a), int(b - a), int(self.nphi[a])) for a, b in zip(lo, hi)]

    def _phase(self, r, c, k):
        m = torch.arange(k, device=self.device, dtype=torch.float64)
        ang = torch.as_tensor(self.phi0[r:r + c], device=self.device)[:, None] * m
        return torch.polar(torch.ones_like(ang), ang)

    def spectra(self, f, M):
        """[B, npix] real -> X[M, R, B] with X_m = sum_j f_j e^{-i m phi_j}, m <= nphi / 2."""
        X = torch.zeros(M, len(self.nphi), f.shape[0], dtype=torch.complex128, device=self.device)
        for r, c, n in self._groups():
            k = min(M, n // 2 + 1)
            s = int(self.start[r])
            F = torch.fft.rfft(f[:, s:s + c * n].reshape(-1, c, n).to(torch.float64))[..., :k]
            X[:k, r:r + c] = (F * self._phase(r, c, k).conj()).permute(2, 1, 0)
        return X

    def maps(self, X):
        """Ring spectra X[M, R, B] -> [B, npix]: f_j = Re X_0 + 2 sum Re X_m e^{i m phi_j} (the last
        order of a ring counts once)."""
        f = torch.empty(X.shape[2], self.npix, dtype=torch.float64, device=self.device)
        for r, c, n in self._groups():
            k = min(X.shape[0], n // 2 + 1)
            S = X[:k, r:r + c].permute(2, 1, 0) * self._phase(r, c, k)
            S[..., 0].imag.zero_()
            if 2 * (k - 1) == n:
                S[..., -1].imag.zero_()
            s = int(self.start[r])
            f[:, s:s + c * n] = torch.fft.irfft(S, n=n, norm="forward").reshape(-1, c * n)
        return f

    def adjoint_scale(self, M):
        """[M, R]: 2 for the orders a real ring counts twice, 1 for m = 0 and m = nphi / 2, 0 above."""
        m = torch.arange(M, device=self.device)[:, None]
        h = torch.as_tensor(self.nphi // 2, device=self.device)[None, :]
        return torch.where((m == 0) | (m == h), 1.0, torch.where(m < h, 2.0, 0.0)).to(torch.float64)

    def legendre(self, L, M):
        """Yield (l, P[M, R]): orthonormal Legendre values without the (-1)^m sign, zero for m > l.
        Values are carried with a binary exponent of their own, so that none underflows on the way."""
        m = torch.arange(M, device=self.device, dtype=torch.float64)
        lg = torch.zeros(M, device=self.device, dtype=torch.float64)
        lg[1:] = 0.5 * torch.cumsum(torch.log2((2 * m[1:] + 1) / (2 * m[1:])), 0)
        lg = lg - 0.5 * math.log2(4 * math.pi)
        start = lg[:, None] + torch.where(m[:, None] == 0, torch.zeros_like(self.z), 0.5 * m[:, None] * torch.log2(self.s2))
        E = torch.floor(start)
        mant = torch.where(torch.isfinite(start), torch.exp2(start - E), torch.zeros_like(start))
        E = torch.where(torch.isfinite(E), E, torch.full_like(E, -5000.0))
        p, pm = torch.zeros_like(mant), torch.zeros_like(mant)
        scale = None
        for l in range(L):
            k = min(l, M)  # orders below l step, order l starts
            if k:
                q, fl = m[:k], float(l)
                a = torch.sqrt((2 * fl - 1) / (fl - q) * (2 * fl + 1) / (fl + q))
                b = torch.sqrt((fl + q - 1) / (fl - q) * (2 * fl + 1) / max(2 * fl - 3, 1.0) * (fl - q - 1) / (fl + q))
                new = torch.mul(p[:k], self.z).mul_(a[:, None]).sub_(pm[:k] * b[:, None])
                pm[:k] = p[:k]
                p[:k] = new
            if l < M:
                p[l] = mant[l]
            if l % 16 == 0:
                big = p.abs() > 2.0 ** 300
                p, pm = torch.where(big, p * 2.0 ** -300, p), torch.where(big, pm * 2.0 ** -300, pm)
                E = torch.where(big, E + 300.0, E)
                scale = torch.where(E > -1000.0, torch.exp2(E.clamp(min=-1000.0)), torch.zeros_like(E))
            yield l, p * scale

    def blocks(self, L, M, step=16):
        """Legendre values by blocks of degrees: (first degree, P[M, degrees, R])."""
        blk, l0 = None, 0
        for l, P in self.legendre(L, M):
            if l % step == 0:
                l0, blk = l, torch.empty(M, min(step, L - l), len(self.nphi), dtype=torch.float64, device=self.device)
            blk[:, l - l0] = P
            if l - l0 == blk.shape[1] - 1:
                yield l0, blk

    def analysis(self, X, L):
        """a[B, L, M] = sum over rings of P X."""
        M, R, B = X.shape
        out = torch.empty(B, L, M, dtype=torch.complex128, device=self.device)
        Xr = torch.view_as_real(X).reshape(M, R, 2 * B)
        for l0, P in self.blocks(L, M):
            v = torch.bmm(P, Xr).reshape(M, P.shape[1], B, 2)
            out[:, l0:l0 + P.shape[1]] = torch.view_as_complex(v).permute(2, 1, 0)
        return out

    def synthesis(self, a, M):
        """X[M, R, B] = sum over degrees of P a."""
        B, L, _ = a.shape
        acc = torch.zeros(M, len(self.nphi), 2 * B, dtype=torch.float64, device=self.device)
        for l0, P in self.blocks(L, M):
            A = torch.view_as_real(a[:, l0:l0 + P.shape[1]].permute(2, 1, 0).contiguous()).reshape(M, -1, 2 * B)
            acc.baddbmm_(P.transpose(1, 2), A)
        return torch.view_as_complex(acc.reshape(M, -1, B, 2))

    def sht(self, f, L, M, refine=0):
        a = self.analysis(self.spectra(f, M) * self.w[:, None], L)
        for _ in range(refine):
            a = a + self.analysis(self.spectra(f.to(torch.float64) - self.isht(a, M), M) * self.w[:, None], L)
        return a

    def isht(self, a, M):
        return self.maps(self.synthesis(a, M))

    def sht_adjoint(self, g, M):
        """Transpose of sht with respect to <x, y> = sum Re(conj(x) y)."""
        c = self.adjoint_scale(M)
        half = torch.where(c > 1, 0.5, c)
        return self.maps(self.synthesis(g, M) * (half * self.w)[..., None])

    def isht_adjoint(self, g, L, M):
        return self.analysis(self.spectra(g, M) * self.adjoint_scale(M)[..., None], L)

    # ---- spin 1: D0, D1 of the derivative table, odd orders negated
    def _vector_rows(self, L, M):
        m = torch.arange(M, device=self.device, dtype=torch.float64)[:, None]
        sign = (1.0 - 2.0 * (m % 2))
        rows = None
        for l, P in self.legendre(L + 1, M + 1):
            low = torch.cat([-P[1:2], P[:M - 1]])  # order m - 1 (order -1 is minus order 1)
            high = P[1:M + 1]
            if rows is not None:
                k = float(l - 1)
                h = 0.5 * math.sqrt((2 * k + 1) / (2 * k + 3))
                in_l = m <= k
                d1 = h * (torch.sqrt(((k - m + 1) * (k - m + 2)).clamp(min=0)) * low
                          + torch.sqrt((k + m + 1) * (k + m + 2)) * high)
                yield l - 1, rows, torch.where(in_l & (m > 0), d1 * sign, torch.zeros_like(d1))
            k = float(l)
            d0 = 0.5 * (torch.sqrt(((k + m) * (k - m + 1)).clamp(min=0)) * low
                        - torch.sqrt(((k - m) * (k + m + 1)).clamp(min=0)) * high)
            rows = torch.where(m <= k, d0 * sign, torch.zeros_like(d0))

    def vsht(self, f, L, M):
        B = f.shape[0]
        X = self.spectra(f.reshape(2 * B, -1), M) * self.w[:, None]
        Xr = torch.view_as_real(X).reshape(M, -1, 4 * B)
        out = torch.empty(B, 2, L, M, dtype=torch.complex128, device=self.device)
        for l, d0, d1 in self._vector_rows(L, M):
            v = torch.view_as_complex(torch.bmm(torch.stack([d0, d1], 1), Xr).reshape(M, 2, B, 2, 2))
            nf = 1.0 / (l * (l + 1)) if l else 1.0
            out[:, 0, l] = nf * (v[:, 0, :, 0] - 1j * v[:, 1, :, 1]).T
            out[:, 1, l] = nf * (-v[:, 0, :, 1] - 1j * v[:, 1, :, 0]).T
        return out

    def visht(self, a, M):
        B, _, L, _ = a.shape
        X = torch.zeros(M, len(self.nphi), B, 2, dtype=torch.complex128, device=self.device)
        for l, d0, d1 in self._vector_rows(L, M):
            S, T = a[:, 0, l].T[:, None], a[:, 1, l].T[:, None]  # [M, 1, B]
            d0, d1 = d0[..., None], d1[..., None]
            X[..., 0] += d0 * S + 1j * d1 * T
            X[..., 1] += -d0 * T + 1j * d1 * S
        return self.maps(X.reshape(M, -1, 2 * B)).reshape(B, 2, -1)


def exact(case, seed):
    """What run() returns, in float64."""
    kind = case["kind"]
    if kind == "remap":
        return None  # bytes moved, none computed
    device = torch.device("cuda", torch.cuda.current_device())
    with torch.no_grad():
        s = _inputs(case, seed, device)
        if kind == "ragged":
            alm, maps = [], []
            for n, x in zip(_ints(case["nsides"]), s["x"]):
                sp = _Sphere.healpix(n, "ring", device)
                alm.append(sp.sht(x, 2 * n - 1, 2 * n - 1))
                maps.append(sp.isht(alm[-1], 2 * n - 1))
            return {"alm": alm, "map": maps}
        L, M = case["lmax"], case["mmax"]
        sp = _Sphere.healpix(case["nside"], case.get("weights", "ring"), device)
        if kind == "sht":
            return sp.sht(s["x"], L, M, case["refine"])
        if kind == "isht":
            return sp.isht(s["a"].to(torch.complex128), M)
        if kind == "round":
            a = sp.sht(s["x"], L, M)
            return {"alm": a, "map": sp.isht(a, M)}
        if kind == "vec":
            a = sp.vsht(s["x"], L, M)
            return {"alm": a, "map": sp.visht(a, M)}
        if kind == "layer":
            w = s["w"].to(torch.float64)
            a = sp.sht(s["x"], L, M)
            y = sp.isht(w * a, M)
            ga = sp.isht_adjoint(s["gy"].to(torch.float64), L, M)
            gw = (a.conj() * ga).real.sum((0, 2))[:, None]
            return {"y": y, "gx": sp.sht_adjoint(w * ga, M), "gw": gw}
        ll = _Sphere.equiangular(case["nlat"], case["nlon"], device)
        y = ll.isht(sp.sht(s["x"], L, M), M).reshape(case["batch"], case["nlat"], case["nlon"])
        g = s["gy"].reshape(case["batch"], -1).to(torch.float64)
        return {"y": y, "gx": sp.sht_adjoint(ll.isht_adjoint(g, L, M), M)}

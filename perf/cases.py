"""The work that users of this framework have it do, as timed cases.

Each case is one call through the public entry points: the Python API
(`ccfj.fj_noise`, `ccfj.fj_earthquake`, ...) on host arrays, or the C ABI
(include/ccfj_b200.h) on device-resident arrays, as a program that keeps its
spectra on the GPU calls it. Sizes are those of this repository's tests and
benchmark workloads, and sizes between them.

`exact` restates each transform in 64 bits: Gauss-Legendre quadrature of the
linearly interpolated spectrum times r Z0(k r) on pieces that are short
against the wavelength (or the trapezoid sum), with torch's Bessel functions.
"""
import ctypes
import math
import os
import sys
import warnings

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cc-fjpy_b200"))

import ccfj  # noqa: E402
from ccfj import _batch, _cc, _eq, _lib  # noqa: E402


# ------------------------------------------------------------------ cases
def listed():
    return [
        # A first look at a small array from a notebook: host arrays, the
        # call's fixed cost is what counts (the tests' small case).
        dict(name="noise_notebook", kind="noise", host=True, nr=60, nf=40, nc=50, itype=1, func=0,
             fstride=1, rmin=1e3, rmax=5e4, spread="uniform", fmin=0.01, fmax=1.0, cmin=1000.0,
             cmax=5000.0),
        # A small array on the GPU (the benchmark's small workload).
        dict(name="noise_small", kind="noise", host=False, nr=200, nf=512, nc=300, itype=1, func=0,
             fstride=1, rmin=1e3, rmax=5e4, spread="uniform", fmin=0.01, fmax=1.0, cmin=1000.0,
             cmax=5000.0),
        # Both bases (Hankel): a 50-station array; an odd velocity count.
        dict(name="noise_hankel", kind="noise", host=False, nr=1225, nf=512, nc=401, itype=1,
             func=1, fstride=1, rmin=5e2, rmax=1e5, spread="array", fmin=0.01, fmax=1.5,
             cmin=800.0, cmax=4500.0),
        # The trapezoid rule on every second column, 100 stations, odd sizes.
        dict(name="noise_trapezoid", kind="noise", host=False, nr=4950, nf=1001, nc=501, itype=0,
             func=0, fstride=2, rmin=5e2, rmax=2e5, spread="array", fmin=0.01, fmax=1.5,
             cmin=800.0, cmax=4500.0),
        # 100 stations through the Python API, from and to host arrays.
        dict(name="noise_host", kind="noise", host=True, nr=4950, nf=1024, nc=500, itype=1, func=0,
             fstride=1, rmin=5e2, rmax=2e5, spread="array", fmin=0.01, fmax=1.5, cmin=800.0,
             cmax=4500.0),
        # A dense array's all pairs of 200 stations (the benchmark's headline).
        dict(name="noise_large", kind="noise", host=False, nr=19900, nf=2048, nc=1000, itype=1,
             func=0, fstride=1, rmin=5e2, rmax=4e5, spread="array", fmin=0.005, fmax=2.0,
             cmin=500.0, cmax=5000.0),
        # Earthquake records of a network (the benchmark's workload).
        dict(name="earthquake", kind="earthquake", host=False, nr=500, npts=8192, Fs=20.0, nf=1024,
             nc=800, itype=1, func=0, rmin=1e4, rmax=2e6, cmin=2000.0, cmax=5000.0),
        # A few records through the Python API with the Hankel basis; a
        # window length that is not a power of two.
        dict(name="earthquake_host", kind="earthquake", host=True, nr=60, npts=3000, Fs=10.0,
             nf=300, nc=201, itype=1, func=1, rmin=2e4, rmax=4e5, cmin=2000.0, cmax=5000.0),
        # Group-velocity windows over a network's records: many windows share
        # the geometry.
        dict(name="windows", kind="mwfj", host=False, nr=400, npts=8192, Fs=10.0, nf=512, nc=800,
             nwin=32, itype=1, func=0, rmin=5e3, rmax=1.5e6, cmin=1500.0, cmax=5000.0),
        # Subarrays of a dense deployment, uneven in size, in one call.
        dict(name="subarrays", kind="batch", host=False, nsets=128, nrmin=50, nrmax=20000, nf=512,
             nc=500, itype=1, func=0, rmin=5e2, rmax=3e5, fmin=0.01, fmax=1.0, cmin=1000.0,
             cmax=5000.0),
        # A quarter of a day of continuous records to cross-spectra (the
        # reference example's window shape: 14,400 samples, 0.9 overlap).
        dict(name="cross_spectra", kind="cc", host=False, nsta=100, npts=86400, fftlen=14400,
             overlap=0.9, nf=1000, fstride=3, onebit=0, whiten=1),
        # Records to a dispersion spectrum from host arrays, one call.
        dict(name="records_to_spectrum", kind="cc_noise", host=True, nsta=24, npts=43200,
             fftlen=7200, overlap=0.75, nf=501, fstride=2, onebit=0, whiten=1, nc=300, itype=1,
             func=0, Fs=4.0, rmin=1e3, rmax=8e4, cmin=1000.0, cmax=4500.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: sizes log-uniform, odd ones
    included, bounded so that none costs more than the largest listed."""
    kind = rng.choice(["noise", "noise", "noise", "earthquake", "mwfj", "batch", "cc", "cc_noise"])
    if kind == "noise":
        while True:
            nr, nf, nc = _logint(rng, 20, 19900), _logint(rng, 30, 2048), _logint(rng, 40, 1000)
            if nr * nf * nc <= 1e10:
                break
        return dict(kind="noise", host=rng.random() < 0.4, nr=nr, nf=nf, nc=nc,
                    itype=int(rng.random() < 0.75), func=int(rng.random() < 0.3),
                    fstride=rng.choice([1, 1, 1, 2]), rmin=rng.choice([2e2, 5e2, 1e3]),
                    rmax=rng.uniform(3e4, 4e5), spread=rng.choice(["uniform", "array"]),
                    fmin=rng.choice([0.005, 0.01, 0.05]), fmax=rng.uniform(0.5, 2.0),
                    cmin=rng.uniform(500.0, 1500.0), cmax=rng.uniform(3000.0, 5000.0))
    if kind == "earthquake":
        npts = rng.choice([1024, 2048, 4096, 8192, _logint(rng, 600, 4000)])
        return dict(kind=kind, host=rng.random() < 0.4, nr=_logint(rng, 16, 500), npts=npts,
                    Fs=rng.choice([10.0, 20.0]), nf=_logint(rng, 30, min(1024, npts // 2)),
                    nc=_logint(rng, 40, 800), itype=int(rng.random() < 0.8),
                    func=int(rng.random() < 0.3), rmin=rng.choice([5e3, 1e4, 2e4]),
                    rmax=rng.uniform(2e5, 2e6), cmin=rng.uniform(1500.0, 2500.0), cmax=5000.0)
    if kind == "mwfj":
        npts = rng.choice([1024, 2048, 4096, 8192])
        return dict(kind=kind, host=False, nr=_logint(rng, 16, 400), npts=npts, Fs=10.0,
                    nf=_logint(rng, 24, min(512, npts // 2)), nc=_logint(rng, 40, 800),
                    nwin=_logint(rng, 2, 32), itype=1, func=int(rng.random() < 0.2), rmin=5e3,
                    rmax=rng.uniform(2e5, 1.5e6), cmin=rng.uniform(1500.0, 2500.0), cmax=5000.0)
    if kind == "batch":
        nsets = _logint(rng, 4, 64)
        return dict(kind=kind, host=rng.random() < 0.3, nsets=nsets, nrmin=_logint(rng, 20, 60),
                    nrmax=_logint(rng, 100, 4000), nf=_logint(rng, 30, 400),
                    nc=_logint(rng, 40, 500), itype=int(rng.random() < 0.8),
                    func=int(rng.random() < 0.25), rmin=5e2, rmax=rng.uniform(5e4, 3e5), fmin=0.01,
                    fmax=rng.uniform(0.5, 1.5), cmin=rng.uniform(800.0, 1500.0), cmax=5000.0)
    fftlen = rng.choice([3600, 4096, 7200, 8192, 14400])
    npts = fftlen * rng.randint(3, 6)
    fstride = rng.choice([1, 2, 3])
    nf = _logint(rng, 64, min(1000, fftlen // (2 * fstride)))
    # one-bit records or whitened spectra: a one-bit window has bins that are
    # zero to rounding, which whitening turns into arbitrary phases
    onebit = int(rng.random() < 0.3)
    base = dict(kind=kind, host=kind == "cc_noise", nsta=_logint(rng, 6, 60), npts=npts,
                fftlen=fftlen, overlap=rng.choice([0.5, 0.75, 0.9]), nf=nf, fstride=fstride,
                onebit=onebit, whiten=1 - onebit)
    if kind == "cc_noise":
        base.update(nc=_logint(rng, 40, 500), itype=1, func=int(rng.random() < 0.25), Fs=4.0,
                    rmin=1e3, rmax=rng.uniform(3e4, 2e5), cmin=rng.uniform(800.0, 1500.0),
                    cmax=4500.0)
    return base


# ----------------------------------------------------------------- inputs
def _f32(x):
    return np.ascontiguousarray(x, dtype=np.float32)


def _distances(rng, nr, rmin, rmax, spread):
    """Pair distances in no particular order: uniform, log-uniform (epicentral
    distances) or those of stations scattered over a square."""
    if spread == "log":
        return np.exp(rng.uniform(math.log(rmin), math.log(rmax), nr))
    if spread == "uniform":
        return rng.uniform(rmin, rmax, nr)
    n = int(math.ceil((1 + math.sqrt(1 + 8 * nr)) / 2))
    xy = rng.uniform(0.0, rmax / math.sqrt(2.0), (n, 2))
    i, j = np.triu_indices(n, k=1)
    pick = rng.permutation(len(i))[:nr]
    return np.maximum(np.hypot(xy[i, 0] - xy[j, 0], xy[i, 1] - xy[j, 1])[pick], rmin)


def _c_law(f):
    return 2000.0 + 1500.0 * torch.exp(-f / 0.2)


def _spectra(seed, r, f, sigma=0.2):
    """complex64 [nr, nf] on the GPU: a fundamental mode and an overtone of
    the dispersion law, and noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.from_numpy(np.asarray(r, dtype=np.float64)).cuda()
    f = torch.from_numpy(np.asarray(f, dtype=np.float64)).cuda()
    k0, k1 = 2 * math.pi * f / _c_law(f), 2 * math.pi * f / (_c_law(f) + 800.0)
    out = torch.empty((len(r), len(f)), dtype=torch.complex64, device="cuda")
    for a in range(0, len(r), 2048):
        x = r[a:a + 2048, None]
        out.real[a:a + 2048] = (torch.special.bessel_j0((x * k0).float()) +
                                0.5 * torch.special.bessel_j0((x * k1).float()))
        out.imag[a:a + 2048] = 0.0
    v = torch.view_as_real(out)
    for a in range(0, len(r), 2048):
        v[a:a + 2048] += sigma * torch.randn(v[a:a + 2048].shape, generator=g, device="cuda")
    return out


def _records(seed, r, npts, Fs, fc=0.1, snr=5.0):
    """float32 [n, npts] on the GPU: dispersed Ricker wavelets and noise."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.from_numpy(np.asarray(r, dtype=np.float64)).cuda()
    fb = torch.arange(npts // 2 + 1, dtype=torch.float64, device="cuda") * Fs / npts
    w = fb ** 2 * torch.exp(-(fb / fc) ** 2)
    ph = -2 * math.pi * fb[None] * r[:, None] / _c_law(fb.clamp(min=1e-3))[None]
    u = torch.fft.irfft(torch.polar(w[None].expand_as(ph), ph), n=npts, dim=1)
    u = u / u.std(dim=1, keepdim=True)
    u = u + torch.randn(u.shape, generator=g, device="cuda", dtype=torch.float64) / snr
    return u.float().contiguous()


def _inputs(case, seed):
    """The host-side arrays and the GPU tensors that one call reads."""
    rng = np.random.default_rng(seed)
    d = dict(case=case)
    kind = case["kind"]
    if kind in ("noise", "batch", "earthquake", "mwfj", "cc_noise"):
        d["c"] = np.linspace(case["cmin"], case["cmax"], case["nc"])
    if kind == "noise":
        d["r"] = _distances(rng, case["nr"], case["rmin"], case["rmax"], case["spread"])
        ncols = case["nf"] * case["fstride"]
        ff = np.linspace(case["fmin"], case["fmax"], ncols)
        d["f"] = ff[::case["fstride"]]
        d["u"] = _spectra(seed, d["r"], ff)
    elif kind == "batch":
        n = np.exp(rng.uniform(math.log(case["nrmin"]), math.log(case["nrmax"]), case["nsets"]))
        d["rs"] = [rng.uniform(case["rmin"], case["rmax"], int(k)) for k in n]
        d["f"] = np.linspace(case["fmin"], case["fmax"], case["nf"])
        d["u"] = _spectra(seed, np.concatenate(d["rs"]), d["f"])
    elif kind in ("earthquake", "mwfj"):
        d["r"] = _distances(rng, case["nr"], case["rmin"], case["rmax"], "log")
        d["f"] = case["Fs"] * np.arange(case["nf"]) / case["npts"]
        d["u"] = _records(seed, d["r"], case["npts"], case["Fs"])
        if kind == "mwfj":
            # windows around group arrivals, a tenth to a quarter of the record
            L = rng.integers(case["npts"] // 10, case["npts"] // 4, (case["nwin"], case["nr"]))
            s = rng.integers(0, case["npts"] - L)
            d["winl"], d["winr"], d["taper"] = s / case["Fs"], (s + L) / case["Fs"], 0.9
    else:
        # ambient noise: a common wavefield delayed by station, plus local noise
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, npts = case["nsta"], case["npts"]
        src = torch.randn(npts + 4096, generator=g, device="cuda")
        x = torch.randn((n, npts), generator=g, device="cuda")
        for i, lag in enumerate(rng.integers(0, 4096, n)):
            x[i] += src[lag:lag + npts]
        d["x"] = x
        d["pairs"] = ccfj.GetStationPairs(n)
        d["startend"] = np.stack([rng.integers(0, npts // 8, n),
                                  npts - rng.integers(0, npts // 8, n)], 1).reshape(-1).astype(np.int32)
        if kind == "cc_noise":
            d["r"] = _distances(rng, n * (n - 1) // 2, case["rmin"], case["rmax"], "uniform")
            d["f"] = case["Fs"] * np.arange(case["nf"]) * case["fstride"] / case["fftlen"] + 1e-3
    return d


def _sorted_on_gpu(d):
    idx = np.argsort(d["r"])
    return dict(r=torch.from_numpy(_f32(d["r"][idx])).cuda(),
                perm=torch.from_numpy(idx.astype(np.int64)).cuda(),
                f=torch.from_numpy(_f32(d["f"])).cuda(), c=torch.from_numpy(_f32(d["c"])).cuda())


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    d = _inputs(case, seed)
    s = dict(case=case)
    kind = case["kind"]
    if case["host"]:
        for k in ("r", "rs", "f", "c", "pairs", "startend"):
            if k in d:
                s[k] = d[k]
        if kind == "batch":
            off = np.cumsum([0] + [len(r) for r in d["rs"]])
            u = d["u"].cpu().numpy()
            s["us"] = [u[a:b] for a, b in zip(off[:-1], off[1:])]
        elif "u" in d:
            s["u"] = d["u"].cpu().numpy()
        if "x" in d:
            s["x"] = d["x"].cpu().numpy().reshape(-1)
        return s
    if kind == "cc":
        a = _cc.CcArgs()
        a.struct_size = ctypes.sizeof(a)
        a.nsta, a.npts, a.nf = case["nsta"], case["npts"], case["nf"]
        a.npairs, a.fstride = len(d["pairs"]) // 2, case["fstride"]
        a.fftlen, a.steplen = case["fftlen"], int(case["fftlen"] * (1 - case["overlap"]))
        a.onebit, a.whiten, a.device_ptrs, a.accumulate, a.out_layout = case["onebit"], case["whiten"], 1, 0, 1
        s["out"] = torch.empty((a.npairs, a.nf), dtype=torch.complex64, device="cuda")
        s["keep"] = (d["pairs"], d["startend"], d["x"])
        a.pairs, a.startend = d["pairs"].ctypes.data, d["startend"].ctypes.data
        a.data, a.out_re, a.out_im = d["x"].data_ptr(), s["out"].data_ptr(), None
        s["args"] = a
        return s
    if kind == "batch":
        d["r"] = np.concatenate(d["rs"])
        off = np.cumsum([0] + [len(r) for r in d["rs"]]).astype(np.int64)
        perm = np.concatenate([o + np.argsort(r) for o, r in zip(off, d["rs"])]).astype(np.int64)
        t = dict(off=torch.from_numpy(off).cuda(), perm=torch.from_numpy(perm).cuda(),
                 r=torch.from_numpy(_f32(d["r"][perm])).cuda(),
                 f=torch.from_numpy(_f32(d["f"])).cuda(), c=torch.from_numpy(_f32(d["c"])).cuda())
        a = _batch.BatchArgs()
        a.nsets, a.variant, a.use_graph = len(d["rs"]), 0, 0
        a.offsets, a.total_pairs = t["off"].data_ptr(), int(off[-1])
        rows, shape = int(off[-1]), (len(d["rs"]), case["nc"], case["nf"])
    else:
        t = _sorted_on_gpu(d)
        rows, shape = case["nr"], (case["nc"], case["nf"])
        if kind == "noise":
            a = _lib.FjArgs()
            a.nr = rows
        else:
            a = _eq.EqArgs()
            a.ntr, a.npts, a.func = rows, case["npts"], case["func"]
            a.u, a.u_ld, a.u_rows, a.fstride = d["u"].data_ptr(), case["npts"], rows, 1
            if kind == "mwfj":
                shape = (case["nwin"],) + shape
                wins = _eq._win_params(case["npts"], case["Fs"], d["winl"], d["winr"], d["taper"])
                t["wins"] = [torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in wins]
                a.nwin = case["nwin"]
                a.win_n1, a.win_n2, a.win_delta = (w.data_ptr() for w in t["wins"])
    if kind in ("noise", "batch"):
        a.mode = _lib.MODE_J if case["func"] == 0 else _lib.MODE_J_MINUS_Y
        a.hilbert = case["func"]
        stride = case.get("fstride", 1)
        a.u[0] = d["u"].data_ptr()
        a.u_ld, a.u_rows, a.u_es = 2 * d["u"].shape[1], rows, 2
        a.u_ncols, a.fstride = d["u"].shape[1], stride
    a.struct_size = ctypes.sizeof(a)
    a.nf, a.nc, a.itype = case["nf"], case["nc"], case["itype"]
    a.precision, a.normalize, a.device_ptrs = _lib.PREC_FP32, 1, 1
    a.perm, a.r, a.f, a.c = (t[k].data_ptr() for k in ("perm", "r", "f", "c"))
    s["out"] = torch.empty(shape, dtype=torch.float32, device="cuda")
    a.out = s["out"].data_ptr()
    s["keep"], s["args"] = (t, d["u"]), a
    return s


# -------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    kind = case["kind"]
    if case["host"]:
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            if kind == "noise":
                return ccfj.fj_noise(s["u"], s["r"], s["c"], s["f"], fstride=case["fstride"],
                                     itype=case["itype"], func=case["func"])
            if kind == "earthquake":
                return ccfj.fj_earthquake(s["u"], s["r"], s["c"], s["f"], itype=case["itype"],
                                          func=case["func"])
            if kind == "batch":
                return np.stack(ccfj.fj_noise_batch(s["us"], s["rs"], s["c"], s["f"],
                                                    itype=case["itype"], func=case["func"]))
            return ccfj.cc_fj_noise(case["npts"], case["nsta"], case["nf"], case["fftlen"],
                                    s["pairs"], s["startend"], s["x"], s["r"], s["c"], s["f"],
                                    overlaprate=case["overlap"], fstride=case["fstride"],
                                    ifonebit=case["onebit"], ifspecwhittenning=case["whiten"],
                                    itype=case["itype"], func=case["func"])
    lib = _lib.load()
    call = {"noise": lib.ccfj_fj_v1, "batch": lib.ccfj_fj_batch_v1, "cc": lib.ccfj_cc_v1,
            "earthquake": lib.ccfj_fj_earthquake_v1, "mwfj": lib.ccfj_fj_earthquake_v1}[kind]
    _lib.check(call(ctypes.byref(s["args"]),
                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return s["out"]


# ------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs read once, results written once. Flops: every input
    value enters its column's sum (2 flops); real FFTs 2.5 n log2 n, products
    of cross-spectra 8 per pair, bin and window."""
    kind = case["kind"]
    if kind in ("cc", "cc_noise"):
        n, step = case["nsta"], int(case["fftlen"] * (1 - case["overlap"]))
        shifts = max(1, (case["npts"] - case["fftlen"]) // step)
        pairs = n * (n - 1) // 2
        fft = 2.5 * case["fftlen"] * math.log2(case["fftlen"]) * n * shifts
        flops = fft + 8.0 * pairs * case["nf"] * shifts
        if kind == "cc":
            return dict(bytes=4.0 * n * case["npts"] + 8.0 * pairs * case["nf"], flops=flops)
        return dict(bytes=4.0 * n * case["npts"] + 4.0 * case["nc"] * case["nf"],
                    flops=flops + 2.0 * pairs * case["nf"])
    cols = case["nf"] * case["nc"]
    if kind == "noise":
        pairs = case["nr"]
        return dict(bytes=8.0 * pairs * case["nf"] * case["fstride"] + 4.0 * cols,
                    flops=2.0 * pairs * case["nf"])
    if kind == "batch":
        lo, hi = case["nrmin"], case["nrmax"]
        pairs = case["nsets"] * (hi - lo) / math.log(hi / lo)
        return dict(bytes=8.0 * pairs * case["nf"] + 4.0 * cols * case["nsets"],
                    flops=2.0 * pairs * case["nf"])
    nwin = case.get("nwin", 1)
    fft = 2.5 * case["npts"] * math.log2(case["npts"]) * case["nr"] * nwin
    return dict(bytes=4.0 * case["nr"] * case["npts"] + 4.0 * cols * nwin,
                flops=fft + 4.0 * case["nr"] * case["nf"] * nwin)


# ------------------------------------------------------------------ exact
def _gpu64(x):
    return torch.from_numpy(_f32(x).astype(np.float64)).cuda()


def _quadrature(r, kmax, itype):
    """(position, left station, weight of the left and of the right station's
    value) of every quadrature point over the sorted distances r."""
    dev = r.device
    n = len(r)
    d = r[1:] - r[:-1]
    d0 = d.clamp(min=float(np.float32(0.1)))
    if itype == 0:
        w = torch.zeros_like(r)
        w[1:] += d0
        w[:-1] += d0
        return r, torch.arange(n, device=dev), 0.5 * w * r, torch.zeros_like(r)
    dense = bool((kmax * d).max() <= 0.5)
    x, w = np.polynomial.legendre.leggauss(5 if dense else 8)
    x, w = (torch.from_numpy(v).to(dev) for v in (x, w))
    m = torch.ones_like(d, dtype=torch.int64) if dense else \
        torch.ceil(kmax * d / 2.0).to(torch.int64).clamp(min=1)
    left = torch.repeat_interleave(torch.arange(n - 1, device=dev), m)
    first = torch.cumsum(m, 0) - m
    piece = torch.arange(len(left), device=dev) - first[left]
    h = (d / m)[left]
    lo = r[left] + piece * h
    p = lo[:, None] + 0.5 * h[:, None] * (1 + x[None])
    wt = 0.5 * h[:, None] * w[None] * p
    t = (p - r[left][:, None]) / d0[left][:, None]
    left = left[:, None].expand_as(p).reshape(-1)
    return p.reshape(-1), left, (wt * (1 - t)).reshape(-1), (wt * t).reshape(-1)


def _exact_transform(g0, r, c, f, itype, mode, g1=None):
    """g0, g1: [n, nr, nf] real spectra of n sets on the same sorted distances;
    mode J, J_MINUS_Y (g1 the second input), ABS_J, ABS_H (g1 the imaginary
    part). Unnormalised [n, nc, nf]."""
    nset, nr, nf = g0.shape
    out = torch.zeros((nset, len(c), nf), dtype=torch.float64, device="cuda")
    if nr < 2:
        return out
    for i in range(nf):
        k = 2 * math.pi * f[i] / c
        if float(f[i]) == 0.0 and itype == 1:
            out[:, :, i] = float("nan")
            continue
        p, left, wl, wr = _quadrature(r, float(k.max()), itype)
        right = (left + 1).clamp(max=nr - 1)

        def weights(g):
            return wl[:, None] * g[:, left, i].T + wr[:, None] * g[:, right, i].T

        a, b = weights(g0), weights(g1) if g1 is not None else None
        o = [torch.zeros((len(c), nset), dtype=torch.float64, device="cuda") for _ in range(2)]
        step = max(1, int(6e7 // len(p)))
        for q in range(0, len(c), step):
            x = k[q:q + step, None] * p[None]
            J = torch.special.bessel_j0(x)
            Y = torch.special.bessel_y0(x) if mode in ("J_MINUS_Y", "ABS_H") else None
            if mode == "J":
                o[0][q:q + step] = J @ a
            elif mode == "J_MINUS_Y":
                o[0][q:q + step] = J @ a - Y @ b
            elif mode == "ABS_J":
                o[0][q:q + step], o[1][q:q + step] = J @ a, J @ b
            else:
                o[0][q:q + step], o[1][q:q + step] = J @ a - Y @ b, J @ b + Y @ a
        v = torch.hypot(o[0], o[1]) if mode.startswith("ABS") else o[0]
        out[:, :, i] = v.T
    return out


def _normalised(o):
    return o / o.abs().amax(dim=-2, keepdim=True)


def _hilbert(g):
    """scipy.fftpack.hilbert of real rows."""
    n = g.shape[-1]
    s = torch.fft.fft(g, dim=-1)
    h = torch.zeros(n, dtype=torch.complex128, device=g.device)
    h[1:(n + 1) // 2], h[n // 2 + 1:] = 1j, -1j
    return torch.fft.ifft(s * h, dim=-1).real


def _exact_noise(u, r, c, f, case):
    idx = torch.from_numpy(np.argsort(r)).cuda()
    g = u[idx].real.double()
    st = case.get("fstride", 1)
    rs, c, f = _gpu64(np.sort(r)), _gpu64(c), _gpu64(f)
    if case["func"] == 0:
        o = _exact_transform(g[None, :, ::st], rs, c, f, case["itype"], "J")
    else:
        o = _exact_transform(g[None, :, ::st], rs, c, f, case["itype"], "J_MINUS_Y",
                             _hilbert(g)[None, :, ::st])
    return _normalised(o)[0]


def _taper(npts, Fs, l, r, taper):
    """One trace's window: sine ramps at both ends of samples [n1, n2)."""
    n1, n2 = max(0, int(math.floor(l * Fs))), min(npts, int(math.floor(r * Fs)))
    w = np.zeros(npts)
    w[n1:n2] = 1.0
    m = int(math.floor((n2 - n1) * (1 - taper) / 2))
    ramp = np.sin(np.pi / 2 * np.arange(m) / max(m, 1))
    w[n1:n1 + m] = ramp
    w[n2 - m:n2] = ramp[::-1]
    return torch.from_numpy(w).cuda()


def _exact_cross(d):
    case = d["case"]
    x = d["x"].double()
    if case["onebit"]:
        x = torch.sign(x)
    F, step, n = case["fftlen"], int(case["fftlen"] * (1 - case["overlap"])), case["nsta"]
    se = d["startend"].reshape(-1, 2).astype(np.int64)
    shifts = (case["npts"] - F) // step + 1
    num = torch.zeros((n, n, case["nf"]), dtype=torch.complex128, device="cuda")
    cnt = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for k in range(shifts):
        keep = torch.from_numpy(((k * step >= se[:, 0]) & (k * step + F < se[:, 1])).astype(np.float64)).cuda()
        X = torch.fft.rfft(x[:, k * step:k * step + F], dim=1)
        X = X[:, :case["nf"] * case["fstride"]:case["fstride"]]
        if case["whiten"]:
            X = X / X.abs().clamp(min=1e-8)
        X = X * keep[:, None]
        num += X.conj()[:, None] * X[None]
        cnt += keep[:, None] * keep[None]
    pr = d["pairs"].reshape(-1, 2)
    a, b = torch.from_numpy(pr[:, 0].astype(np.int64)).cuda(), torch.from_numpy(pr[:, 1].astype(np.int64)).cuda()
    c = cnt[a, b]
    return torch.where(c[:, None] > 0, num[a, b] / c[:, None].clamp(min=1), torch.zeros((), dtype=torch.complex128, device="cuda"))


def exact(case, seed):
    kind = case["kind"]
    # Bessel evaluations that the quadrature takes, about 8e9 a second
    if kind in ("noise", "batch"):
        pairs = case["nr"] if kind == "noise" else work(case)["flops"] / (2.0 * case["nf"])
        evals = case["nf"] * case["nc"] * pairs * (1 if case["itype"] == 0 else 8) * (1 + case["func"])
        if evals > 5e10 or case["nf"] * case.get("nsets", 1) > 8000:
            return None
    if kind in ("cc", "cc_noise") and case["nsta"] ** 2 * case["nf"] > 2e7:
        return None
    d = _inputs(case, seed)
    if kind == "noise":
        return _exact_noise(d["u"], d["r"], d["c"], d["f"], case)
    if kind == "batch":
        off = np.cumsum([0] + [len(r) for r in d["rs"]])
        return torch.stack([_exact_noise(d["u"][a:b], r, d["c"], d["f"], case)
                            for a, b, r in zip(off[:-1], off[1:], d["rs"])])
    if kind in ("earthquake", "mwfj"):
        idx = np.argsort(d["r"])
        u = d["u"].double()
        if kind == "mwfj":
            w = torch.stack([torch.stack([_taper(case["npts"], case["Fs"], d["winl"][i, j],
                                                 d["winr"][i, j], d["taper"])
                                          for j in range(case["nr"])]) for i in range(case["nwin"])])
            u = u[None] * w
        else:
            u = u[None]
        X = torch.fft.rfft(u, dim=-1)[:, torch.from_numpy(idx).cuda(), :case["nf"]]
        o = _exact_transform(X.real, _gpu64(d["r"][idx]), _gpu64(d["c"]), _gpu64(d["f"]),
                             case["itype"], "ABS_J" if case["func"] == 0 else "ABS_H", X.imag)
        o = _normalised(o)
        return o if kind == "mwfj" else o[0]
    X = _exact_cross(d)
    if kind == "cc":
        return X
    return _exact_noise(X, d["r"], d["c"], d["f"], dict(case, fstride=1))

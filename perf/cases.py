"""The work a user of this framework has it do, as timed cases.

Each case is one pass through the public entry points (``Context`` / ``Batch``
and the C ABI they sit on) at sizes from this repository's own benchmark,
tests and the decks of the Fortran drivers it serves:

* ``melt``   -- bulk SCF iterations, or one propagation on device buffers;
* ``cell``   -- free energy and its reverse-mode gradient (unit-cell work);
* ``scan``   -- a batch of melts advanced together (phase-diagram scan);
* ``film1``  -- a single one-line film;   ``films`` -- a batch of them;
* ``film3``  -- a three-dimensional film (Douglas ADI);
* ``brush``  -- a grafted homopolymer on a long line, adaptive contour.

Host buffers are page-locked, as the drivers' are after cudaHostRegister.  A
split-precision context carries its propagators in 32 bits (which line-solver
shape its tuner picked shows at that level already), so its results are taken
in 32 bits, as a program that asked for that precision keeps them; FP64
contexts return 64 bits.

``exact`` restates the same mathematics in plain 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import adscf_gb300 as A
from adscf_gb300 import _lib, mesh

# line lengths of bulk grids: products of 2, 3 and 5
SMOOTH = (15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96,
          100, 108, 120, 125, 128, 135, 144, 150, 160)


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the reference's CPU-size melt in its own precision and mixing depth, past the warm-up
        dict(name="melt_32_fp64", kind="melt", gx=32, gy=32, gz=32, ns=100, f=0.30, chi=25.0, box=4.0,
             prec="fp64", mix="anderson", hist=2, iters=6, arch="AB", call="scf"),
        # the bulk driver's own deck: a 2-D grid of one point in y, Landau-type lambda mixing
        dict(name="melt_64x1x300_fp64", kind="melt", gx=64, gy=1, gz=300, ns=100, f=0.50, chi=18.0, box=4.0,
             prec="fp64", mix="lambda", hist=2, iters=6, arch="AB", call="scf"),
        # an orthorhombic cell: three different mixed-radix line lengths
        dict(name="melt_60x72x100_split", kind="melt", gx=60, gy=72, gz=100, ns=120, f=0.35, chi=20.0, box=4.2,
             prec="split", mix="anderson", hist=4, iters=4, arch="AB", call="scf"),
        # the benchmark melt (128^3, 200 contour steps)
        dict(name="melt_128_split", kind="melt", gx=128, gy=128, gz=128, ns=200, f=0.40, chi=20.0, box=3.8,
             prec="split", mix="anderson", hist=10, iters=6, arch="AB", call="scf"),
        # the largest: a 256^3 triblock propagation of a program that keeps its fields on the GPU
        dict(name="melt_256_split", kind="melt", gx=256, gy=256, gz=256, ns=100, f=0.40, chi=20.0, box=7.6,
             prec="split", mix="simple", hist=2, iters=1, arch="ABA", call="propagate"),
        # cell stress and dF/dchi of one relaxation step
        dict(name="cell_64_fp64", kind="cell", gx=64, gy=64, gz=64, ns=100, f=0.30, chi=20.0, box=4.0),
        # a scan over compositions and boxes on uneven cubic grids
        dict(name="scan_64_split", kind="scan", count=64, lo=24, hi=64, ns_lo=100, ns_hi=200, prec="split",
             hist=10, iters=2),
        # the Film_1D driver's own grid (500 intervals) in its precision
        dict(name="film1_500_fp64", kind="film1", gz=500, ns=100, depth=8.0, prec="fp64", iters=8),
        # the benchmark's film batch
        dict(name="films_4096_split", kind="films", count=4096, gz_lo=64, gz_hi=192, ns_lo=100, ns_hi=300,
             prec="split", iters=4),
        # the benchmark's Film_3D
        dict(name="film3_64x64x64_split", kind="film3", gx=64, gy=64, gz=64, ns=150, depth=3.0, prec="split",
             iters=4),
        # the Film_3D driver's own grid in its precision
        dict(name="film3_20x35x100_fp64", kind="film3", gx=20, gy=35, gz=100, ns=100, depth=4.0, prec="fp64",
             iters=1),
        # the brush driver's own line (1000 intervals) on an adaptive contour
        dict(name="brush_1000_fp64", kind="brush", gz=1000, ns=1200, depth=10.0, prec="fp64", iters=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, lo, hi):
    v = _log(rng, lo, hi)
    return min((n for n in SMOOTH if lo <= n <= hi), key=lambda n: abs(math.log(n / v)))


def draw(rng):
    kind = rng.choice(["melt"] * 5 + ["cell", "scan", "film1", "films", "film3", "film3", "brush"])
    prec = rng.choice(["fp64", "split"])
    if kind == "melt":
        shape = rng.choice(["cube", "cube", "box", "box", "plane"])
        gx = _smooth(rng, 15, 160)
        gy, gz = gx, gx
        if shape == "box":
            gy, gz = _smooth(rng, 15, 160), _smooth(rng, 15, 160)
        elif shape == "plane":
            gy, gz = 1, 2 * _smooth(rng, 15, 160)
        steps = int((1.0e8 if prec == "fp64" else 4.0e8) / (gx * gy * gz))   # contour steps of the whole pass
        ns = min(_log(rng, 40, 200), max(30, steps))
        call = rng.choice(["scf", "scf", "propagate"])
        mix = rng.choice(["anderson", "simple"]) if prec == "split" else rng.choice(["anderson", "lambda"])
        hist = rng.choice([2, 4, 10])
        # a few iterations: the fixed-point map amplifies rounding, the more so past Anderson's warm-up
        most = min(4, hist) if prec == "split" else hist + 2 if mix == "anderson" and hist < 10 else 8
        iters = 1 if call == "propagate" else max(1, min(most, steps // ns))
        return dict(kind=kind, gx=gx, gy=gy, gz=gz, ns=ns, f=round(rng.uniform(0.25, 0.5), 2),
                    chi=round(rng.uniform(15.0, 25.0), 1), box=round(rng.uniform(3.5, 5.0), 2), prec=prec, mix=mix,
                    hist=hist, iters=iters, arch=rng.choice(["AB", "AB", "AB", "ABA", "A"]),
                    call=call)
    if kind == "cell":
        gx, gy, gz = (_smooth(rng, 16, 64) for _ in range(3)) if rng.random() < 0.5 else (_smooth(rng, 16, 80),) * 3
        return dict(kind=kind, gx=gx, gy=gy, gz=gz, ns=_log(rng, 40, 120), f=round(rng.uniform(0.25, 0.5), 2),
                    chi=round(rng.uniform(15.0, 25.0), 1), box=round(rng.uniform(3.5, 5.0), 2))
    if kind == "scan":
        n = _log(rng, 8, 64) if prec == "split" else _log(rng, 4, 12)
        return dict(kind=kind, count=n, lo=24, hi=64 if prec == "split" else 40, ns_lo=60, ns_hi=_log(rng, 61, 200),
                    prec=prec, hist=rng.choice([2, 10]), iters=1)
    if kind == "film1":
        return dict(kind=kind, gz=_log(rng, 48, 600), ns=_log(rng, 50, 300), depth=round(rng.uniform(2.0, 10.0), 2),
                    prec=prec, iters=rng.randint(2, 8))
    if kind == "films":
        lo = _log(rng, 32, 128)
        return dict(kind=kind, count=_log(rng, 32, 2048), gz_lo=lo, gz_hi=_log(rng, lo, 250), ns_lo=100,
                    ns_hi=_log(rng, 100, 300), prec=prec, iters=1 if prec == "fp64" else 3)
    if kind == "film3":
        small = prec == "fp64"
        return dict(kind=kind, gx=_log(rng, 12, 40 if small else 96), gy=_log(rng, 12, 40 if small else 96),
                    gz=_log(rng, 24, 100), ns=_log(rng, 50, 100 if small else 150),
                    depth=round(rng.uniform(2.0, 4.0), 2), prec=prec, iters=1 if small else rng.randint(1, 3))
    return dict(kind="brush", gz=_log(rng, 100, 1000), ns=_log(rng, 300, 3000),
                depth=round(rng.uniform(5.0, 12.0), 2), prec=prec, iters=1)


# --------------------------------------------------------------------------
# parameters and inputs
# --------------------------------------------------------------------------
def _prec(case):
    return A.SPLIT if case.get("prec") == "split" else A.FP64


def _segments(case):
    """(contour steps, type) of each block."""
    ns, f = case["ns"], case["f"]
    na = max(1, min(ns - 1, round(f * ns)))
    if case.get("arch", "AB") == "AB":
        return [(na, 0), (ns - na, 1)]
    if case["arch"] == "ABA":
        a1 = max(1, na // 2)
        return [(a1, 0), (ns - na, 1), (na - a1 if na > a1 else 1, 0)]
    return [(ns, 0)]


def _melt_params(case):
    seg = _segments(case)
    n = sum(s for s, _ in seg)
    ds = 1.0 / n
    g = (case["gx"], case["gy"], case["gz"])
    big = max(g)
    size = tuple(case["box"] * (0.4 + 0.6 * v / big) for v in g)
    kw = dict(grid=g, size=size, ds=ds, kappa=25.0, chi=case["chi"], precision=_prec(case),
              mixing_type={"anderson": A.MIX_ANDERSON, "lambda": A.MIX_LAMBDA, "simple": A.MIX_SIMPLE}[case.get("mix", "simple")],
              mixing_dim=case.get("hist", 2), lam=0.1, lam_warm=0.1, warm_iters=case.get("hist", 2))
    if case.get("arch", "AB") == "AB":
        kw["block_length"] = (seg[0][0] * ds, seg[1][0] * ds)
    else:
        kw["blocks"] = [s * ds for s, _ in seg]
        kw["block_types"] = [t for _, t in seg]
    return kw


def _melt_field(shape, f, chi, seed, gen=None):
    """A modulated start field with per-point noise, [2][z][y][x] on the GPU."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = gen or torch.Generator(device=dev).manual_seed(seed)
    gz, gy, gx = shape
    z, y, x = (torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n) for n in shape)
    ph = torch.rand(3, generator=gen, device=dev, dtype=torch.float64) * (2 * math.pi)
    s = (torch.cos(x + ph[0])[None, None, :] + torch.cos(2 * z + ph[2])[:, None, None]
         + (torch.cos(y + ph[1])[None, :, None] if gy > 1 else 0.0)) / 3.0
    a = 0.5 * chi * (0.6 - f)
    w = torch.stack([a * s, -a * s])
    w += 0.1 * torch.randn(w.shape, generator=gen, device=dev, dtype=torch.float64)
    return w


def _scan_cases(case):
    r = np.random.default_rng(5)                  # the scan's parameters are the case's, its fields the seed's
    sizes = [n for n in (24, 32, 40, 48, 64) if case["lo"] <= n <= case["hi"]]
    out = []
    for _ in range(case["count"]):
        n = int(r.choice(sizes))
        out.append(dict(gx=n, gy=n, gz=n, ns=int(r.integers(case["ns_lo"], case["ns_hi"] + 1)),
                        f=float(r.uniform(0.25, 0.45)), chi=float(r.uniform(15.0, 25.0)),
                        box=float(r.uniform(3.0, 5.0)), prec=case["prec"], mix="anderson", hist=case["hist"]))
    return out


def _film_mesh(gz, depth):
    return mesh.tanh_mesh(gz, depth, 2.0)


def _film_params(case, r=None):
    """One film: a diblock between walls with a surface potential on A."""
    gz, depth, ns = case["gz"], case["depth"], case["ns"]
    ns += ns % 2
    h = 0.5 if r is None else float(r.uniform(-1.0, 1.0))
    d3 = case["kind"] == "film3"
    if case["kind"] == "film1":                   # the Film_1D driver's uniform mesh and steps
        dz, zr = mesh.generate_mesh(0, gz, depth)
        dss = mesh.contour_steps(ns, ds_scheme=0)
    else:
        dz, zr = _film_mesh(gz, depth)
        dss = mesh.contour_steps(ns, ds_scheme=1)
    gx, gy = (case["gx"], case["gy"]) if d3 else (1, 1)
    lx = 6.0 * gx / max(gx, gy) if d3 else 1.0
    ly = 6.0 * gy / max(gx, gy) if d3 else 1.0
    fixed = case.get("prec") == "split"           # lambda mixing divides FP32-level differences at its start
    return dict(geometry=A.FILM_3D if d3 else A.FILM_1D, grid=(gx, gy, gz), size=(lx, ly, depth), dz=dz, dss=dss,
                n_a=ns // 2, block_length=(0.5, 0.5), chi=20.0, kappa=25.0,
                ext_potential=mesh.wall_potential(zr, depth, 0.4, (h, 0.0)), int_scheme=1, int_span=0 if d3 else 1,
                ensemble=2, mu=2.25 if d3 else 2.55, precision=_prec(case),
                mixing_type=A.MIX_SIMPLE if fixed else A.MIX_LAMBDA, lam=0.05 if fixed else 0.2)


def _films_params(case):
    r = np.random.default_rng(2)
    out = []
    for _ in range(case["count"]):
        out.append(_film_params(dict(kind="films", gz=int(r.integers(case["gz_lo"], case["gz_hi"] + 1)),
                                     depth=float(r.uniform(2.0, 8.0)), prec=case["prec"],
                                     ns=int(r.integers(case["ns_lo"], case["ns_hi"] + 1))), r))
    return out


def _film_field(kw, rng):
    gx, gy, gz = kw["grid"]
    w = rng.normal(0.0, 0.05, (2, gz + 1, gy, gx))
    if gx > 1:
        x = 2 * np.pi * np.arange(gx) / gx
        y = 2 * np.pi * np.arange(gy) / gy
        s = 0.5 * np.cos(2 * x)[None, :] * np.cos(y + rng.uniform(0, 6.28))[:, None]
        w[0] += s
        w[1] -= s
    w[:, 0] = w[:, -1] = 0.0
    return w


def _brush_params(case):
    gz, depth = case["gz"], case["depth"]
    i = np.arange(gz + 1)
    zr = depth * (0.35 * i / gz + 0.65 * (i / gz) ** 2)      # finer near the grafting wall
    dz = np.zeros(gz + 1)
    dz[1:] = np.diff(zr)
    graft = np.exp(-0.5 * ((zr - 0.3) / 0.1) ** 2)
    graft[0] = graft[-1] = 0.0
    graft /= np.sum(graft[1:] * dz[1:])
    ext = np.zeros(gz + 1)
    return dict(geometry=A.BRUSH, grid=(1, 1, gz), size=(1.0, 1.0, depth), dz=dz,
                dss=mesh.contour_steps(case["ns"], ds_scheme=1), block_length=(1.0, 0.0), rho=0.4, ww=1.5, graft=graft,
                ext_potential=ext, int_scheme=1, int_span=1, ensemble=1, precision=_prec(case),
                mixing_type=A.MIX_SIMPLE, lam=0.1), zr


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _inputs(case, seed):
    """(parameters, start fields): a dict and a tensor, or lists of them."""
    k = case["kind"]
    if k in ("melt", "cell"):
        return _melt_params(case), _melt_field((case["gz"], case["gy"], case["gx"]), case["f"], case["chi"], seed)
    if k == "scan":
        cs = _scan_cases(case)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        gen = torch.Generator(device=dev).manual_seed(seed)
        return [_melt_params(c) for c in cs], [_melt_field((c["gz"], c["gy"], c["gx"]), c["f"], c["chi"], seed, gen) for c in cs]
    rng = np.random.default_rng(seed)
    if k == "films":
        kws = _films_params(case)
        return kws, [torch.from_numpy(_film_field(kw, rng)) for kw in kws]
    if k == "brush":
        kw, zr = _brush_params(case)
        w = 1.2 * np.exp(-zr / 3.0) + rng.normal(0.0, 0.02, zr.shape)
        w[0] = w[-1] = 0.0
        return kw, torch.from_numpy(w)
    kw = _film_params(case)
    return kw, torch.from_numpy(_film_field(kw, rng))


def prepare(case, seed):
    params, field = _inputs(case, seed)
    st = {"case": case}
    if case["kind"] in ("scan", "films"):
        b = st["batch"] = A.Batch([dict(kw, geometry=kw.get("geometry", A.BULK)) for kw in params])
        st["w"] = _pinned(b.offsets[-1])
        st["w"].copy_(torch.cat([f.reshape(-1).cpu() for f in field]))
        n = b.offsets[-1]
    else:
        kw = dict(params)
        c = st["ctx"] = A.Context(kw.pop("geometry", A.BULK), **kw)
        if case["kind"] == "cell" or case.get("call") == "propagate":
            st["w"] = field.contiguous()
            st["d"] = torch.empty_like(st["w"])
            return st
        n = field.numel()
        assert n == c.ntypes * c.npts
        st["w"] = _pinned(n)
        st["w"].copy_(field.reshape(-1))
    st["x"], st["d"] = _pinned(n), _pinned(n)
    if case["prec"] == "split":
        st["x32"], st["d32"] = torch.empty(n), torch.empty(n)
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _num(case, *v):
    t = np.array(v)
    return t.astype(np.float32) if case.get("prec") == "split" else t


def _fields(st, x, d):
    if "x32" in st:
        return st["x32"].copy_(x), st["d32"].copy_(d)
    return x, d


def run(st):
    case = st["case"]
    if case["kind"] in ("scan", "films"):
        b = st["batch"]
        b._ck(b.lib.adscf_batch_set_fields(b.h, _lib.dptr(st["w"].numpy())))
        res = b.scf_run(case["iters"])
        b._ck(b.lib.adscf_batch_get_fields(b.h, _lib.dptr(st["x"].numpy())))
        b._ck(b.lib.adscf_batch_get_densities(b.h, _lib.dptr(st["d"].numpy())))
        x, d = _fields(st, st["x"], st["d"])
        return {"field": x, "density": d, "Q": _num(case, *[r.Qsum for r in res])}
    c = st["ctx"]
    if case["kind"] == "cell":
        F = _lib.C.c_double()
        c._ck(c.lib.adscf_forward_dev(c.h, st["w"].data_ptr(), _lib.C.byref(F)))
        return {"F": F.value, "grad": c.backward()}
    if case.get("call") == "propagate":
        r = _lib.ChainResult()
        c._ck(c.lib.adscf_propagate_diblock_dev(c.h, st["w"].data_ptr(), st["d"].data_ptr(), _lib.C.byref(r)))
        d = st["d"].float() if case["prec"] == "split" else st["d"]
        return {"density": d, "Q": _num(case, r.Qsum)}
    c.set_field(st["w"].numpy())
    r = c.scf_run(case["iters"])
    c._ck(c.lib.adscf_get_field(c.h, _lib.dptr(st["x"].numpy())))
    c._ck(c.lib.adscf_get_density(c.h, _lib.dptr(st["d"].numpy())))
    x, d = _fields(st, st["x"], st["d"])
    return {"field": x, "density": d, "Q": _num(case, r.Qsum)}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _melt_work(case, iters):
    """(bytes, operations): field in, field and density out; per contour step
    of both chains one complex 3-D transform pair, the Boltzmann products, the
    k-space product and the contour products."""
    n = case["gx"] * case["gy"] * case["gz"]
    ns = sum(s for s, _ in _segments(case))
    return 48.0 * n, iters * n * ns * (10.0 * math.log2(n) + 20.0)


def work(case):
    k = case["kind"]
    if k == "melt":
        by, fl = _melt_work(case, case["iters"])
    elif k == "cell":                             # forward chains, their adjoints, and the stress products
        by, fl = _melt_work(case, 1)
        by, fl = by / 3.0, 2.2 * fl
    elif k == "scan":
        got = [_melt_work(c, case["iters"]) for c in _scan_cases(case)]
        by, fl = (sum(v) for v in zip(*got))
    else:
        if k == "films":
            sizes = [(2 * (kw["grid"][2] + 1), len(kw["dss"]) - 1) for kw in _films_params(case)]
        else:
            types = 1 if k == "brush" else 2
            sizes = [(types * case.get("gx", 1) * case.get("gy", 1) * (case["gz"] + 1), case["ns"])]
        sweep = 60.0 if k == "film3" else 20.0    # per point, step and chain: right-hand side and line solves
        by = sum(24.0 * n for n, s in sizes)
        fl = sum(n * s * (sweep + 4.0) for n, s in sizes) * case["iters"]
    return {"bytes": by, "flops": fl}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _k2(n, dev):
    m = torch.arange(n, device=dev, dtype=torch.float64)
    m = torch.where(m > n // 2, m - n, m)
    return (2 * math.pi * m) ** 2


def _melt_propagate(w, kw, seg, length=None):
    """(Q, distribution per type) of a linear block sequence."""
    gx, gy, gz = kw["grid"]
    dev = w.device
    lx, ly, lz = length if length is not None else kw["size"]
    kx = (2 * math.pi * torch.arange(gx // 2 + 1, device=dev, dtype=torch.float64)) ** 2
    ky = _k2(gy, dev)
    kz = _k2(gz, dev)
    ds = kw["ds"]
    g = torch.exp(-ds * (kz[:, None, None] / lz ** 2 + ky[None, :, None] / ly ** 2 + kx[None, None, :] / lx ** 2))
    e = torch.exp(-0.5 * ds * w)
    types = [t for n, t in seg for _ in range(n)]
    ns = len(types)
    q = torch.ones((2,) + w.shape[1:], dtype=torch.float64, device=dev)
    node = [q]
    for s in range(ns):
        ee = torch.stack([e[types[s]], e[types[ns - 1 - s]]])
        q = ee * torch.fft.irfftn(g * torch.fft.rfftn(ee * q, dim=(1, 2, 3)), s=(gz, gy, gx), dim=(1, 2, 3))
        node.append(q)
    dvol = lx * ly * lz / (gx * gy * gz)
    dist = [torch.zeros_like(w[0]), torch.zeros_like(w[0])]
    s0 = 0
    for n, t in seg:
        for s in range(s0, s0 + n + 1):
            dist[t] = dist[t] + (0.5 if s in (s0, s0 + n) else 1.0) * ds * node[s][0] * node[ns - s][1]
        s0 += n
    return dvol * node[ns][0].sum(), torch.stack(dist)


class _Mixer:
    def __init__(self, kw):
        self.kind, self.m, self.lam = kw["mixing_type"], kw.get("mixing_dim", 2), kw["lam"]
        self.warm = max(kw.get("warm_iters", 0), self.m)
        self.lam0 = kw.get("lam_warm", 1.0e-3)
        self.x, self.r = [], []

    def __call__(self, x, r, it):
        self.x.insert(0, x)
        self.r.insert(0, r)
        del self.x[self.m + 1:], self.r[self.m + 1:]
        if self.kind == A.MIX_SIMPLE:
            return x + self.lam * r
        if self.kind == A.MIX_LAMBDA:
            lam = 1.0e-5
            if it > 1:
                nom = float(((r - self.r[1]) ** 2).sum())
                if nom > 1.0e-50:
                    lam = min(max(math.sqrt(float(((x - self.x[1]) ** 2).sum()) / nom), 1.0e-5), self.lam)
            return x + lam * r
        if it <= self.warm:
            return x + self.lam0 * r
        d = torch.stack([(r - v).reshape(-1) for v in self.r[1:]])
        a = torch.linalg.solve((d @ d.T).cpu(), (d @ r.reshape(-1)).cpu()).to(x.device)
        y = torch.stack([(x - v).reshape(-1) for v in self.x[1:]])
        return x - (a @ y).reshape(x.shape) + self.lam * (r - (a @ d).reshape(x.shape))


def _melt_exact(case, kw, w, iters):
    seg = _segments(case)
    vol = kw["size"][0] * kw["size"][1] * kw["size"][2]
    mix = _Mixer(kw)
    for it in range(1, iters + 1):
        q, dist = _melt_propagate(w, kw, seg)
        phi = vol * dist / q
        press = kw["kappa"] * (phi[0] + phi[1] - 1.0)
        r = torch.stack([press + kw["chi"] * phi[1], press + kw["chi"] * phi[0]]) - w
        w = mix(w, r, it)
    return w, phi, float(q)


def _cell_exact(case, kw, w):
    seg = _segments(case)
    length = torch.tensor(kw["size"], dtype=torch.float64, device=w.device, requires_grad=True)
    chi = torch.tensor(kw["chi"], dtype=torch.float64, device=w.device, requires_grad=True)
    q, dist = _melt_propagate(w, kw, seg, length)
    vol = length[0] * length[1] * length[2]
    phi = vol * dist / q
    dvol = vol / w[0].numel()
    tot = phi[0] + phi[1] - 1.0
    F = (torch.log(vol / q) - 1.0) + (dvol * (0.5 * kw["kappa"] * (tot * tot).sum() + chi * (phi[0] * phi[1]).sum()
                                              - (phi * w).sum())) / vol
    F.backward()
    return float(F.detach()), np.array(length.grad.tolist() + [float(chi.grad)])


def _thomas(a, d, c, r):
    """Tridiagonal solves along the last axis (row j: a_j, d_j, c_j)."""
    n = r.shape[-1]
    a, d, c, r = (t.expand(r.shape).movedim(-1, 0) for t in (a, d, c, r))
    cp, u = [c[0] / d[0]], [r[0] / d[0]]
    for j in range(1, n):
        inv = 1.0 / (d[j] - a[j] * cp[-1])
        cp.append(c[j] * inv)
        u.append((r[j] - a[j] * u[-1]) * inv)
    for j in range(n - 2, -1, -1):
        u[j] = u[j] - cp[j] * u[j + 1]
    return torch.stack(u, dim=-1)


def _z_factors(dz):
    """al, be, ga of a mesh, zero on the walls."""
    h1, h2 = dz[1:-1], dz[2:]
    al, ga = np.zeros_like(dz), np.zeros_like(dz)
    al[1:-1] = 1.0 / h1 / (h1 + h2)
    ga[1:-1] = 1.0 / h2 / (h1 + h2)
    return al, al + ga, ga


def _z_weights(dz, full):
    w = np.zeros_like(dz)
    hi = len(dz) if full else len(dz) - 1
    for i in range(1, hi):
        w[i - 1] += 0.5 * dz[i]
        w[i] += 0.5 * dz[i]
    return w


def _line_chains(kw, w, steps, q0):
    """Nodes of one Crank-Nicolson chain on a single line: the step operators
    of one field share eigenvectors, so every step is diagonal there.
    steps: (ds, type) per step; w [types][gz+1]; q0 [gz+1]."""
    al, be, ga = _z_factors(kw["dz"])
    h = np.sqrt(kw["dz"][1:-1] + kw["dz"][2:])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    V, lam = {}, {}
    for t in sorted({t for _, t in steps}):
        off = -ga[1:-2] * h[:-1] / h[1:]
        m = np.diag(be[1:-1] + 0.5 * w[t][1:-1]) + np.diag(off, 1) + np.diag(off, -1)
        lam[t], V[t] = torch.linalg.eigh(torch.from_numpy(m).to(dev))
    hh = torch.from_numpy(h).to(dev)
    nodes = [torch.from_numpy(q0).to(dev)]
    src = torch.zeros(len(h), dtype=torch.float64, device=dev)
    src[0] += al[1] * q0[0]
    src[-1] += ga[-2] * q0[-1]
    c, cur, run_, out = nodes[0][1:-1] * hh, None, [], []
    for k, (ds, t) in enumerate(steps):
        if t != cur:
            if cur is not None:
                c = V[cur] @ c
                out.append((cur, torch.stack(run_)))
                run_ = []
            c, cur = V[t].T @ c, t
        num = (1.0 - ds * lam[t]) * c
        if k == 0:
            num = num + ds * (V[t].T @ (src * hh))
        c = num / (1.0 + ds * lam[t])
        run_.append(c)
    out.append((cur, torch.stack(run_)))
    inner = torch.cat([b @ V[t].T for t, b in out]) / hh
    q = torch.zeros((len(steps) + 1, len(q0)), dtype=torch.float64, device=dev)
    q[0] = nodes[0]
    q[1:, 1:-1] = inner
    return q


def _film_nodes(kws, W, dev):
    """Both chains' nodes of films that may differ in length and steps.
    W [films][2][P] (or [films][2][P][gy][gx] for one three-dimensional film)."""
    nf, P = W.shape[0], W.shape[2]
    ns = [len(kw["dss"]) - 1 for kw in kws]
    fac = np.zeros((3, nf, P))
    DS, TY = np.zeros((2, nf, max(ns) + 1)), np.zeros((2, nf, max(ns) + 1), dtype=np.int64)
    inner = np.zeros((nf, P))
    for i, kw in enumerate(kws):
        n, na = ns[i], kw["n_a"]
        for v, t in zip(_z_factors(kw["dz"]), fac):
            t[i, : len(v)] = v
        inner[i, 1: len(kw["dz"]) - 1] = 1.0
        s = np.arange(1, n + 1)
        DS[0, i, 1: n + 1], DS[1, i, 1: n + 1] = kw["dss"][s], kw["dss"][n + 1 - s]
        TY[0, i, 1: n + 1], TY[1, i, 1: n + 1] = s > na, s <= n - na
    al, be, ga, inner = (torch.from_numpy(v).to(dev) for v in (*fac, inner))
    d3 = W.dim() == 5
    tail = (1, 1) if d3 else ()
    al, be, ga, inner = (v.reshape((1, nf, P) + tail) for v in (al, be, ga, inner))
    DS, TY = torch.from_numpy(DS).to(dev), torch.from_numpy(TY).to(dev)
    q = torch.ones((2, nf) + tuple(W.shape[2:]), dtype=torch.float64, device=dev)
    real = torch.zeros((nf, P), dtype=torch.float64, device=dev)
    for i, kw in enumerate(kws):
        real[i, : len(kw["dz"])] = 1.0
    q = q * real.reshape((1, nf, P) + tail)
    nodes = [q]
    zl = (lambda t: t.movedim(2, -1)) if d3 else (lambda t: t)
    zb = (lambda t: t.movedim(-1, 2)) if d3 else (lambda t: t)
    at = torch.arange(nf, device=dev)
    for s in range(1, max(ns) + 1):
        ds = DS[:, :, s].reshape((2, nf, 1) + tail)
        w = torch.stack([W[at, TY[c, :, s]] for c in range(2)])
        dn, up = torch.zeros_like(q), torch.zeros_like(q)
        dn[:, :, 1:], up[:, :, :-1] = q[:, :, :-1], q[:, :, 1:]
        a, b, c, hw = -ds * al, ds * be, -ds * ga, 0.5 * ds * w * inner
        lz = a * dn + b * q + c * up
        if not d3:
            rhs = inner * (q - lz - hw * q)
        else:
            kw = kws[0]
            dx, dy = kw["size"][0] / kw["grid"][0], kw["size"][1] / kw["grid"][1]
            rx, ry = DS[:, 0, s] / dx / dx, DS[:, 0, s] / dy / dy      # per chain
            sh = (2, 1, 1, 1, 1)
            lx = rx.reshape(sh) * (q - 0.5 * (torch.roll(q, 1, 4) + torch.roll(q, -1, 4)))
            ly = ry.reshape(sh) * (q - 0.5 * (torch.roll(q, 1, 3) + torch.roll(q, -1, 3)))
            u = q - lx - 2.0 * ly - 2.0 * lz - 2.0 * hw * q

            def per(n, r):
                m = torch.zeros((2, n, n), dtype=torch.float64, device=dev)
                i = torch.arange(n, device=dev)
                m[:, i, i] += (1.0 + r)[:, None]
                m[:, i, (i + 1) % n] += -0.5 * r[:, None]
                m[:, i, (i - 1) % n] += -0.5 * r[:, None]
                return torch.linalg.inv(m)
            u = torch.einsum("cij,cfzyj->cfzyi", per(q.shape[4], rx), u)
            u = torch.einsum("cij,cfzjx->cfzix", per(q.shape[3], ry), u + ly)
            rhs = inner * (u + lz + hw * q)
        new = zb(_thomas(zl(a.expand(q.shape)), zl(1.0 + (b + hw) * inner), zl(c.expand(q.shape)), zl(rhs)))
        live = (DS[:, :, s] > 0).reshape((2, nf, 1) + tail)
        q = torch.where(live, new, q)
        nodes.append(q)
    return nodes, ns


def _film_exact(kws, fields, iters):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d3 = kws[0]["geometry"] == A.FILM_3D
    P = max(len(kw["dz"]) for kw in kws)
    nf = len(kws)
    shape = (nf, 2, P) + (tuple(fields[0].shape[2:]) if d3 else ())
    W = torch.zeros(shape, dtype=torch.float64, device=dev)
    ext, wz = torch.zeros((nf, 2, P), dtype=torch.float64, device=dev), torch.zeros((nf, P), dtype=torch.float64, device=dev)
    inner = torch.zeros((nf, P), dtype=torch.float64, device=dev)
    for i, (kw, f) in enumerate(zip(kws, fields)):
        n = len(kw["dz"])
        W[i, :, :n] = (f if d3 else f.reshape(2, n)).to(dev)
        ext[i, :, :n] = torch.from_numpy(kw["ext_potential"]).to(dev)
        area = kw["size"][0] / kw["grid"][0] * kw["size"][1] / kw["grid"][1]
        wz[i, :n] = torch.from_numpy(_z_weights(kw["dz"], d3)).to(dev) * area
        inner[i, 1: n - 1] = 1.0
    tail = (1, 1) if d3 else ()
    ext, inn = ext.reshape((nf, 2, P) + tail), inner.reshape((nf, 1, P) + tail)
    mixers = [_Mixer(kw) for kw in kws]
    line = nf == 1 and not d3
    for it in range(1, iters + 1):
        if line:
            kw = kws[0]
            n, na = len(kw["dss"]) - 1, kw["n_a"]
            w = W[0].cpu().numpy()
            one = np.ones(P)
            qf = _line_chains(kw, w, [(kw["dss"][s], int(s > na)) for s in range(1, n + 1)], one)
            qb = _line_chains(kw, w, [(kw["dss"][n + 1 - s], int(s <= n - na)) for s in range(1, n + 1)], one)
            nodes, ns = [torch.stack([qf[s][None], qb[s][None]]) for s in range(n + 1)], [n]
        else:
            nodes, ns = _film_nodes(kws, W, dev)
        dist = torch.zeros_like(W)
        Q = []
        back = torch.stack([v[1] for v in nodes]) if not d3 else None
        at = torch.arange(nf, device=dev)
        nst = torch.tensor(ns, device=dev)
        wt = torch.zeros((2, nf, max(ns) + 1), dtype=torch.float64)
        for i, kw in enumerate(kws):
            dss = torch.from_numpy(kw["dss"])
            for t, (lo, hi) in enumerate(((0, kw["n_a"]), (kw["n_a"], ns[i]))):
                wt[t, i, lo:hi] += 0.5 * dss[lo + 1: hi + 1]
                wt[t, i, lo + 1: hi + 1] += 0.5 * dss[lo + 1: hi + 1]
        wt = wt.to(dev)
        for s in range(max(ns) + 1):
            other = nodes[ns[0] - s][1] if d3 else back[(nst - s).clamp(min=0), at]
            prod = nodes[s][0] * other
            for t in range(2):
                dist[:, t] += wt[t, :, s].reshape((nf, 1) + tail) * prod
        last = torch.stack([nodes[ns[i]][0][i] for i in range(nf)])
        Q = (wz.reshape((nf, P) + tail) * last).flatten(1).sum(1)
        mu = torch.tensor([kw["mu"] for kw in kws], dtype=torch.float64, device=dev)
        phi = torch.exp(mu).reshape((nf, 1, 1) + tail) * dist
        kap, chi = kws[0]["kappa"], kws[0]["chi"]
        press = kap * (phi[:, 0] + phi[:, 1] - 1.0)
        R = torch.stack([press + chi * phi[:, 1], press + chi * phi[:, 0]], dim=1) + ext - W
        R = R * inn
        if kws[0]["mixing_type"] == A.MIX_SIMPLE:
            W = W + kws[0]["lam"] * R
        else:
            W = torch.stack([mixers[i](W[i] * inn[i], R[i], it) + W[i] * (1.0 - inn[i]) for i in range(nf)])
    cut = lambda T: torch.cat([T[i][:, : len(kw["dz"])].reshape(-1) for i, kw in enumerate(kws)])  # noqa: E731
    return cut(W), cut(phi), Q.cpu().numpy()


def _brush_exact(kw, w):
    dss, n = kw["dss"], len(kw["dss"]) - 1
    W = w.numpy()[None]
    qf = _line_chains(kw, W, [(dss[s], 0) for s in range(1, n + 1)], np.ones(len(kw["dz"])))
    qb = _line_chains(kw, W, [(dss[n + 1 - s], 0) for s in range(1, n + 1)], kw["graft"])
    wz = torch.from_numpy(_z_weights(kw["dz"], False)).to(qf.device)
    Q = float((wz * qb[0] * qf[n]).sum())
    c = torch.zeros(n + 1, dtype=torch.float64)
    c[0] = 0.5 * dss[0]
    c[1:n] = 0.5 * torch.from_numpy(dss[1:n] + dss[2:])
    c[n] = 0.5 * dss[n]
    dist = (c.to(qf.device)[:, None] * qf * qb.flip(0)).sum(0)
    phi = kw["rho"] * kw["size"][2] * dist / Q
    phi[0] = 0.0
    r = (kw["ww"] * phi).cpu() - w
    r[0] = r[-1] = 0.0
    return w + kw["lam"] * r, phi, Q


def exact(case, seed):
    params, field = _inputs(case, seed)
    k = case["kind"]
    out = None
    if k == "cell":
        F, g = _cell_exact(case, params, field)
        return {"F": F, "grad": g}
    if k == "melt":
        w, phi, q = _melt_exact(case, params, field, case["iters"])
        if case["call"] == "propagate":
            return {"density": phi, "Q": np.array([q])}
        out = (w.reshape(-1), phi.reshape(-1), np.array([q]))
    elif k == "scan":
        got = [_melt_exact(c, kw, f, case["iters"]) for c, kw, f in zip(_scan_cases(case), params, field)]
        out = (torch.cat([g[0].reshape(-1) for g in got]), torch.cat([g[1].reshape(-1) for g in got]),
               np.array([g[2] for g in got]))
    elif k == "brush":
        w, phi, q = _brush_exact(params, field)
        out = (w, phi, np.array([q]))
    elif k == "films":
        out = _film_exact(params, field, case["iters"])
    else:
        w, phi, q = _film_exact([params], [field], case["iters"])
        out = (w, phi, q)
    return {"field": out[0], "density": out[1], "Q": out[2]}

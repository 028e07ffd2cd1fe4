"""The work that users of this framework have it do, as measurable cases.

A case is one pass through the public Python API (operators, the device
solver, the request server).  Kinds:

  ts        SENSE<TimeSegmentation<Gnufft>> on device tensors, `dir` one of
            fwd, adj or pair (both), 2-D (nz = 1) or 3-D; L = 1 is SENSE<Gnufft>
  pcts      pcSenseTimeSeg: multishot, one shot phase map per shot, 3-D
  pcg       solve_pwls_pcg_device over one of these operators
  gdft      SENSE<Gdft>, or SENSE<GdftR2> with r2 = True
  pcdft     pcSENSE: one Gdft per shot
  serve     the request server on host arrays: submit all requests, wait for all

Sizes follow the configurations of powergrid_b200/synthetic.py, of the tests
and of bench.py's serving stream (64-256 in-plane, 1-32 slices or 3-D,
4-32 coils, 8k-200k samples, L = 4-12).

The 64-bit values (`exact`) evaluate the operators' definition: the window
bounds and the table entry that a tap reads are float arithmetic by definition
(PowerGrid/gridding.cpp:62-84, griddingSupport.cpp:33-76), everything after
them is evaluated in double.
"""
import math

import numpy as np
import torch

import powergrid_b200 as pg
from powergrid_b200 import serve as pgserve

DEV = "cuda"


# ---- the cases ----------------------------------------------------------------
def listed():
    return [
        # the smallest reconstruction: one coil, no field map, a low-resolution
        # calibration or navigator image (launches and latency count)
        dict(name="pcg_gnufft_64", kind="pcg", op="ts", n=64, nz=1, nc=1, L=1, inter=8, per=512, shots=1, niter=3,
             penalty="quad"),
        # the smallest operator application: a few thousand samples, two coils
        dict(name="ts2d_pair_32", kind="ts", dir="pair", n=32, nz=1, nc=2, L=4, inter=4, per=512),
        # field-corrected 2-D spiral imaging, each direction on its own
        dict(name="ts2d_fwd_128", kind="ts", dir="fwd", n=128, nz=1, nc=4, L=8, inter=16, per=8192),
        dict(name="ts2d_adj_128", kind="ts", dir="adj", n=128, nz=1, nc=4, L=8, inter=16, per=8192),
        # the same problem's reconstruction
        dict(name="pcg_ts2d_128", kind="pcg", op="ts", n=128, nz=1, nc=4, L=8, inter=16, per=8192, shots=1, niter=3,
             penalty="quad"),
        # a matrix size that is no power of two, more coils, a ragged sample count
        dict(name="ts2d_pair_208", kind="ts", dir="pair", n=208, nz=1, nc=12, L=10, inter=13, per=7681),
        # 3-D stack of spirals, no power of two in-plane
        dict(name="ts3d_pair_96", kind="ts", dir="pair", n=96, nz=16, nc=8, L=6, inter=1, per=4099),
        # high-resolution 3-D multishot (diffusion): shot phase maps, both directions
        dict(name="pcts_pair_128", kind="pcts", dir="pair", n=128, nz=64, nc=4, L=12, shots=2, per=2048),
        # 3-D multishot TV reconstruction
        dict(name="pcg_tv_64", kind="pcg", op="pcts", n=64, nz=32, nc=6, L=6, inter=1, per=1024, shots=4, niter=3,
             penalty="tv"),
        # exact field-corrected DFT, 3-D, 8 coils
        dict(name="gdft_fwd_64", kind="gdft", dir="fwd", r2=False, n=64, nz=32, nc=8, per=4096),
        # exact DFT of a multishot acquisition, ragged sizes, an odd number of coils, both directions
        dict(name="pcdft_pair_36", kind="pcdft", dir="pair", n=36, nz=11, nc=3, shots=2, per=1021),
        # the serving path on host arrays: two requests of several slices at once
        dict(name="serve_96", kind="serve", n=96, nc=8, L=6, inter=2, per=8192, slices=6, requests=2, niter=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, lo, hi):
    """An in-plane size: mostly multiples of 8, as scans prescribe them, now and then any integer."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.2 else max(lo, 8 * round(n / 8))


def draw(rng):
    kind = rng.choice(["ts2d", "ts2d", "ts2d", "ts3d", "pcts", "pcg", "pcg", "pcgtv", "gdft", "gdft", "pcdft", "serve"])
    if kind in ("ts2d", "pcg"):
        n = _matrix(rng, 32, 256)
        m = _log(rng, 2048, 200000)
        inter = max(1, round(m / 8192))
        L = rng.choice([1, 4, 5, 6, 8, 10, 12])
        nc = rng.randint(1, 32)
        # grids of one application: at most about the listed 208 case's
        nc = max(1, min(nc, int(24e6 / (4 * n * n * L))))
        d = dict(n=n, nz=1, nc=nc, L=L, inter=inter, per=max(256, m // inter))
        if kind == "ts2d":
            return dict(kind="ts", dir=rng.choice(["fwd", "adj", "pair"]), **d)
        return dict(kind="pcg", op="ts", shots=1, niter=rng.randint(2, 3), penalty="quad", **d)
    if kind == "ts3d":
        n, nz = _matrix(rng, 32, 128), rng.choice([8, 16, 24, 32])
        L = rng.randint(4, 12)
        nc = max(1, min(rng.randint(4, 32), int(60e6 / (8 * n * n * nz * L))))
        return dict(kind="ts", dir=rng.choice(["fwd", "adj", "pair"]), n=n, nz=nz, nc=nc, L=L, inter=1,
                    per=max(256, _log(rng, 8192, 131072) // nz))
    if kind in ("pcts", "pcgtv"):
        n, nz = 8 * round(_log(rng, 32, 96) / 8), rng.choice([8, 16, 32])
        shots, L = rng.randint(2, 4), rng.randint(4, 12)
        nc = max(1, min(rng.randint(2, 16), int((120e6 if kind == "pcts" else 30e6) / (8 * n * n * nz * L * shots))))
        per = max(256, _log(rng, 8192, 65536) // nz)
        if kind == "pcts":
            return dict(kind="pcts", dir="pair", n=n, nz=nz, nc=nc, L=L, shots=shots, per=per)
        return dict(kind="pcg", op="pcts", n=n, nz=nz, nc=nc, L=L, inter=1, per=per, shots=shots,
                    niter=rng.randint(2, 3), penalty="tv")
    if kind == "gdft":
        n, nz = _log(rng, 24, 64), rng.choice([1, 3, 8, 16, 31])
        nc = rng.randint(1, 16)
        m = _log(rng, 2048, 131072)
        m = max(1024, min(m, int(1.2e11 / (n * n * nz * nc))))
        return dict(kind="gdft", dir=rng.choice(["fwd", "adj", "pair"]), r2=rng.random() < 0.2, n=n, nz=nz, nc=nc,
                    per=max(64, m // nz))
    if kind == "pcdft":
        n, nz = _log(rng, 16, 40), rng.choice([4, 8, 11])
        return dict(kind="pcdft", dir="pair", n=n, nz=nz, nc=rng.randint(1, 8), shots=rng.randint(2, 4),
                    per=_log(rng, 128, 1024))
    n = 16 * rng.randint(4, 10)
    inter = rng.randint(1, 3)
    return dict(kind="serve", n=n, nc=rng.randint(4, 8), L=rng.randint(4, 8), inter=inter, per=8192,
                slices=rng.randint(1, 6), requests=rng.randint(1, 3), niter=rng.randint(2, 3))


# ---- inputs -------------------------------------------------------------------
def _coords(n, nz):
    z, x, y = np.meshgrid(np.arange(nz), np.arange(n), np.arange(n), indexing="ij")
    f = lambda v, m: ((v.astype(np.float32) - np.float32(m) / 2) / np.float32(m)).astype(np.float32).ravel()  # noqa: E731
    return f(x, n), f(y, n), f(z, nz)


def _spiral(r, n, inter, per, t_read, which=None):
    """Variable-density spirals, interleave-major, turned by a seeded angle: kx, ky in [-n/2, n/2), t."""
    kmax, turns = n / 2.0 * (1.0 - 1e-3), max(1.0, n / (2.0 * inter))
    phi = r.uniform(0, 2 * math.pi)
    tau = np.arange(per) / per
    kx, ky, t = [], [], []
    for s in range(inter) if which is None else which:
        th = 2 * math.pi * (turns * tau + s / inter) + phi
        kx.append(kmax * tau ** 1.5 * np.cos(th))
        ky.append(kmax * tau ** 1.5 * np.sin(th))
        t.append(tau * t_read)
    return [np.concatenate(v).astype(np.float32) for v in (kx, ky, t)]


def _stack(r, n, nz, inter, per, t_read, which=None):
    kx, ky, t = _spiral(r, n, inter, per, t_read, which)
    kz = np.repeat(np.arange(nz) - nz / 2.0, kx.size).astype(np.float32) if nz > 1 else np.zeros_like(kx)
    return np.tile(kx, nz), np.tile(ky, nz), kz, np.tile(t, nz)


def _field(r, n, nz, amp_hz):
    """Three smooth bumps, rad/s."""
    ix, iy, iz = _coords(n, nz)
    f = np.zeros(ix.shape)
    for _ in range(3):
        a, sg = r.uniform(-amp_hz, amp_hz), r.uniform(0.1, 0.3)
        cx, cy, cz = r.uniform(-0.5, 0.5, 3)
        f += a * np.exp(-((ix - cx) ** 2 + (iy - cy) ** 2 + ((iz - cz) ** 2 if nz > 1 else 0)) / (2 * sg * sg))
    return (2 * math.pi * np.clip(f, -amp_hz, amp_hz)).astype(np.float32)


def _coils(r, n, nz, nc):
    ix, iy, iz = _coords(n, nz)
    ph = r.uniform(-math.pi, math.pi, nc)
    out = np.empty((nc, ix.size), np.complex64)
    for c in range(nc):
        a = 2 * math.pi * c / nc
        d2 = (ix - 0.6 * math.cos(a)) ** 2 + (iy - 0.6 * math.sin(a)) ** 2
        if nz > 1:
            d2 = d2 + (iz - (0.25 if c % 2 else -0.25)) ** 2
        out[c] = np.exp(-d2 / 0.32) * np.exp(1j * ph[c])
    return out


def _shot_phases(r, n, nz, shots):
    ix, iy, iz = _coords(n, nz)
    out = np.empty((shots, ix.size), np.float32)
    for s in range(shots):
        a, bx, by, bz = r.uniform(-math.pi, math.pi, 4)
        out[s] = a + bx * ix + by * iy + (bz * iz if nz > 1 else 0)
    return out


def _noise(r, *shape):
    return (r.standard_normal(shape) + 1j * r.standard_normal(shape)).astype(np.complex64)


def _signal(r, kx, ky, kz, t, nc, nz):
    """Coil data (nc x M, unit RMS) of an object of Gaussian blobs with known transform, plus noise."""
    g = lambda v: torch.as_tensor(v, dtype=torch.float64, device=DEV)  # noqa: E731
    kx, ky, kz, t = (g(v) for v in (kx, ky, kz, t))
    y = torch.zeros(nc, kx.numel(), dtype=torch.complex128, device=DEV)
    for _ in range(12):
        cx, cy, cz = r.uniform(-0.35, 0.35, 3)
        sg, amp, om = r.uniform(0.01, 0.1), r.uniform(0.3, 1.0), 2 * math.pi * r.uniform(-80, 80)
        mag = amp * sg * sg * torch.exp(-2 * (math.pi * sg) ** 2 * (kx ** 2 + ky ** 2))
        ph = -2 * math.pi * (kx * cx + ky * cy + (kz * cz if nz > 1 else 0)) - om * t
        for c in range(nc):
            a = 2 * math.pi * c / nc
            w = math.exp(-((cx - 0.6 * math.cos(a)) ** 2 + (cy - 0.6 * math.sin(a)) ** 2) / 0.32)
            y[c] += w * torch.polar(mag, ph)
    e = g(r.standard_normal((nc, kx.numel(), 2)))
    y += 0.02 * y.abs().pow(2).mean().sqrt() * torch.view_as_complex(e)
    y = y / y.abs().pow(2).mean().sqrt()
    return y.to(torch.complex64)


def _inputs(case, seed):
    """Trajectory, maps and vectors of a case (numpy, and y on the device where it is a solve's data)."""
    r = np.random.RandomState((seed * 7919 + 17) % (2 ** 31))
    k = case["kind"] if case["kind"] != "pcg" else case["op"]
    n, nz, nc = case["n"], case.get("nz", 1), case["nc"]
    d = dict(n=n, nz=nz, nc=nc, N=n * n * nz, L=case.get("L", 1), shots=case.get("shots", 1))
    t_read = 20e-3 if nz == 1 else 10e-3
    if k in ("pcts", "pcdft"):
        parts = [_stack(r, n, nz, 16 if k == "pcts" else d["shots"], case["per"], t_read, [s])
                 for s in range(d["shots"])]
        d["kx"], d["ky"], d["kz"], d["t"] = (np.concatenate(v) for v in zip(*parts))
        d["pm"] = _shot_phases(r, n, nz, d["shots"])
    else:
        d["kx"], d["ky"], d["kz"], d["t"] = _stack(r, n, nz, case.get("inter", 1), case["per"], t_read)
    d["M"] = d["kx"].size // d["shots"]                 # samples per shot
    d["fm"] = _field(r, n, nz, 100.0 if nz == 1 else 150.0)
    d["sm"] = _coils(r, n, nz, nc) if nc > 1 else np.ones((1, d["N"]), np.complex64)
    ndata = nc * d["kx"].size                           # data order [coil][shot][sample]
    if case["kind"] == "pcg":
        d["y"] = _signal(r, d["kx"], d["ky"], d["kz"], d["t"], nc, nz)
        d["y"] = (d["y"] * (1.0 if nz == 1 else 1e-2)).reshape(-1).contiguous()   # clear of the solver's 1e25 guard
    elif case["kind"] == "serve":
        s = case["slices"]
        d["fm"] = np.stack([_field(r, n, 1, 100.0) for _ in range(s)])
        d["sm"] = np.stack([_coils(r, n, 1, nc) for _ in range(s)])
        d["y"] = np.stack([_signal(r, d["kx"], d["ky"], d["kz"], d["t"], nc, 1).cpu().numpy() for _ in range(s)])
    else:
        d["x"] = torch.from_numpy(_noise(r, d["N"])).to(DEV)
        d["y"] = torch.from_numpy(_noise(r, ndata)).to(DEV)
    return d


def _parts(case, seed):
    """The input sets of a case: one, or one per request of the server."""
    if case["kind"] != "serve":
        return [_inputs(case, seed)]
    return [_inputs(case, seed * 16 + q) for q in range(case["requests"])]


def _operator(case, d):
    k = case["kind"] if case["kind"] != "pcg" else case["op"]
    n, nz, N, M, nc = d["n"], d["nz"], d["N"], d["M"], d["nc"]
    if k == "pcts":
        return pg.pcSenseTimeSeg(d["kx"], d["ky"], d["kz"], n, n, nz, nc, d["t"], d["L"], 1, d["sm"], d["fm"], d["pm"])
    if k == "pcdft":
        return pg.pcSENSE(d["kx"], d["ky"], d["kz"], n, n, nz, nc, d["t"], d["sm"], d["fm"], d["pm"])
    if k == "gdft":
        ix, iy, iz = _coords(n, nz)
        a = (M, N, d["kx"], d["ky"], d["kz"], ix, iy, iz, d["fm"], d["t"])
        return pg.SENSE(pg.GdftR2(*a, n, n, nz) if case["r2"] else pg.Gdft(*a), d["sm"], M, N, nc)
    A = pg.Gnufft(M, 2.0, n, n, nz, d["kx"], d["ky"], d["kz"])
    if d["L"] > 1:
        A = pg.TimeSegmentation(A, d["fm"], d["t"], M, N, d["L"], 1, 1)
    return pg.SENSE(A, d["sm"], M, N, nc)


_BETA, _DELTA = 1e-3, 0.1


def prepare(case, seed):
    parts = _parts(case, seed)
    if case["kind"] == "serve":
        reqs = [pgserve.ReconRequest(nx=d["n"], ny=d["n"], nz=1, nc=d["nc"], L=d["L"], niter=case["niter"], beta=_BETA,
                                     kx=d["kx"], ky=d["ky"], kz=d["kz"], t=d["t"], field_map=d["fm"],
                                     sense_map=d["sm"], data=d["y"], n_slices=case["slices"]) for d in parts]
        return dict(case=case, srv=pgserve.Server(32 << 30, 8), reqs=reqs)
    d = parts[0]
    s = dict(case=case, A=_operator(case, d), x=d.get("x"), y=d["y"])
    if case["kind"] == "pcg":
        s["R"] = (pg.QuadPenalty(d["n"], d["n"], d["nz"], _BETA) if case["penalty"] == "quad" else
                  pg.TVPenalty(d["n"], d["n"], d["nz"], _BETA, _DELTA))
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "serve":
        tickets = [s["srv"].submit(q) for q in s["reqs"]]
        return [s["srv"].wait(t)[0] for t in tickets]
    if case["kind"] == "pcg":
        x = torch.empty(s["A"].n_image, dtype=torch.complex64, device=DEV)
        return pg.solve_pwls_pcg_device(s["A"], s["y"], s["R"], case["niter"], x)
    if case["dir"] == "fwd":
        return s["A"] * s["x"]
    if case["dir"] == "adj":
        return s["A"] / s["y"]
    return [s["A"] * s["x"], s["A"] / s["y"]]


# ---- what a pass cannot do without ---------------------------------------------
def work(case):
    k = case["kind"] if case["kind"] != "pcg" else case["op"]
    n, nz, nc = case["n"], case.get("nz", 1), case["nc"]
    N, shots, L = n * n * nz, case.get("shots", 1), case.get("L", 1)
    dim = 2 if nz == 1 else 3
    M = (case["per"] * case.get("inter", 1) if k in ("ts", "serve") else case["per"]) * nz
    # one application: trajectory and times, maps, phases, image and data once each
    by = shots * M * (4 * dim + 4) + 12 * N + 8 * N * nc + 8 * nc * shots * M + (4 * N * shots if shots > 1 else 0)
    if k in ("gdft", "pcdft"):
        # phase: dim + 1 products, sine and cosine; one complex multiply-add per coil
        fl = shots * M * N * (2 * (dim + 1) + 2 + 8 * nc)
    else:
        G = N * 2 ** dim
        K = 1 if L == 1 else 2
        # pruned transforms (half the lines of every axis but the last), gridding taps, image weights
        lines = sum(0.5 ** (dim - 1 - a) for a in range(dim))
        fl = shots * nc * (L * (5 * G * math.log2(2 * n) * lines + 14 * N) + M * K * (8 ** dim * 4 + 8))
    if case["kind"] == "pcg":
        it = case["niter"]
        return {"bytes": it * (2 * by + 8 * (6 * nc * shots * M + 6 * N)),
                "flops": it * (2 * fl + 20 * nc * shots * M + 60 * N)}
    if case["kind"] == "serve":
        q = case["slices"] * case["requests"] * case["niter"]
        return {"bytes": q * (2 * by + 8 * (6 * nc * M + 6 * N)), "flops": q * (2 * fl + 20 * nc * M + 60 * N)}
    f = 2 if case["dir"] == "pair" else 1
    return {"bytes": f * by, "flops": f * fl}


def tolerance(case):
    # About four times the largest distance from the 64-bit values (see `exact`) over the ranges.
    # Operators in 32 bits: gridding 1.5e-6 (window weights and transforms), exact DFT 4.8e-7.
    # Solves: conjugate gradients amplify the operator's rounding from step to step, most for one
    # coil without a field map (9.2e-5 after five steps), least under the total-variation penalty.
    if case["kind"] == "pcg":
        return {"rel": 4e-4 if case["penalty"] == "quad" else 2e-5}
    if case["kind"] == "serve":
        return {"rel": 2e-5}
    if case["kind"] in ("gdft", "pcdft"):
        return {"rel": 2e-6}
    return {"rel": 6e-6}


# ---- 64-bit values ---------------------------------------------------------------
def _lut():
    """The Kaiser-Bessel table of oversampling 2, width 4, and its beta (griddingSupport.cpp:33-76, Gnufft.cpp:84-88)."""
    f = np.float32
    beta = f(float(f(math.pi)) * math.sqrt(1.5 * 1.5 * (4.0 * 4.0 * 4.0) / 4.0 - 0.8))
    v = np.arange(40000, dtype=f) / f(40000)
    ax = (float(beta) * np.sqrt(1.0 - v.astype(np.float64))).astype(f)
    lo = (ax / 3.75).astype(f)
    lo = (lo * lo).astype(f).astype(np.float64)
    small = 1.0 + lo * (3.5156229 + lo * (3.0899424 + lo * (1.2067492 + lo * (0.2659732 + lo * (
        0.360768e-1 + lo * 0.45813e-2)))))
    a = np.maximum(ax, f(3.75))
    y = (3.75 / a).astype(f).astype(np.float64)
    big = (np.exp(a) / np.sqrt(a)).astype(np.float64) * (
        0.39894228 + y * (0.1328592e-1 + y * (0.225319e-2 + y * (-0.157565e-2 + y * (0.916281e-2 + y * (
            -0.2057706e-1 + y * (0.2635537e-1 + y * (-0.1647633e-1 + y * 0.392377e-2))))))))
    return (np.where(ax < 3.75, small, big).astype(f) / f(4)).astype(np.float64), float(beta)


class _Grid:
    """Gnufft's definition for a set of samples, in double: centred grid of 2n per axis."""

    def __init__(self, kx, ky, kz, n, nz):
        self.dims = [n, n] if nz == 1 else [n, n, nz]           # x, y (, z)
        lut, beta = _lut()
        lut = torch.as_tensor(lut, device=DEV)
        self.taps = []
        for k, m in zip((kx, ky, kz), self.dims):
            k = torch.as_tensor(k, dtype=torch.float32, device=DEV)
            s = 2.0 * (k + m / 2.0)
            lo, hi = (s - 4).ceil().clamp(min=0), (s + 4).floor().clamp(max=2 * m - 1)
            st = torch.where(hi - lo == 8, lo + 1, lo)          # of nine cells the end ones weigh 0
            idx, w = [], []
            for a in range(8):
                c = st + a
                dist = (s - c).abs() / 2
                e = ((dist * dist * 4.0) / 16.0 * 40000.0).to(torch.int64)
                ok = (c <= hi) & (e < 40000)
                w.append(torch.where(ok, lut[e.clamp(max=39999)], torch.zeros((), dtype=torch.float64, device=DEV)))
                idx.append(c.to(torch.int64).clamp(max=2 * m - 1))
            self.taps.append((idx, w))
        f, dims = np.float32, self.dims
        de = []
        for m in dims:
            i = np.arange(m)
            u = ((i - (m // 2)).astype(f) / f(m) if nz == 1 else ((i - m / 2.0).astype(f) / f(m)).astype(f))
            pi = f(math.pi)
            c = (((pi * pi * f(4)) * f(4)) * u * u - f(beta) * f(beta)).astype(np.float64)
            r = np.sqrt(np.abs(c))
            de.append(np.where(c >= 0, np.sin(r) / np.where(r == 0, 1, r), np.sinh(r) / np.where(r == 0, 1, r)))
        k = de[0][:, None] * de[1][None, :]                     # [x, y]
        if nz > 1:
            k = de[2][:, None, None] * k[None]                  # [z, x, y]
        self.deap = torch.as_tensor(1.0 / (2.0 ** len(dims) * k), device=DEV)
        self.shape = [2 * n, 2 * n] if nz == 1 else [2 * nz, 2 * n, 2 * n]
        order = [0, 1] if nz == 1 else [2, 0, 1]
        self.sl = tuple(slice(int(dims[a] - dims[a] / 2.0), int(dims[a] - dims[a] / 2.0) + dims[a]) for a in order)
        self.axes = list(range(1, 1 + len(dims)))

    def _each(self, sel):
        """Flat cell index and weight of every tap of the selected samples."""
        n2 = 2 * self.dims[0]
        (xi, xw), (yi, yw) = self.taps[:2]
        for a in range(8):
            for b in range(8):
                cell, w = xi[a][sel] * n2 + yi[b][sel], xw[a][sel] * yw[b][sel]
                if len(self.taps) == 2:
                    yield cell, w
                else:
                    for zi, zw in zip(*self.taps[2]):
                        yield cell + zi[sel] * n2 * n2, w * zw[sel]

    def forward(self, u, sel):
        """u: B x image (z, x, y order) -> B x selected samples."""
        B = u.shape[0]
        g = torch.zeros([B] + self.shape, dtype=torch.complex128, device=DEV)
        g[(slice(None),) + self.sl] = u.reshape([B] + list(self.deap.shape)) * self.deap
        g = torch.fft.ifftshift(torch.fft.fftn(torch.fft.fftshift(g, self.axes), dim=self.axes), self.axes)
        g = g.reshape(B, -1)
        y = torch.zeros(B, sel.numel(), dtype=torch.complex128, device=DEV)
        for cell, w in self._each(sel):
            y += g[:, cell] * w
        return y

    def adjoint(self, v, sel):
        B = v.shape[0]
        g = torch.zeros(B, math.prod(self.shape), dtype=torch.complex128, device=DEV)
        for cell, w in self._each(sel):
            g.index_add_(1, cell, v * w)
        g = g.reshape([B] + self.shape)
        g = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(g, self.axes), dim=self.axes, norm="forward"),
                               self.axes)
        return (g[(slice(None),) + self.sl] * self.deap).reshape(B, -1)


def _d(v):
    v = v if isinstance(v, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(v))
    return v.to(DEV).to(torch.complex128 if v.is_complex() else torch.float64)


class _ExactTs:
    """SENSE<TimeSegmentation<Gnufft>> per shot, with shot phases where the case has them."""

    def __init__(self, d):
        self.d, self.S = d, _d(d["sm"])
        M, L = d["M"], d["L"]
        self.shots = []
        for s in range(d["shots"]):
            q = slice(s * M, (s + 1) * M)
            g = _Grid(d["kx"][q], d["ky"][q], d["kz"][q], d["n"], d["nz"])
            E = torch.polar(torch.ones(d["N"], dtype=torch.float64, device=DEV), -_d(d["pm"][s])) if "pm" in d else None
            segs = []
            if L == 1:
                segs.append((None, None, torch.arange(M, device=DEV)))
            else:
                t = d["t"][q]
                tmin = t.min()
                tau = np.float32((np.float32(t.max() - tmin) + np.finfo(np.float64).eps) / L)
                tm = (t - tmin).astype(np.float32)
                for l in range(L):
                    df = (tm - np.float32(l) * tau).astype(np.float32)
                    aa = np.where(np.abs(df) <= tau, 0.5 + 0.5 * np.cos(math.pi * df.astype(np.float64) / float(tau)), 0)
                    sel = np.nonzero(aa)[0]
                    sft = np.float32(np.float32(l) * tau + tmin)
                    ph = -_d((d["fm"] * sft).astype(np.float32))
                    segs.append((torch.polar(torch.ones_like(ph), ph), _d(aa[sel]), torch.as_tensor(sel, device=DEV)))
            self.shots.append((g, E, segs))

    def forward(self, x):
        d = self.d
        y = torch.zeros(d["nc"], d["shots"], d["M"], dtype=torch.complex128, device=DEV)
        for s, (g, E, segs) in enumerate(self.shots):
            xs = x * self.S if E is None else x * self.S * E
            for wo, aa, sel in segs:
                v = g.forward(xs if wo is None else xs * wo, sel)
                y[:, s, sel] += v if aa is None else v * aa
        return y.reshape(-1)

    def adjoint(self, y):
        d = self.d
        y = y.reshape(d["nc"], d["shots"], d["M"])
        x = torch.zeros(d["N"], dtype=torch.complex128, device=DEV)
        for s, (g, E, segs) in enumerate(self.shots):
            for wo, aa, sel in segs:
                v = y[:, s, sel]
                im = g.adjoint(v if aa is None else v * aa, sel) * self.S.conj()
                if wo is not None:
                    im = im * wo.conj()
                x += im.sum(0) if E is None else im.sum(0) * E.conj()
        return x


class _ExactDft:
    """SENSE<Gdft>, SENSE<GdftR2> (r2) and pcSENSE (shot phases, +iP in both directions as in pcSENSE.cpp:103, 146)."""

    def __init__(self, d, r2):
        self.d, self.S, self.r2 = d, _d(d["sm"]), r2
        self.r = [_d(v) for v in _coords(d["n"], d["nz"])]
        self.fm = _d(d["fm"])
        if r2:
            n, N, fm = d["n"], d["N"], self.fm
            self.gr = []
            for off in (1, n, n * n):                           # GdftR2.cpp:62-110
                g = torch.zeros_like(fm)
                if off < N:
                    i = torch.arange(N, device=DEV)
                    up, dn = torch.where(i < N - off, i + off, i), torch.where(i < off, i, i - off)
                    g = fm[up] - fm[dn]
                self.gr.append(g)

    def _chunks(self, s):
        d = self.d
        M, step = d["M"], max(1, int(1.5e8) // d["N"])
        dims = [d["n"], d["n"], d["nz"]]
        for a in range(0, M, step):
            q = slice(s * M + a, s * M + min(M, a + step))
            k = [_d(d[c][q]) for c in ("kx", "ky", "kz")]
            t = _d(d["t"][q])
            ph = t[:, None] * self.fm
            for kk, r in zip(k, self.r):
                ph += 2 * math.pi * kk[:, None] * r
            e = torch.polar(torch.ones_like(ph), -ph)
            if self.r2:
                for kk, m, g in zip(k, dims, self.gr):
                    e *= torch.sinc(kk[:, None] / m + t[:, None] * g)
            yield slice(a, min(M, a + step)), e

    def _E(self, s):
        if "pm" not in self.d:
            return 1.0
        p = _d(self.d["pm"][s])
        return torch.polar(torch.ones_like(p), p)

    def forward(self, x):
        d = self.d
        y = torch.zeros(d["nc"], d["shots"], d["M"], dtype=torch.complex128, device=DEV)
        for s in range(d["shots"]):
            xs = (x * self._E(s) * self.S).T.contiguous()
            for q, e in self._chunks(s):
                y[:, s, q] = (e @ xs).T
        return y.reshape(-1)

    def adjoint(self, y):
        d = self.d
        y = y.reshape(d["nc"], d["shots"], d["M"])
        x = torch.zeros(d["N"], dtype=torch.complex128, device=DEV)
        for s in range(d["shots"]):
            im = torch.zeros(d["nc"], d["N"], dtype=torch.complex128, device=DEV)
            for q, e in self._chunks(s):
                im += y[:, s, q] @ e.conj()
            x += self._E(s) * (im * self.S.conj()).sum(0)
        return x


def _gradient(pen, z, offs):
    """Robject::Gradient with its boundary rules (Robject.cpp:76-117); delta None: quadratic."""
    beta, delta = pen
    g = torch.zeros_like(z)
    N = z.numel()
    for off in offs:
        if off >= N:
            continue
        c = torch.zeros_like(z)
        c[off:] = z[off:] - z[:-off]
        if delta:
            c = c / torch.sqrt(1 + (c / delta).abs() ** 2)
        o = torch.zeros_like(z)
        o[:N - 1 - off] = c[:N - 1 - off] - c[off:N - 1]
        o[N - 1 - off] = c[N - 1 - off]
        g += o
    return beta * g


def _denom(pen, d, z, offs):
    beta, delta = pen
    s = 0.0
    for off in offs:
        if off >= z.numel():
            continue
        cd, cz = d[off:] - d[:-off], z[off:] - z[:-off]
        w = 1.0 / torch.sqrt(1 + (cz / delta).abs() ** 2) if delta else 1.0
        s += float((w * cd.abs() ** 2).sum())
    return beta * s


def _solve(A, y, pen, offs, N, niter):
    """solve_pwls_pcg (solve_pwls_pcg.hpp:48-167) with W = 1 and a zero start."""
    dot = lambda a, b: float((a.conj() * b).real.sum())  # noqa: E731
    x = torch.zeros(N, dtype=torch.complex128, device=DEV)
    Ax, d, old, yy = torch.zeros_like(y), torch.zeros_like(x), 0.0, dot(y, y)
    for it in range(niter):
        r = y - Ax
        g = A.adjoint(r)
        if math.sqrt(dot(g, g)) / yy < 1e-10:
            break
        g = g - _gradient(pen, x, offs)
        new = dot(g, g)
        gamma = 0.0 if it == 0 or abs(old) < 1e-10 else new / old
        old = new
        d = g + gamma * d
        if dot(d, g) < 0:
            break
        Ad = A.forward(d)
        daw, dr, step = dot(Ad, Ad), dot(Ad, r), 0.0
        for _ in range(3):
            z = x + step * d
            den = daw + _denom(pen, d, z, offs)
            if abs(den) < 1e-20 or abs(den) > 1e25:
                return x
            step -= (-dr + step * daw + dot(d, _gradient(pen, z, offs))) / den
        Ax, x = Ax + step * Ad, x + step * d
    return x


def exact(case, seed):
    parts = _parts(case, seed)
    if case["kind"] == "serve":
        out = []
        for d in parts:
            im = []
            for s in range(case["slices"]):
                A = _ExactTs(dict(d, fm=d["fm"][s], sm=d["sm"][s]))
                im.append(_solve(A, _d(d["y"][s]).reshape(-1), (_BETA, None), [1, d["n"]], d["N"], case["niter"]))
            out.append(torch.stack(im).cpu().numpy())
        return out
    d = parts[0]
    k = case["kind"] if case["kind"] != "pcg" else case["op"]
    A = _ExactDft(d, case.get("r2", False)) if k in ("gdft", "pcdft") else _ExactTs(d)
    if case["kind"] == "pcg":
        offs = [1, d["n"]] + ([d["n"] ** 2] if d["nz"] > 1 else [])
        return _solve(A, _d(d["y"]), (_BETA, _DELTA if case["penalty"] == "tv" else None), offs, d["N"], case["niter"])
    if case["dir"] == "fwd":
        return A.forward(_d(d["x"]))
    if case["dir"] == "adj":
        return A.adjoint(_d(d["y"]))
    return [A.forward(_d(d["x"])), A.adjoint(_d(d["y"]))]
